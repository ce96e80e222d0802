// Entry points of the LayerNorm kernels (norm.cu), as torch_norm.cpp and ops/norm.py call them.
#pragma once

extern "C" {
int ccf_layernorm_max_d();
int ccf_layernorm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows, int d, float eps,
                      int fp16, void* stream);
int ccf_layernorm_bwd_parts(int rows, int d);
int ccf_layernorm_bwd(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd, void* dx, float* part,
                      void* dgamma, void* dbeta, int rows, int d, int fp16, int* status, unsigned long long wait_limit_ns, void* stream);
}
