"""Operands off a 16-byte boundary never reach a kernel: the entry points refuse them before any CUDA call. No GPU, made-up addresses."""
import ctypes as C

import pytest

from ccfuser_b200 import native as N

A = 1 << 20      # an address that nothing reads


@pytest.mark.parametrize("off", range(4))
def test_layernorm_entry_points_refuse(off):
    lib = N.load()
    x, w, b, y = (A + (2 if off == i else 0) for i in range(4))
    assert lib.ccf_layernorm_fwd(x, w, b, y, A, A, 4, 64, 1e-5, 0, None) == -2
    x, dy, w, dx = (A + (8 if off == i else 0) for i in range(4))
    assert lib.ccf_layernorm_bwd(x, dy, w, A, A, dx, A, A, A, 4, 64, 0, A, 1, None) == -2


@pytest.mark.parametrize("epi,backward", [(N.EPI_BIAS_ACT, 0), (N.EPI_DSWIGLU, 1)])
def test_dispatch_role_refuses(epi, backward):
    L = N.GemmLaunch()
    L.device, L.epi, L.a_major, L.b_major = -1, epi, N.MAJ_K, N.MAJ_MN if backward else N.MAJ_K
    g = L.args
    g.num_groups, g.n, g.k, g.n_comm_ctas = 1, 64, 64, 4
    g.disp.backward, g.disp.x = backward, A + 2
    assert N.load().ccf_gemm_launch(C.byref(L), None) == -14
