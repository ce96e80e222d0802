// Entry point of the one-kernel routing + plan (route.cu).
#pragma once
#include "gemm_args.h"

// slots one cluster holds: 8 CTAs x 1024 threads x 8 slots
#define CCF_ROUTE_CLUSTER_SLOTS 65536

extern "C" int ccf_route_plan(const int* expert, int S, int E, int cap, int* pos, int* count_raw, int* count_kept,
                              int* order_off, int* sorted_slot, int* slot_row, int first_expert, int* raw_order,
                              const CcfPlanArgs* plan, int* epoch_counter, void* stream);
