// What the kernels of the windowed attention share (attention_window.cu, attention_window_tc.cu).
#pragma once
#include "common.cuh"
#include "../../include/phi3_b200.h"

// first position that a query at `pos` sees (kept first tokens aside): the start of its window, the start of its chunk, or 0. It
// never falls as pos grows.
__device__ __forceinline__ int first_key(const p3_attn_window_args& a, int pos) {
    int lo = 0;
    if (a.window > 0) lo = max(lo, pos - a.window + 1);
    if (a.chunk > 0) lo = max(lo, pos - pos % a.chunk);
    return lo;
}
