// What the kernels of p3_gemm_any share: the parameters of a launch and the walk over its row tiles.
#pragma once
#include "common.cuh"

namespace {
struct AnyP {
    const void* X; int64_t ldx; const int32_t* x_rows; int x_row_div;
    const void* W; int64_t ldw; int64_t w_gstride;
    const float* bias; int64_t bias_gstride;
    void* out; int64_t ldo;
    int64_t M; int N, K;
    const int32_t* seg; int n_groups;
    // a batch of nb products over column blocks of X and out: blockIdx.x = m-tile * nb + product, so that the CTAs in flight
    // together read whole rows of X and write whole rows of out (neighbouring column blocks) instead of one narrow column each
    int nb; int64_t x_bs, w_bs, o_bs; const float* gate; int64_t ld_gate;
};

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<bf16>(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

// which (group, first row, end row) does the m-tile `tile` of TM rows cover? Groups are walked in order; a launch has at most
// ceil(M / TM) + n_groups tiles, surplus CTAs leave.
template <int TM>
__device__ __forceinline__ bool find_tile(const AnyP& p, int tile, int& g, int64_t& m0, int64_t& m1) {
    if (!p.seg) { g = 0; m0 = (int64_t)tile * TM; m1 = p.M; return m0 < m1; }
    int t = tile;
    for (int e = 0; e < p.n_groups; e++) {
        const int a = p.seg[e], b = p.seg[e + 1], nt = (b - a + TM - 1) / TM;
        if (t < nt) { g = e; m0 = a + (int64_t)t * TM; m1 = b; return true; }
        t -= nt;
    }
    return false;
}
}  // namespace
