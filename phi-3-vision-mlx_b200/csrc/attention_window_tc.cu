// Windowed / chunked / gated prefill attention over the page pools (the contract of attention_window.cu) on the 5th-gen tensor cores, for
// bf16 with key sizes and value sizes that are multiples of 16 up to 128.
//
// One CTA = NX blocks of 128 query rows against the pages of ONE sequence and K/V head; a block is two halves of 64 rows, a half is one
// tile record x one query head. The halves of a CTA are n_hc query heads of one group x n_tc neighbouring tile records (n_hc n_tc <= 2 NX),
// so that grouped-query heads share the K/V pages that a CTA stages. Records of different sequences in one CTA take a pass each.
//   warps 0 .. 4 NX - 1: softmax, thread = query row (TMEM lane). S is double buffered in TMEM, so a block's scores of the next two pages are
//               computed while this one is swept; P (bf16) goes back over the consumed S columns and is the A operand of P.V straight from
//               TMEM. P is formed against the running reference maximum of the pages before (base-2 domain; the sink is the first
//               reference, with a denominator of 1); the page's own maximum is found in the same sweep. O and l are rescaled when the
//               reference falls 2^8 behind, and the page is swept again when it falls 2^64 behind or there was none. Scores, penalties,
//               weights before their rounding and all sums are fp32, two per instruction where that goes.
//   warp 4 NX:  TMA producer, one page = 64-column SWIZZLE_128B boxes of K and of V, two mbarrier rings
//   warps behind it: one MMA issuer per block: O += P(j) V(j), then S(j + 2) = Q K(j + 2)^T into the columns P(j) left
// Q rows are copied by the softmax warps (rows beyond a tile's end are not read). The penalties of a warp's 95 distances to a page are staged
// by that warp, read one page ahead.
//
// Every wait has an iteration limit: when one runs out the CTA stops waiting, writes NaN and ends.
#include "tc_common.cuh"
#include "../../include/phi3_b200.h"
#include <climits>
#include <type_traits>

namespace {
constexpr float LOG2E = 1.4426950408889634f;
constexpr int BOX = 64 * 128;                                // bytes of one 64-row x 64-column box

__device__ __forceinline__ void wait_lim(uint32_t bar, uint32_t parity, volatile int* fail) {
    uint32_t ok, spins = 0;
    do {
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (!ok && (++spins & 1023u) == 0) {
            if (*fail) return;
            if (spins > (1u << 24)) { *fail = 1; return; }
        }
    } while (!ok);
}
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcpf(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
// two fp32 operations per instruction
__device__ __forceinline__ void fma2(float& x, float& y, float a0, float a1, float b0, float b1, float c0, float c1) {
    asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\nfma.rn.f32x2 d, a, b, c;\nmov.b64 {%0, %1}, d;\n}"
        : "=f"(x), "=f"(y) : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void add2(float& x, float& y, float a0, float a1, float b0, float b1) {
    asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nadd.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
        : "=f"(x), "=f"(y) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
// first position that a query at `pos` sees (kept first tokens aside), as in attention_window.cu
__device__ __forceinline__ int first_key(const p3_attn_window_args& a, int pos) {
    int lo = 0;
    if (a.window > 0) lo = max(lo, pos - a.window + 1);
    if (a.chunk > 0) lo = max(lo, pos - pos % a.chunk);
    return lo;
}

struct WinMaps { CUtensorMap k, v; };
// penalties of a warp's 32 rows against a page: entry t = distance (first row + 31 - t) to the page's first key, so that a row's 64 columns are
// neighbours; four copies shifted by 0 .. 3 entries let every lane read 16-byte pieces, and their pitch keeps a quarter-warp on different banks
constexpr int PEN_LD = 104;

template <int NX> struct WinCfg {
    static constexpr int ST = NX == 2 ? 4 : 2;               // pages in flight
    static constexpr int THREADS = 32 * (5 * NX + 1);
    static constexpr int TMEM = 256 * NX, O_COL = 128 * NX;  // S_x(buffer) at 128 x + 64 buffer, O_x at O_COL + 128 x
    // Q blocks of up to 2 boxes x 128 rows, K and V pages of up to 2 boxes, penalty slices, barriers
    static size_t smem(int kb, int vb) { return (size_t)NX * kb * 2 * BOX + (size_t)ST * (kb + vb) * BOX + NX * 4 * 4 * PEN_LD * 4 + 256 + 1024; }
};

template <int NX, bool PEN, bool SIG>
__global__ void __launch_bounds__(WinCfg<NX>::THREADS, NX == 2 ? 1 : 2)
attn_window_prefill_tc_kernel(const __grid_constant__ WinMaps tm, p3_attn_window_args a, int n_hc, int n_tc) {
    using C = WinCfg<NX>;
    constexpr int ST = C::ST, W_TMA = 4 * NX, W_MMA = W_TMA + 1;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int fail_s;
    __shared__ uint32_t tmem_s;
    volatile int* fail = &fail_s;
    const int d = a.dim, dv = a.vdim, kb = (d + 63) / 64, vb = (dv + 63) / 64, rep = a.n_heads / a.n_kv;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    const uint32_t sQ = base, q_bytes = (uint32_t)kb * 2 * BOX, sK = sQ + NX * q_bytes, sV = sK + ST * kb * BOX;
    const uint32_t pen_off = sV + ST * vb * BOX - raw, bars = sV + ST * vb * BOX + NX * 4 * 4 * PEN_LD * 4;
    const uint32_t q_full = bars;
    auto k_full = [&](int s) { return bars + 8u * (1 + s); };
    auto k_empty = [&](int s) { return bars + 8u * (1 + ST + s); };
    auto v_full = [&](int s) { return bars + 8u * (1 + 2 * ST + s); };
    auto v_empty = [&](int s) { return bars + 8u * (1 + 3 * ST + s); };
    auto s_full = [&](int x, int j) { return bars + 8u * (1 + 4 * ST + 2 * x + (j & 1)); };
    auto sm_done = [&](int x, int j) { return bars + 8u * (1 + 4 * ST + 2 * NX + 2 * x + (j & 1)); };
    auto o_done = [&](int x, int j) { return bars + 8u * (1 + 4 * ST + 4 * NX + 2 * x + (j & 1)); };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hgs = a.n_heads / n_hc, groups = (a.n_tiles + n_tc - 1) / n_tc;
    const int hg = blockIdx.x % hgs, grp = groups - 1 - blockIdx.x / hgs;      // later tiles (more keys) first
    const int h0 = hg * n_hc, g = h0 / rep;

    auto init_bars = [&]() {
        mbar_init(q_full, 4 * NX);
        for (int s = 0; s < ST; s++) { mbar_init(k_full(s), 1); mbar_init(k_empty(s), NX); mbar_init(v_full(s), 1); mbar_init(v_empty(s), NX); }
        for (int x = 0; x < NX; x++)
            for (int j = 0; j < 2; j++) { mbar_init(s_full(x, j), 1); mbar_init(o_done(x, j), 1); mbar_init(sm_done(x, j), 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    };
    if (warp == W_TMA && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tm.k)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tm.v)) : "memory");
    }
    if (warp == W_MMA) {
        if (lane == 0) { init_bars(); fail_s = 0; }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "n"(C::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_s);
    pdl_trigger();
    pdl_wait();                                              // q, the pools, the tile records and `out` belong to earlier kernels until here

    const int t_end = min(a.n_tiles, (grp + 1) * n_tc);
    const int4* recs = reinterpret_cast<const int4*>(a.tiles);
    for (int ta = grp * n_tc; ta < t_end;) {
        // ---- one pass: the records [ta, tb) of one sequence
        const int slot = recs[ta].z;
        int tb = ta, first = INT_MAX, last = 0, last_x[2] = {-1, -1};
        for (; tb < t_end; tb++) {
            const int4 r = recs[tb];
            if (r.z != slot) break;
            first = min(first, first_key(a, r.w));
            const int l = r.w + r.y - 1, u0 = (tb - grp * n_tc) * n_hc;         // this record's halves: u0 .. u0 + n_hc - 1
            last = max(last, l);
#pragma unroll
            for (int x = 0; x < NX; x++) if (u0 < 2 * x + 2 && u0 + n_hc > 2 * x) last_x[x] = max(last_x[x], l);
        }
        // pages: those of the kept first tokens before the window's pages, then from the first visible key to the last row's position
        const int lo_pg = first / 64, n_keep = min((a.keep_first + 63) / 64, lo_pg);
        auto page_at = [&](int it) { return it < n_keep ? it : lo_pg + it - n_keep; };
        int n_x[2];
#pragma unroll
        for (int x = 0; x < NX; x++) n_x[x] = last_x[x] < 0 ? 0 : n_keep + max(0, last_x[x] / 64 - lo_pg + 1);
        const int n = n_keep + last / 64 - lo_pg + 1;
        const int32_t* bt = a.block_table + (size_t)slot * a.bt_stride;

        if (warp == W_TMA) {
            if (lane == 0) {
                for (int it = 0; it < n; it++) {
                    const int st = it % ST;
                    const uint32_t ph = (uint32_t)(it / ST) & 1u;
                    const int row = (bt[page_at(it)] * a.n_kv + g) * 64;
                    wait_lim(k_empty(st), ph ^ 1u, fail);
                    mbar_expect_tx(k_full(st), kb * BOX);
                    for (int b = 0; b < kb; b++) tma_load_2d(sK + (st * kb + b) * BOX, &tm.k, k_full(st), 64 * b, row);
                    wait_lim(v_empty(st), ph ^ 1u, fail);
                    mbar_expect_tx(v_full(st), vb * BOX);
                    for (int b = 0; b < vb; b++) tma_load_2d(sV + (st * vb + b) * BOX, &tm.v, v_full(st), 64 * b, row);
                }
                for (int it = max(0, n - ST); it < n; it++) {          // every release has arrived before the barriers may be set up anew
                    wait_lim(k_empty(it % ST), (uint32_t)(it / ST) & 1u, fail);
                    wait_lim(v_empty(it % ST), (uint32_t)(it / ST) & 1u, fail);
                }
            }
        } else if (warp >= W_MMA) {
            // MMA issuer of block x (whole warp converged, one elected lane issues). A stage is released by a commit of every issuer, also of
            // one whose block needs fewer pages.
            const int x = warp - W_MMA, nx = n_x[x], ks = d / 16;
            constexpr uint32_t ID = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
            const uint32_t id_qk = ID | ((64u >> 3) << 17), id_pv = ID | (1u << 16) | ((uint32_t)(dv >> 3) << 17);
            const uint32_t s_col = tmem + 128 * x, o_col = tmem + C::O_COL + 128 * x, qa = sQ + x * q_bytes;
            wait_lim(q_full, 0, fail);
            for (int t = 0; t < n + 2; t++) {
                const int j = t - 2;
                if (j >= 0) {                                // O += P(j) V(j)
                    wait_lim(v_full(j % ST), (uint32_t)(j / ST) & 1u, fail);
                    if (j < nx) wait_lim(sm_done(x, j), (uint32_t)(j >> 1) & 1u, fail);
                    tc_fence_after();
                    if (elect_one()) {
                        if (j < nx) {
                            const uint32_t p_col = s_col + (j & 1) * 64, vs = sV + (j % ST) * vb * BOX;
#pragma unroll
                            for (int kk = 0; kk < 4; kk++)
                                tc_mma_bf16_ts(o_col, p_col + 8 * kk, umma_desc_mn_sw128(vs + kk * (16 * 128), BOX, 1024), id_pv, (j | kk) ? 1u : 0u);
                            tc_commit(o_done(x, j));
                        }
                        tc_commit(v_empty(j % ST));
                    }
                    __syncwarp();
                }
                if (t < n) {                                 // S(t) = Q K(t)^T, behind the P.V that reads the same columns
                    wait_lim(k_full(t % ST), (uint32_t)(t / ST) & 1u, fail);
                    tc_fence_after();
                    if (elect_one()) {
                        if (t < nx) {
                            const uint32_t ksm = sK + (t % ST) * kb * BOX, dst = s_col + (t & 1) * 64;
                            for (int kk = 0; kk < ks; kk++)
                                tc_mma_bf16(dst, umma_desc_sw128(qa + (kk >> 2) * 2 * BOX) + 2 * (kk & 3), umma_desc_sw128(ksm + (kk >> 2) * BOX) + 2 * (kk & 3),
                                            id_qk, kk ? 1u : 0u);
                            tc_commit(s_full(x, t));
                        }
                        tc_commit(k_empty(t % ST));
                    }
                    __syncwarp();
                }
            }
        } else {
            // ---- softmax: warp wq of block x; its 32 rows belong to one half (one record, one head)
            const int x = warp >> 2, wq = warp & 3, u = 2 * x + (wq >> 1), rec_i = grp * n_tc + u / n_hc, h = h0 + u % n_hc;
            const bool mine = rec_i >= ta && rec_i < tb;
            const int4 rec = recs[mine ? rec_i : ta];
            const int r0 = (wq & 1) * 32, i = r0 + lane, nq = mine ? rec.y : 0, pos = rec.w + i;
            const bool row_ok = i < nq;
            {   // the warp's 32 query rows -> shared memory, swizzled as the UMMA reads them
                const bf16* q = (const bf16*)a.q + (size_t)rec.x * a.ld_q + (size_t)h * d;
                const int ch = d / 8;
                for (int e0 = lane; e0 < 32 * ch; e0 += 256) {       // eight loads in flight per lane
                    uint4 v[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int e = e0 + 32 * k, rr = e / ch, c = e - rr * ch;
                        v[k] = e < 32 * ch && r0 + rr < nq ? *reinterpret_cast<const uint4*>(q + (size_t)(r0 + rr) * a.ld_q + 8 * c) : make_uint4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int e = e0 + 32 * k, rr = e / ch, c = e - rr * ch, lr = (wq >> 1) * 64 + r0 + rr;
                        const uint32_t dst = sQ + x * q_bytes + (c >> 3) * 2 * BOX + lr * 128 + (((c & 7) ^ (lr & 7)) << 4);
                        if (e < 32 * ch) asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v[k].x), "r"(v[k].y), "r"(v[k].z), "r"(v[k].w) : "memory");
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(q_full);
            }
            const int nx = n_x[x];
            const uint32_t t_lane = tmem + ((uint32_t)(wq * 32) << 16), t_o = t_lane + C::O_COL + 128 * x;
            const float scale2 = a.scale * LOG2E, sb2 = SIG ? a.sig_bias[h] * LOG2E : 0.f;
            float m = a.sink ? a.sink[h] * LOG2E : -INFINITY, l = a.sink ? 1.f : 0.f, pend = 1.f;
            bool has_pend = false;
            const int lo = first_key(a, pos), warp_lo = rec.w + r0, warp_hi = rec.w + min(nq - 1, r0 + 31), lo_hi = first_key(a, max(warp_hi, 0));
            const bool any_rows = r0 < nq, all_rows = r0 + 32 <= nq;
            float* ps = reinterpret_cast<float*>(smem_raw + pen_off) + warp * 4 * PEN_LD;
            const float* pl = ps + ((31 - lane) & 3) * PEN_LD + ((31 - lane) & ~3);          // this lane's copy, column 0
            float pn[3];
            auto pen_fetch = [&](int it) {
                const float* p = a.penalty + (size_t)h * a.n_penalty;
                const int dist = warp_lo + 31 - page_at(it) * 64 - lane;
#pragma unroll
                for (int k = 0; k < 3; k++) pn[k] = p[min(max(dist - 32 * k, 0), a.n_penalty - 1)];
            };
            if (PEN && nx > 0) pen_fetch(0);
            for (int it = 0; it < nx; it++) {
                const int j0 = page_at(it) * 64;
                const uint32_t t_s = t_lane + 128 * x + (it & 1) * 64;
                if (PEN) {
                    __syncwarp();                            // the page before is read
#pragma unroll
                    for (int k = 0; k < 3; k++)
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (lane + 32 * k >= c) ps[c * PEN_LD + lane + 32 * k - c] = -LOG2E * pn[k];
                    __syncwarp();
                    if (it + 1 < nx) pen_fetch(it + 1);
                }
                wait_lim(s_full(x, it), (uint32_t)(it >> 1) & 1u, fail);
                tc_fence_after();
                auto scale_o = [&](float cf) {
                    if (it > 0) { wait_lim(o_done(x, it - 1), (uint32_t)((it - 1) >> 1) & 1u, fail); tc_fence_after(); }
#pragma unroll 1
                    for (int c = 0; c < dv; c += 32) {
                        uint32_t v[32];
                        tc_ld32(t_o + c, v);
#pragma unroll
                        for (int k = 0; k < 32; k++) v[k] = __float_as_uint(__uint_as_float(v[k]) * cf);
                        tc_st32(t_o + c, v);
                    }
                };
                if (!SIG && __any_sync(0xffffffffu, has_pend)) scale_o(has_pend ? pend : 1.f);
                if (has_pend) { l *= pend; has_pend = false; }
                // every key of the page is visible to every row of the warp: behind its first row, and its last row still sees it
                const bool full = all_rows && j0 + 63 <= warp_lo && (j0 >= lo_hi || j0 + 63 < a.keep_first);
                const bool none = !any_rows || j0 > warp_hi;
                uint32_t pk[32];
                // one sweep over the row's 64 scores: maximum and / or weights against the reference mu
                auto sweep = [&](auto do_max, auto do_exp, float mu, float& mx_out, float& ls_out) {
                    constexpr bool DM = decltype(do_max)::value, DE = decltype(do_exp)::value;
                    uint32_t buf[2][32];
                    tc_ld32_nowait(t_s, buf[0]);
                    tc_ld32_nowait(t_s + 32, buf[1]);
                    tc_wait_ld();
                    tc_reg_fence32(buf[0]);
                    tc_reg_fence32(buf[1]);
                    float mx0 = -INFINITY, mx1 = -INFINITY, sA0 = 0.f, sA1 = 0.f, sB0 = 0.f, sB1 = 0.f;
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        float v[32];
#pragma unroll
                        for (int k = 0; k < 32; k++) v[k] = __uint_as_float(buf[c][k]);
                        if (PEN) {
#pragma unroll
                            for (int k = 0; k < 32; k += 4) {
                                const float4 pv = *reinterpret_cast<const float4*>(pl + 32 * c + k);
                                fma2(v[k], v[k + 1], v[k], v[k + 1], scale2, scale2, pv.x, pv.y);
                                fma2(v[k + 2], v[k + 3], v[k + 2], v[k + 3], scale2, scale2, pv.z, pv.w);
                            }
                        }
                        if (!full) {
#pragma unroll
                            for (int k = 0; k < 32; k++) {
                                const int j = j0 + 32 * c + k;
                                if (!(row_ok && j <= pos && (j >= lo || j < a.keep_first))) v[k] = -INFINITY;
                            }
                        }
                        if (DM) {
#pragma unroll
                            for (int k = 0; k < 32; k += 4) { mx0 = max3(mx0, v[k], v[k + 1]); mx1 = max3(mx1, v[k + 2], v[k + 3]); }
                        }
                        if (DE) {
#pragma unroll
                            for (int k = 0; k < 32; k += 2) {
                                float p0, p1;
                                if (SIG) {                   // 1 / (1 + 2^-(score + bias)); a masked key gives 1 / inf = 0
                                    if (PEN) add2(p0, p1, -v[k], -v[k + 1], -sb2, -sb2);
                                    else fma2(p0, p1, v[k], v[k + 1], -scale2, -scale2, -sb2, -sb2);
                                    add2(p0, p1, ex2f(p0), ex2f(p1), 1.f, 1.f);
                                    p0 = rcpf(p0); p1 = rcpf(p1);
                                } else {
                                    if (PEN) add2(p0, p1, v[k], v[k + 1], -mu, -mu);
                                    else fma2(p0, p1, v[k], v[k + 1], scale2, scale2, -mu, -mu);
                                    p0 = ex2f(p0); p1 = ex2f(p1);
                                    if (k & 2) add2(sA0, sA1, sA0, sA1, p0, p1); else add2(sB0, sB1, sB0, sB1, p0, p1);
                                }
                                pk[16 * c + k / 2] = pack_bf16(p0, p1);
                            }
                        }
                    }
                    if (DM) mx_out = fmaxf(mx0, mx1) * (PEN ? 1.f : scale2);
                    if (DE) ls_out = (sA0 + sA1) + (sB0 + sB1);
                };
                float mx = -INFINITY, ls = 0.f;
                if (none) {
#pragma unroll
                    for (int k = 0; k < 32; k++) pk[k] = 0u;
                } else if (SIG) {
                    sweep(std::false_type{}, std::true_type{}, 0.f, mx, ls);
                } else {
                    bool redo = true;
                    if (it > 0 || a.sink) {
                        sweep(std::true_type{}, std::true_type{}, m == -INFINITY ? 0.f : m, mx, ls);
                        redo = m == -INFINITY ? mx != -INFINITY : mx - m > 64.f;
                    } else {
                        sweep(std::true_type{}, std::false_type{}, 0.f, mx, ls);
                    }
                    if (__any_sync(0xffffffffu, redo)) {
                        float corr = 1.f;
                        if (redo) { corr = m == -INFINITY ? 0.f : ex2f(m - mx); m = mx; }
                        if (it > 0) scale_o(corr);
                        l *= corr;
                        sweep(std::false_type{}, std::true_type{}, m == -INFINITY ? 0.f : m, mx, ls);
                    }
                    l += ls;
                    const float grow = mx - m;               // NaN (no key yet) compares false
                    if (grow > 8.f) { pend = ex2f(-grow); has_pend = true; m = mx; }
                }
                tc_st32(t_s, pk);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(sm_done(x, it));
            }
            // ---- epilogue: O / l, gates
            if (nx > 0) {
                if (nx > 1) wait_lim(o_done(x, nx - 2), (uint32_t)((nx - 2) >> 1) & 1u, fail);
                wait_lim(o_done(x, nx - 1), (uint32_t)((nx - 1) >> 1) & 1u, fail);
                tc_fence_after();
            }
            if (mine && nx > 0 && any_rows) {
                // 64 columns at a time (32 with one box of keys): row-wise out of TMEM into the warp's quarter of the (consumed) Q block, swizzled
                // by 16-byte pieces, and from there in whole rows to memory, so that gates are read and outputs written in full lines
                float inv = (a.gate && row_ok ? a.gate[((size_t)rec.x + i) * a.n_heads + h] : 1.f) * (a.out_scale != 0.f ? a.out_scale : 1.f);
                if (!SIG) inv = l > 0.f ? inv / l : 0.f;
                if (*fail) inv = __int_as_float(0x7fc00000);
                const uint32_t ob = sQ + x * q_bytes + wq * (q_bytes / 4);
                const int cols = 32 * kb;
                const bool quads = a.ld_elem_gate % 4 == 0 && ((uintptr_t)a.elem_gate & 15) == 0;
                for (int c0 = 0; c0 < dv; c0 += cols) {
                    const int nc = min(cols, dv - c0);
                    __syncwarp();                            // the round before is read
#pragma unroll 1
                    for (int c = 0; c < nc; c += 16) {
                        uint32_t v[16];
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                                     "tcgen05.wait::ld.sync.aligned;"
                                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                                       "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(t_o + c0 + c));
#pragma unroll
                        for (int k = 0; k < 16; k += 4) {
                            const uint32_t dst = ob + lane * cols * 4 + ((((c + k) >> 2) ^ (lane & 7)) << 4);
                            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "f"(__uint_as_float(v[k]) * inv), "f"(__uint_as_float(v[k + 1]) * inv),
                                         "f"(__uint_as_float(v[k + 2]) * inv), "f"(__uint_as_float(v[k + 3]) * inv) : "memory");
                        }
                    }
                    __syncwarp();
                    const int per = nc / 4;                  // 16-byte pieces per row
                    for (int e = lane; e < 32 * per; e += 32) {
                        const int rr = e / per, c = (e - rr * per) * 4;
                        if (r0 + rr >= nq) break;
                        float4 y;
                        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(y.x), "=f"(y.y), "=f"(y.z), "=f"(y.w)
                                     : "r"(ob + rr * cols * 4 + (((c >> 2) ^ (rr & 7)) << 4)));
                        const size_t row = (size_t)rec.x + r0 + rr, col = (size_t)h * dv + c0 + c;
                        if (a.elem_gate) {
                            const float* eg = a.elem_gate + row * a.ld_elem_gate + col;
                            const float4 t = quads ? *reinterpret_cast<const float4*>(eg) : make_float4(eg[0], eg[1], eg[2], eg[3]);
                            y.x *= 1.0f / (1.0f + expf(-t.x)); y.y *= 1.0f / (1.0f + expf(-t.y));
                            y.z *= 1.0f / (1.0f + expf(-t.z)); y.w *= 1.0f / (1.0f + expf(-t.w));
                        }
                        *reinterpret_cast<uint2*>((bf16*)a.out + row * a.ld_out + col) = make_uint2(pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
                    }
                }
            }
        }
        ta = tb;
        tc_fence_before();
        __syncthreads();                                     // the pass is over for every warp: nothing is in flight, O is read
        if (ta < t_end) {
            if (warp == W_MMA && lane == 0) {
                const int n_bars = 1 + 4 * ST + 6 * NX;
                for (int b = 0; b < n_bars; b++) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bars + 8u * b) : "memory");
                init_bars();
            }
            __syncthreads();
        }
        tc_fence_after();
    }
    if (warp == W_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(C::TMEM) : "memory");
}

template <int NX, bool PEN, bool SIG>
int launch(const p3_attn_window_args* a, const WinMaps& tm, int n_hc, int n_tc, cudaStream_t st) {
    const size_t bytes = WinCfg<NX>::smem((a->dim + 63) / 64, (a->vdim + 63) / 64);
    static P3DevFlags flags; bool& set = flags.cur();
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(attn_window_prefill_tc_kernel<NX, PEN, SIG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)WinCfg<NX>::smem(2, 2));
        P3_CHECK_ARG(e == cudaSuccess, "attn_window_prefill: shared memory attribute: %s", cudaGetErrorString(e));
        set = true;
    }
    const int64_t grid = (int64_t)((a->n_tiles + n_tc - 1) / n_tc) * (a->n_heads / n_hc);
    p3_launch_pdl(attn_window_prefill_tc_kernel<NX, PEN, SIG>, dim3((unsigned)grid), dim3(WinCfg<NX>::THREADS), bytes, st, tm, *a, n_hc, n_tc);
    return 0;
}
}  // namespace

// whole boxes of 16-byte pieces everywhere, and a positive scale (maxima are taken before it is applied)
bool attn_window_tc_ok(const p3_attn_window_args* a) {
    return !a->act_f32 && a->dim % 16 == 0 && a->vdim % 16 == 0 && a->dim <= 128 && a->vdim <= 128 && a->ld_q % 8 == 0 && a->ld_out % 8 == 0 &&
           a->v_ld % 8 == 0 && (((uintptr_t)a->q | (uintptr_t)a->out | (uintptr_t)a->k_pool | (uintptr_t)a->v_pool) & 15) == 0 && a->scale > 0.f;
}

int launch_attn_window_tc(const p3_attn_window_args* a, cudaStream_t st) {
    WinMaps tm;
    const int v_ld = a->v_ld > 0 ? a->v_ld : a->vdim;
    // rows: an upper bound, pages are addressed through the block table
    CUresult r = tc_encode_2d(&tm.k, a->k_pool, (int64_t)1 << 31, a->dim, a->dim, 64);
    if (r == CUDA_SUCCESS) r = tc_encode_2d(&tm.v, a->v_pool, (int64_t)1 << 31, a->vdim, v_ld, 64);
    P3_CHECK_ARG(r == CUDA_SUCCESS, "attn_window_prefill: cuTensorMapEncodeTiled failed (%d)", (int)r);
    const int rep = a->n_heads / a->n_kv;
    int n_hc = rep % 4 == 0 ? 4 : rep % 2 == 0 ? 2 : 1, n_tc = 4 / n_hc;
    auto ctas = [&]() { return (int64_t)((a->n_tiles + n_tc - 1) / n_tc) * (a->n_heads / n_hc); };
    while (ctas() < 148 && n_tc * n_hc > 1) { if (n_tc > 1) n_tc /= 2; else n_hc /= 2; }
#define GO(NX) (a->sig_bias ? (a->penalty ? launch<NX, true, true>(a, tm, n_hc, n_tc, st) : launch<NX, false, true>(a, tm, n_hc, n_tc, st)) \
                            : (a->penalty ? launch<NX, true, false>(a, tm, n_hc, n_tc, st) : launch<NX, false, false>(a, tm, n_hc, n_tc, st)))
    return n_hc * n_tc > 2 ? GO(2) : GO(1);
#undef GO
}
