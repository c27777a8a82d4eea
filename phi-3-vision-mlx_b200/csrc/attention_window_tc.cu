// Windowed / chunked / gated prefill attention over the page pools (the contract of attention_window.cu) on the 5th-gen tensor cores, for
// bf16 with key sizes and value sizes that are multiples of 16 up to 128.
//
// One CTA = 128 query rows against the pages of one sequence and K/V head, in two halves of 64 rows; a half is one tile record x one query
// head. The halves are n_hc query heads of one group x n_tc neighbouring tile records (n_hc n_tc <= 2), so that grouped-query heads share the
// K/V pages that a CTA stages. Records of different sequences in one CTA take a pass each.
//   warps 0-7:  softmax. A query row (TMEM lane) belongs to two threads, one per 32 of a page's 64 keys: sixteen such warps on an SM (two CTAs)
//               hide one another's trips to TMEM and barriers; with a thread per row and eight warps a page of 256 rows took 2200 cycles, 1500
//               of them arithmetic. S is double buffered in TMEM, so the scores of the next two pages are computed while this one is swept; P
//               goes back over the consumed S columns and is the A operand of P.V straight from TMEM. P is formed against the running
//               reference maximum of the pages before (base-2 domain; the sink is the first reference, with a denominator of 1); the page's own
//               maximum is found in the same sweep and shared by the row's two threads. O and l are rescaled when the reference falls 2^8
//               behind, and the page is swept again when it falls 2^64 behind or there was none. Scores, penalties, weights and all sums are
//               fp32, two per instruction where that goes.
//               A weight is two bf16 numbers, its upper 16 bits and what they leave, and takes part in two products: with one rounded
//               number the error against 64 bits was 2.4e-3 of the outputs (4 x 2048 tokens, 16 heads of 128 over 4, window 1024), above
//               the 2.0e-3 of weights against each page's exact maximum, which took 142 us to form; with two it is 1.7e-3 in 119 us
//               (108 with one; 298 on mma.sync).
//   warp 8:     TMA producer, one page = 64-column SWIZZLE_128B boxes of K and of V, two mbarrier rings
//   warp 9:     MMA issuer: O += P(j) V(j), then S(j + 2) = Q K(j + 2)^T into the columns P(j) left
// Q rows are copied by the softmax warps (rows beyond a tile's end are not read). The penalties of a warp's 63 distances to its keys are staged
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
__device__ __forceinline__ void ld16(uint32_t t, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                   "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(t));
}
__device__ __forceinline__ void st16(uint32_t t, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
                 "tcgen05.wait::st.sync.aligned;"
                 ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
                   "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
// first position that a query at `pos` sees (kept first tokens aside), as in attention_window.cu
__device__ __forceinline__ int first_key(const p3_attn_window_args& a, int pos) {
    int lo = 0;
    if (a.window > 0) lo = max(lo, pos - a.window + 1);
    if (a.chunk > 0) lo = max(lo, pos - pos % a.chunk);
    return lo;
}

struct WinMaps { CUtensorMap k, v; };
// penalties of a warp's 32 rows against its 32 keys: entry t = distance (first row + 31 - t) to the warp's first key, so that a row's columns are
// neighbours; four copies shifted by 0 .. 3 entries let every lane read 16-byte pieces, and their pitch keeps a quarter-warp on different banks
constexpr int PEN_LD = 72;

constexpr int ST = 2;                                        // pages in flight
constexpr int W_TMA = 8, W_MMA = 9, THREADS = 320;
constexpr int TMEM = 256, O_COL = 128;                       // S(buffer) at 64 buffer, O at O_COL
constexpr int N_BARS = 1 + 4 * ST + 6;
// Q of up to 2 boxes x 128 rows, K and V pages of up to 2 boxes, penalty slices, row exchange, barriers
size_t win_smem(int kb, int vb) { return (size_t)kb * 2 * BOX + (size_t)ST * (kb + vb) * BOX + 8 * 4 * PEN_LD * 4 + 4 * 128 * 4 + 256 + 1024; }

template <bool PEN, bool SIG>
__global__ void __launch_bounds__(THREADS, 2)
attn_window_prefill_tc_kernel(const __grid_constant__ WinMaps tm, p3_attn_window_args a, int n_hc, int n_tc) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ int fail_s;
    __shared__ uint32_t tmem_s;
    volatile int* fail = &fail_s;
    const int d = a.dim, dv = a.vdim, kb = (d + 63) / 64, vb = (dv + 63) / 64, rep = a.n_heads / a.n_kv;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    const uint32_t sQ = base, q_bytes = (uint32_t)kb * 2 * BOX, sK = sQ + q_bytes, sV = sK + ST * kb * BOX;
    const uint32_t pen_off = sV + ST * vb * BOX - raw, ex_off = pen_off + 8 * 4 * PEN_LD * 4, bars = raw + ex_off + 4 * 128 * 4;
    const uint32_t q_full = bars;
    auto k_full = [&](int s) { return bars + 8u * (1 + s); };
    auto k_empty = [&](int s) { return bars + 8u * (1 + ST + s); };
    auto v_full = [&](int s) { return bars + 8u * (1 + 2 * ST + s); };
    auto v_empty = [&](int s) { return bars + 8u * (1 + 3 * ST + s); };
    auto s_full = [&](int j) { return bars + 8u * (1 + 4 * ST + (j & 1)); };
    auto sm_done = [&](int j) { return bars + 8u * (3 + 4 * ST + (j & 1)); };
    auto o_done = [&](int j) { return bars + 8u * (5 + 4 * ST + (j & 1)); };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hgs = a.n_heads / n_hc, groups = (a.n_tiles + n_tc - 1) / n_tc;
    const int hg = blockIdx.x % hgs, grp = groups - 1 - blockIdx.x / hgs;      // later tiles (more keys) first
    const int h0 = hg * n_hc, g = h0 / rep;

    auto init_bars = [&]() {
        mbar_init(q_full, 8);
        for (int s = 0; s < ST; s++) { mbar_init(k_full(s), 1); mbar_init(k_empty(s), 1); mbar_init(v_full(s), 1); mbar_init(v_empty(s), 1); }
        for (int j = 0; j < 2; j++) { mbar_init(s_full(j), 1); mbar_init(o_done(j), 1); mbar_init(sm_done(j), 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    };
    if (warp == W_TMA && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tm.k)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tm.v)) : "memory");
    }
    if (warp == W_MMA) {
        if (lane == 0) { init_bars(); fail_s = 0; }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "n"(TMEM) : "memory");
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
        int tb = ta, first = INT_MAX, last = 0;
        for (; tb < t_end; tb++) {
            const int4 r = recs[tb];
            if (r.z != slot) break;
            first = min(first, first_key(a, r.w));
            last = max(last, r.w + r.y - 1);
        }
        // pages: those of the kept first tokens before the window's pages, then from the first visible key to the last row's position
        const int lo_pg = first / 64, n_keep = min((a.keep_first + 63) / 64, lo_pg);
        auto page_at = [&](int it) { return it < n_keep ? it : lo_pg + it - n_keep; };
        const int n = n_keep + last / 64 - lo_pg + 1;
        const int32_t* bt = a.block_table + (size_t)slot * a.bt_stride;

        if (warp == W_TMA) {
            if (lane == 0) {
                for (int it = -1; it < n; it++) {            // K one page ahead of V: its stage comes free earlier
                    if (it + 1 < n) {
                        const int st = (it + 1) % ST, row = (bt[page_at(it + 1)] * a.n_kv + g) * 64;
                        wait_lim(k_empty(st), ((uint32_t)((it + 1) / ST) & 1u) ^ 1u, fail);
                        mbar_expect_tx(k_full(st), kb * BOX);
                        for (int b = 0; b < kb; b++) tma_load_2d(sK + (st * kb + b) * BOX, &tm.k, k_full(st), 64 * b, row);
                    }
                    if (it >= 0) {
                        const int st = it % ST, row = (bt[page_at(it)] * a.n_kv + g) * 64;
                        wait_lim(v_empty(st), ((uint32_t)(it / ST) & 1u) ^ 1u, fail);
                        mbar_expect_tx(v_full(st), vb * BOX);
                        for (int b = 0; b < vb; b++) tma_load_2d(sV + (st * vb + b) * BOX, &tm.v, v_full(st), 64 * b, row);
                    }
                }
                for (int it = max(0, n - ST); it < n; it++) {          // every release has arrived before the barriers may be set up anew
                    wait_lim(k_empty(it % ST), (uint32_t)(it / ST) & 1u, fail);
                    wait_lim(v_empty(it % ST), (uint32_t)(it / ST) & 1u, fail);
                }
            }
        } else if (warp >= W_MMA) {
            // MMA issuer (whole warp converged, one elected lane issues)
            const int ks = d / 16;
            constexpr uint32_t ID = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
            const uint32_t id_qk = ID | ((64u >> 3) << 17), id_pv = ID | (1u << 16) | ((uint32_t)(dv >> 3) << 17);
            // operand descriptors; what changes is added to their address fields (16-byte units)
            const uint64_t qd = umma_desc_sw128(sQ), kd0 = umma_desc_sw128(sK), vd0 = umma_desc_mn_sw128(sV, BOX, 1024);
            wait_lim(q_full, 0, fail);
            for (int t = 0; t < n + 2; t++) {
                const int j = t - 2;
                if (j >= 0) {                                // O += P(j) V(j)
                    wait_lim(v_full(j % ST), (uint32_t)(j / ST) & 1u, fail);
                    wait_lim(sm_done(j), (uint32_t)(j >> 1) & 1u, fail);
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t p_col = tmem + (j & 1) * 64;
                        const uint64_t vd = vd0 + (uint32_t)((j % ST) * vb * (BOX >> 4));
#pragma unroll
                        for (int kk = 0; kk < 8; kk++)       // P of keys 0-31 in columns 0-15, of keys 32-63 in columns 32-47; the rest 16 columns on
                            tc_mma_bf16_ts(tmem + O_COL, p_col + 16 * (kk >> 2) + 32 * ((kk >> 1) & 1) + 8 * (kk & 1), vd + (kk & 3) * (16 * 128 >> 4), id_pv,
                                           kk ? 1u : (uint32_t)j);
                        tc_commit(o_done(j));
                        tc_commit(v_empty(j % ST));
                    }
                    __syncwarp();
                }
                if (t < n) {                                 // S(t) = Q K(t)^T, behind the P.V that reads the same columns
                    wait_lim(k_full(t % ST), (uint32_t)(t / ST) & 1u, fail);
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t dst = tmem + (t & 1) * 64;
                        const uint64_t kd = kd0 + (uint32_t)((t % ST) * kb * (BOX >> 4));
                        tc_mma_bf16(dst, qd, kd, id_qk, 0u);
#pragma unroll
                        for (int kk = 1; kk < 8; kk++)
                            if (kk < ks) tc_mma_bf16(dst, qd + ((kk >> 2) * (2 * BOX >> 4) + 2 * (kk & 3)), kd + ((kk >> 2) * (BOX >> 4) + 2 * (kk & 3)), id_qk, 1u);
                        tc_commit(s_full(t));
                        tc_commit(k_empty(t % ST));
                    }
                    __syncwarp();
                }
            }
        } else {
            // ---- softmax: warps wq and wq + 4 share 32 rows of one half (one record, one head); `hf`: which 32 keys of a page
            const int wq = warp & 3, hf = warp >> 2, u = wq >> 1, rec_i = grp * n_tc + u / n_hc, h = h0 + u % n_hc;
            const bool mine = rec_i >= ta && rec_i < tb;
            const int4 rec = recs[mine ? rec_i : ta];
            const int r0 = (wq & 1) * 32, i = r0 + lane, nq = mine ? rec.y : 0, pos = rec.w + i;
            const bool row_ok = i < nq;
            {   // half of the 32 query rows -> shared memory, swizzled as the UMMA reads them
                const bf16* q = (const bf16*)a.q + (size_t)rec.x * a.ld_q + (size_t)h * d;
                const int sh = kb == 2 ? 4 : 3, c = lane & ((1 << sh) - 1);          // 16 or 8 lanes per row
                const int per = 32 >> sh;                                            // rows per step of the warp
                const bool in = 8 * c < d;
                const uint32_t box = sQ + (c >> 3) * 2 * BOX;
                {
                    const int b = 16 * hf;
                    uint4 v[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int rr = r0 + b + k * per + (lane >> sh);
                        v[k] = in && k * per < 16 && rr < nq ? *reinterpret_cast<const uint4*>(q + (size_t)rr * a.ld_q + 8 * c) : make_uint4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int lr = (wq >> 1) * 64 + r0 + b + k * per + (lane >> sh);
                        const uint32_t dst = box + lr * 128 + (((c & 7) ^ (lr & 7)) << 4);
                        if (k * per < 16) asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v[k].x), "r"(v[k].y), "r"(v[k].z), "r"(v[k].w) : "memory");
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(q_full);
            }
            const uint32_t t_lane = tmem + ((uint32_t)(wq * 32) << 16), t_o = t_lane + O_COL;
            float* ex = reinterpret_cast<float*>(smem_raw + ex_off) + wq * 32 + lane;       // [page parity][half] x 128 rows
            auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + wq) : "memory"); };
            const float scale2 = a.scale * LOG2E, sb2 = SIG ? a.sig_bias[h] * LOG2E : 0.f;
            float m = a.sink ? a.sink[h] * LOG2E : -INFINITY, l = a.sink && hf == 0 ? 1.f : 0.f, pend = 1.f;
            bool has_pend = false;
            const int lo = first_key(a, pos), warp_lo = rec.w + r0, warp_hi = rec.w + min(nq - 1, r0 + 31), lo_hi = first_key(a, max(warp_hi, 0));
            const bool any_rows = r0 < nq, all_rows = r0 + 32 <= nq;
            float* ps = reinterpret_cast<float*>(smem_raw + pen_off) + warp * 4 * PEN_LD;
            const float* pl = ps + ((31 - lane) & 3) * PEN_LD + ((31 - lane) & ~3);          // this lane's copy, column 0
            float pn[2];
            auto pen_fetch = [&](int it) {
                const float* p = a.penalty + (size_t)h * a.n_penalty;
                const int dist = warp_lo + 31 - page_at(it) * 64 - 32 * hf - lane;
#pragma unroll
                for (int k = 0; k < 2; k++) pn[k] = p[min(max(dist - 32 * k, 0), a.n_penalty - 1)];
            };
            if (PEN) pen_fetch(0);
            for (int it = 0; it < n; it++) {
                const int j0 = page_at(it) * 64 + 32 * hf;   // first of this thread's keys
                const uint32_t t_s = t_lane + (it & 1) * 64 + 32 * hf;
                if (PEN) {
                    __syncwarp();                            // the page before is read
#pragma unroll
                    for (int k = 0; k < 2; k++)
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (lane + 32 * k >= c) ps[c * PEN_LD + lane + 32 * k - c] = -LOG2E * pn[k];
                    __syncwarp();
                    if (it + 1 < n) pen_fetch(it + 1);
                }
                wait_lim(s_full(it), (uint32_t)(it >> 1) & 1u, fail);
                tc_fence_after();
                auto scale_o = [&](float cf) {               // this thread's half of the row: every other 16 columns
                    if (it > 0) { wait_lim(o_done(it - 1), (uint32_t)((it - 1) >> 1) & 1u, fail); tc_fence_after(); }
#pragma unroll 1
                    for (int c = 16 * hf; c < dv; c += 32) {
                        uint32_t v[16];
                        ld16(t_o + c, v);
#pragma unroll
                        for (int k = 0; k < 16; k++) v[k] = __float_as_uint(__uint_as_float(v[k]) * cf);
                        st16(t_o + c, v);
                    }
                };
                if (!SIG && __any_sync(0xffffffffu, has_pend)) scale_o(has_pend ? pend : 1.f);
                if (has_pend) { l *= pend; has_pend = false; }
                // every key of the half page is visible to every row of the warp: behind its first row, and its last row still sees it
                const bool full = all_rows && j0 + 31 <= warp_lo && (j0 >= lo_hi || j0 + 31 < a.keep_first);
                const bool none = !any_rows || j0 > warp_hi;
                uint32_t pk[32];                             // weights: upper 16 bits, then what they leave
                // one sweep over 32 scores of the row: maximum and / or weights against the reference mu
                auto sweep = [&](auto do_max, auto do_exp, float mu, float& mx_out, float& ls_out) {
                    constexpr bool DM = decltype(do_max)::value, DE = decltype(do_exp)::value;
                    uint32_t buf[32];
                    tc_ld32_nowait(t_s, buf);
                    tc_wait_ld();
                    tc_reg_fence32(buf);
                    float mx0 = -INFINITY, mx1 = -INFINITY, sA0 = 0.f, sA1 = 0.f, sB0 = 0.f, sB1 = 0.f;
                    {
                        float v[32];
#pragma unroll
                        for (int k = 0; k < 32; k++) v[k] = __uint_as_float(buf[k]);
                        if (PEN) {
#pragma unroll
                            for (int k = 0; k < 32; k += 4) {
                                const float4 pv = *reinterpret_cast<const float4*>(pl + k);
                                fma2(v[k], v[k + 1], v[k], v[k + 1], scale2, scale2, pv.x, pv.y);
                                fma2(v[k + 2], v[k + 3], v[k + 2], v[k + 3], scale2, scale2, pv.z, pv.w);
                            }
                        }
                        if (!full) {
#pragma unroll
                            for (int k = 0; k < 32; k++) {
                                const int j = j0 + k;
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
                                pk[k / 2] = __byte_perm(__float_as_uint(p0), __float_as_uint(p1), 0x7632);
                                float r0, r1;
                                fma2(r0, r1, __uint_as_float(__float_as_uint(p0) & 0xffff0000u), __uint_as_float(__float_as_uint(p1) & 0xffff0000u), -1.f, -1.f, p0, p1);
                                pk[16 + k / 2] = pack_bf16(r0, r1);
                            }
                        }
                    }
                    if (DM) mx_out = fmaxf(mx0, mx1) * (PEN ? 1.f : scale2);
                    if (DE) ls_out = (sA0 + sA1) + (sB0 + sB1);
                };
                float mx = -INFINITY, ls = 0.f;
                const bool known = it > 0 || a.sink;         // there is a reference to form weights against
                if (none) {
#pragma unroll
                    for (int k = 0; k < 32; k++) pk[k] = 0u;
                } else if (SIG) sweep(std::false_type{}, std::true_type{}, 0.f, mx, ls);
                else if (known) sweep(std::true_type{}, std::true_type{}, m == -INFINITY ? 0.f : m, mx, ls);
                else sweep(std::true_type{}, std::false_type{}, 0.f, mx, ls);
                if (!SIG) {
                    float* e = ex + (it & 1) * 256;          // the row's maximum over the page: with the thread of the other 32 keys
                    e[128 * hf] = mx;
                    pair_sync();
                    mx = fmaxf(mx, e[128 * (hf ^ 1)]);
                    const bool redo = !known || (m == -INFINITY ? mx != -INFINITY : mx - m > 64.f);
                    if (__any_sync(0xffffffffu, redo)) {     // the same for both warps: they hold the same rows
                        float corr = 1.f, unused;
                        if (redo) { corr = m == -INFINITY ? 0.f : ex2f(m - mx); m = mx; }
                        if (it > 0) scale_o(corr);
                        l *= corr;
                        if (!none) sweep(std::false_type{}, std::true_type{}, m == -INFINITY ? 0.f : m, unused, ls);
                    }
                    l += ls;
                    const float grow = mx - m;               // NaN (no key yet) compares false
                    if (grow > 8.f) { pend = ex2f(-grow); has_pend = true; m = mx; }
                }
                st16(t_s, pk);
                st16(t_s + 16, pk + 16);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(sm_done(it));
            }
            // ---- epilogue: O / l, gates
            if (n > 1) wait_lim(o_done(n - 2), (uint32_t)((n - 2) >> 1) & 1u, fail);
            wait_lim(o_done(n - 1), (uint32_t)((n - 1) >> 1) & 1u, fail);
            tc_fence_after();
            if (!SIG) {                                      // the denominator: both threads' parts (the sink's 1 is in the first one's)
                float* e = ex + (n & 1) * 256;
                e[128 * hf] = l;
                pair_sync();
                l += e[128 * (hf ^ 1)];
            }
            if (mine && any_rows) {
                // a warp writes half of the columns, 32 at a time (16 with one box of keys): row-wise out of TMEM into its part of the (consumed)
                // Q block, swizzled by 16-byte pieces, and from there in rows to memory, so that gates and outputs move in whole sectors
                float inv = (a.gate && row_ok ? a.gate[((size_t)rec.x + i) * a.n_heads + h] : 1.f) * (a.out_scale != 0.f ? a.out_scale : 1.f);
                if (!SIG) inv = l > 0.f ? inv / l : 0.f;
                if (*fail) inv = __int_as_float(0x7fc00000);
                const uint32_t ob = sQ + warp * (q_bytes / 8);
                const int cols = 16 * kb, mid = (dv / 16 + 1) / 2 * 16, c_end = hf ? dv : mid;
                const bool quads = a.ld_elem_gate % 4 == 0 && ((uintptr_t)a.elem_gate & 15) == 0;
                auto piece = [&](int row, int pc) { return ob + row * cols * 4 + ((pc ^ (kb == 2 ? row & 7 : (row >> 1) & 3)) << 4); };
                for (int c0 = hf ? mid : 0; c0 < c_end; c0 += cols) {
                    const int nc = min(cols, c_end - c0);
                    __syncwarp();                            // the round before is read
#pragma unroll 1
                    for (int c = 0; c < nc; c += 16) {
                        uint32_t v[16];
                        ld16(t_o + c0 + c, v);
#pragma unroll
                        for (int k = 0; k < 16; k += 4)
                            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(piece(lane, (c + k) >> 2)), "f"(__uint_as_float(v[k]) * inv),
                                         "f"(__uint_as_float(v[k + 1]) * inv), "f"(__uint_as_float(v[k + 2]) * inv), "f"(__uint_as_float(v[k + 3]) * inv) : "memory");
                    }
                    __syncwarp();
                    const int sh = kb == 2 ? 3 : 2, c = (lane & ((1 << sh) - 1)) * 4, per = 32 >> sh;    // 8 or 4 lanes per row
                    const size_t col = (size_t)h * dv + c0 + c;
                    for (int b = 0; b < 32; b += 4 * per) {  // four rows (and their gates) in flight per lane
                        float4 y[4], t[4];
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int rr = b + k * per + (lane >> sh);
                            const bool in = c < nc && r0 + rr < nq;
                            t[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (a.elem_gate && in) {
                                const float* eg = a.elem_gate + ((size_t)rec.x + r0 + rr) * a.ld_elem_gate + col;
                                t[k] = quads ? *reinterpret_cast<const float4*>(eg) : make_float4(eg[0], eg[1], eg[2], eg[3]);
                            }
                            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(y[k].x), "=f"(y[k].y), "=f"(y[k].z), "=f"(y[k].w)
                                         : "r"(piece(rr, c >> 2)));
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int rr = b + k * per + (lane >> sh);
                            if (a.elem_gate) {
                                y[k].x *= rcpf(1.0f + ex2f(-LOG2E * t[k].x)); y[k].y *= rcpf(1.0f + ex2f(-LOG2E * t[k].y));
                                y[k].z *= rcpf(1.0f + ex2f(-LOG2E * t[k].z)); y[k].w *= rcpf(1.0f + ex2f(-LOG2E * t[k].w));
                            }
                            if (c < nc && r0 + rr < nq)
                                *reinterpret_cast<uint2*>((bf16*)a.out + ((size_t)rec.x + r0 + rr) * a.ld_out + col) = make_uint2(pack_bf16(y[k].x, y[k].y), pack_bf16(y[k].z, y[k].w));
                        }
                    }
                }
            }
        }
        ta = tb;
        tc_fence_before();
        __syncthreads();                                     // the pass is over for every warp: nothing is in flight, O is read
        if (ta < t_end) {
            if (warp == W_MMA && lane == 0) {
                for (int b = 0; b < N_BARS; b++) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bars + 8u * b) : "memory");
                init_bars();
            }
            __syncthreads();
        }
        tc_fence_after();
    }
    if (warp == W_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM) : "memory");
}

template <bool PEN, bool SIG>
int launch(const p3_attn_window_args* a, const WinMaps& tm, int n_hc, int n_tc, cudaStream_t st) {
    const size_t bytes = win_smem((a->dim + 63) / 64, (a->vdim + 63) / 64);
    static P3DevFlags flags; bool& set = flags.cur();
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(attn_window_prefill_tc_kernel<PEN, SIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)win_smem(2, 2));
        P3_CHECK_ARG(e == cudaSuccess, "attn_window_prefill: shared memory attribute: %s", cudaGetErrorString(e));
        set = true;
    }
    const int64_t grid = (int64_t)((a->n_tiles + n_tc - 1) / n_tc) * (a->n_heads / n_hc);
    p3_launch_pdl(attn_window_prefill_tc_kernel<PEN, SIG>, dim3((unsigned)grid), dim3(THREADS), bytes, st, tm, *a, n_hc, n_tc);
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
    // both halves of a CTA in use unless that would leave SMs without one (a half alone takes about as long as two)
    int n_hc = (a->n_heads / a->n_kv) % 2 == 0 ? 2 : 1, n_tc = 2 / n_hc;
    if ((int64_t)((a->n_tiles + n_tc - 1) / n_tc) * (a->n_heads / n_hc) < 148) n_hc = n_tc = 1;
    if (a->sig_bias) return a->penalty ? launch<true, true>(a, tm, n_hc, n_tc, st) : launch<false, true>(a, tm, n_hc, n_tc, st);
    return a->penalty ? launch<true, false>(a, tm, n_hc, n_tc, st) : launch<false, false>(a, tm, n_hc, n_tc, st);
}
