// Windowed / chunked / gated prefill attention over the page pools (the contract of attention_window.cu) on the 5th-gen tensor cores, for
// bf16 with key sizes and value sizes that are multiples of 16 up to 128.
//
// A pass = 128 query rows against the pages of one sequence and K/V head, in two halves of 64 rows; a half is one tile record x one query
// head. The halves are two query heads of one group, so that grouped-query heads share the K/V pages that a CTA stages, or, in groups of odd
// size, two neighbouring tile records of a sequence (the block of the second takes both; records whose neighbour is another sequence's take a
// pass each, with one half idle). Two CTAs share an SM.
//   warps 0-3:  softmax, a query row (TMEM lane) per thread. S is double buffered in TMEM, so the scores of the next two pages are computed while
//               this one is swept, 32 keys at a time; P goes back over the consumed S columns and is the A operand of P.V straight from TMEM.
//               P is formed against the reference maximum of the pages before (base-2 domain; the sink is the first reference, with a
//               denominator of 1), so that no weight waits for the page's own maximum: O and l are rescaled when the reference fell 2^8 behind,
//               and the weights are formed again when it fell 2^64 behind or there was none. Scores, penalties, weights and all sums are fp32, two
//               per instruction where that goes. The penalties of a warp's 95 distances to a page are staged by the warp, read one page ahead.
//               A weight is two bf16 numbers, its upper 16 bits and what they leave, and takes part in two products: with one rounded
//               number the error against 64 bits was 2.4e-3 of the outputs (4 x 2048 tokens, 16 heads of 128 over 4, window 1024), above
//               the 2.0e-3 of weights against each page's exact maximum; with two it is 1.7e-3.
//   warp 4:     finds the passes and copies queries and pages (cp.async, the addresses that the mma.sync kernel reads; as 64-column boxes swizzled
//               for the tensor cores), two stages. No tensor maps: what a map may touch beyond the rows that exist is not asked.
//               The grid's next CTA that has not started is taken over (cluster launch control): its first pages and scores are under way while
//               the outputs of this one are written; as CTAs of their own they cost 17 000 clocks beside their pages.
//   warp 5:     one thread issues the MMAs: O += P(j) V(j), then S(j + 2) = Q K(j + 2)^T into the columns P(j) left
// A page that belongs to one record of a pass only is multiplied by weights of zero for the other, which a value that is not finite would make something
// else: the idle half's warps look the page's values over, and where there is one they hold O across the page.
// Where the passes of a step leave places on the chip empty, two to eight CTAs of a cluster share the pages of each (the caller says how many pages a pass
// has at most): every CTA sweeps a run of them, and each adds up a share of the rows from the sums of all, through distributed shared memory.
// Bound by the softmax warps: their instructions issue in the order of a page's 64 keys a row, a third of the time a warp waits for the next one from
// the cache of instructions (so the sweep is two runs of 32 keys, and what a page needs only rarely is a function), and two CTAs share the SM's
// exponentials; the MMAs keep the tensor cores busy half of the time. 4 x 2048 tokens, 16 heads of 128 over 4, window 1024, penalties: 110 us (before
// the functions 113, mma.sync 298); 333 rows of 32 x 96 behind 704: 32 (one CTA a pass 37, mma.sync 67); 16 prompts of 60 tokens behind 500, 16 heads of
// 96: 0.6 of mma.sync. Not kept: two threads a row and eight warps a CTA (125 for 115: a third more instructions), a loader in warps of its own with
// the softmax warps' registers raised (130), runs of 16 keys (116).
//
// Every wait of a CTA has a limit: when one runs out no thread of the CTA waits any more, the loader takes over nothing more, and the CTA ends with its last
// blocks of the grid (and one that it had taken over already) written as not a number and the status word set. A cluster's barriers have none of their
// own: every CTA comes to them, as its waits end, and one whose waits ran out tells the others, which write the rows of the pass as not a number.
#include "tc_common.cuh"
#include "attention_window.cuh"
#include <type_traits>

namespace {
constexpr float LOG2E = 1.4426950408889634f;
constexpr int BOX = 64 * 128;                                // bytes of one 64-row x 64-column box

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
// 32 columns of the lane, as 16 pairs. Pairs stay pairs from TMEM to TMEM: packed anew for every operation, a page took four times the
// instructions.
__device__ __forceinline__ void ld32(uint32_t t, f2* v) {
    asm volatile("{\n.reg .b32 a<32>;\n"
                 "tcgen05.ld.sync.aligned.32x32b.x32.b32 {a0,a1,a2,a3,a4,a5,a6,a7,a8,a9,a10,a11,a12,a13,a14,a15,a16,a17,a18,a19,a20,a21,a22,a23,a24,a25,a26,"
                 "a27,a28,a29,a30,a31}, [%16];\n"
                 "tcgen05.wait::ld.sync.aligned;\n"
                 "mov.b64 %0,{a0,a1};\nmov.b64 %1,{a2,a3};\nmov.b64 %2,{a4,a5};\nmov.b64 %3,{a6,a7};\nmov.b64 %4,{a8,a9};\nmov.b64 %5,{a10,a11};\n"
                 "mov.b64 %6,{a12,a13};\nmov.b64 %7,{a14,a15};\nmov.b64 %8,{a16,a17};\nmov.b64 %9,{a18,a19};\nmov.b64 %10,{a20,a21};\n"
                 "mov.b64 %11,{a22,a23};\nmov.b64 %12,{a24,a25};\nmov.b64 %13,{a26,a27};\nmov.b64 %14,{a28,a29};\nmov.b64 %15,{a30,a31};\n}"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]), "=l"(v[4]), "=l"(v[5]), "=l"(v[6]), "=l"(v[7]), "=l"(v[8]), "=l"(v[9]), "=l"(v[10]),
                   "=l"(v[11]), "=l"(v[12]), "=l"(v[13]), "=l"(v[14]), "=l"(v[15]) : "r"(t));
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

// penalties of a warp's 32 rows against its 32 keys: entry t = distance (first row + 31 - t) to the warp's first key, so that a row's columns are
// neighbours; four copies shifted by 0 .. 3 entries let every lane read 16-byte pieces, and their pitch keeps a quarter-warp on different banks
constexpr int PEN_LD = 104;

constexpr int ST = 2;                                        // pages in flight (as many as score buffers)
constexpr int W_LOAD = 4, W_MMA = 5, THREADS = 192;
constexpr int TMEM = 256, O_COL = 128;                       // S(buffer) at 64 buffer, O at O_COL
constexpr int ITEMS = 8;                                     // passes whose grid blocks a CTA remembers: the loader is at most four ahead of the outputs
constexpr int TURN = 2048;                                   // bytes of a warp's block of outputs: 32 rows x 64 bytes
// Q of up to 2 boxes x 128 rows, K and V pages of up to 2 boxes, penalty slices, blocks of outputs
size_t win_smem(int kb, int vb) { return (size_t)kb * 2 * BOX + (size_t)ST * (kb + vb) * BOX + 4 * 4 * PEN_LD * 4 + 4 * TURN + 1024; }

// barriers: index of the first of two (by page or pass), but for Q_FULL, NEXT_FULL and DRAINED
enum { Q_FULL = 0, K_FULL = 1, K_EMPTY = 3, V_FULL = 5, V_EMPTY = 7, S_FULL = 9, SM_DONE = 11, O_DONE = 13, PASS_FULL = 15, PASS_EMPTY = 17, NEXT_FULL = 19, DRAINED = 20, BARS = 21 };
__device__ __forceinline__ uint32_t ph(int p) { return (uint32_t)(p >> 1) & 1u; }

// One pass: up to two records of one sequence, found by the loader for the other warps
// n: pages (0: no more work); mine: bit i: record i belongs to the pass. Split: the CTA's pages are those from `first` on of n_all
struct Pass { int4 rec[2]; int n, lo_pg, n_keep, h0, mine, first, n_all; };

// O of the row (its last product waited for) times cf, and the weights of the page's first 32 keys: behind an older reference
__device__ __noinline__ void scale_o_far(uint32_t t_o, int dv, uint32_t wait_bar, uint32_t wait_ph, bool wait, volatile int* fail, float cf) {
    if (wait) { mbar_wait_lim<false>(wait_bar, wait_ph, fail); tc_fence_after(); }
#pragma unroll 1
    for (int c = 0; c < dv; c += 16) {
        uint32_t v[16];
        ld16(t_o + c, v);
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = __float_as_uint(__uint_as_float(v[k]) * cf);
        st16(t_o + c, v);
    }
}
__device__ __noinline__ void scale_p_far(uint32_t t_s, float cf) {
    uint32_t w[32];
    tc_wait_st();
    tc_ld32_nowait(t_s, w);
    tc_wait_ld();
    tc_reg_fence32(w);
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const float2 a0 = unpack_bf16(w[k]), a1 = unpack_bf16(w[16 + k]);
        const float p0 = (a0.x + a1.x) * cf, p1 = (a0.y + a1.y) * cf;
        w[k] = __byte_perm(__float_as_uint(p0), __float_as_uint(p1), 0x7632);
        w[16 + k] = pack_bf16(p0 - __uint_as_float(__float_as_uint(p0) & 0xffff0000u), p1 - __uint_as_float(__float_as_uint(p1) & 0xffff0000u));
    }
    tc_st32_nowait(t_s, w);
}

// A page of the other record (softmax warps): weights of zero, and O, zero before the pass's first page, held across the page if a value of it is not finite
// (two rows a lane; a number times zero, added up, stays zero)
__device__ __noinline__ void other_page(uint32_t bars, int p, bool first, uint32_t t_lane, uint32_t sv, int dv, volatile int* fail) {
    const int lane = threadIdx.x & 31;
    auto bar = [&](int first_of_two, int q) { return bars + 8u * (first_of_two + (q & 1)); };
    uint32_t w[32], z[2] = {0u, 0u};
#pragma unroll
    for (int k = 0; k < 32; k++) w[k] = 0u;
    mbar_wait_lim<false>(bar(S_FULL, p), ph(p), fail);
    tc_fence_after();
    tc_st32_nowait(t_lane + (p & 1) * 64, w);
    tc_st32_nowait(t_lane + (p & 1) * 64 + 32, w);
    mbar_wait_lim<false>(bar(V_FULL, p), ph(p), fail);
#pragma unroll 2
    for (int k = 0; k < dv / 8; k++)
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint4 x;
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w)
                         : "r"(sv + (k >> 3) * BOX + (lane + 32 * r) * 128 + (((k & 7) ^ (lane & 7)) << 4)) : "memory");
            asm("{\n.reg .b32 t;\nfma.rn.bf16x2 t, %1, %5, %0;\nfma.rn.bf16x2 t, %2, %5, t;\nfma.rn.bf16x2 t, %3, %5, t;\nfma.rn.bf16x2 %0, %4, %5, t;\n}"
                : "+r"(z[r]) : "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w), "r"(0));
        }
    const bool hold = __any_sync(0xffffffffu, ((z[0] | z[1]) & 0x7fff7fffu) != 0u);
    uint32_t held[128];
    if (hold) {
        if (!first) { mbar_wait_lim<false>(bar(O_DONE, p - 1), ph(p - 1), fail); tc_fence_after(); }
#pragma unroll 1
        for (int c = 0; c < dv; c += 16) {
            uint32_t v[16];
            ld16(t_lane + O_COL + c, v);
#pragma unroll
            for (int k = 0; k < 16; k++) held[c + k] = first ? 0u : v[k];
        }
    }
    tc_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(SM_DONE, p));
    if (hold) {
        mbar_wait_lim<false>(bar(O_DONE, p), ph(p), fail);
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < dv; c += 16) {
            uint32_t v[16];
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = held[c + k];
            st16(t_lane + O_COL + c, v);
        }
    }
}

// Tile record of the i-th blocks of the grid: later ones (more keys) first. With pairs those that always have a pass, the second records and the last if it has
// no partner, before the first records, most of which went with their partners.
template <bool PAIR>
__device__ __forceinline__ int tile_of(int i, int n) {
    if (!PAIR) return n - 1 - i;
    const int early = (n + 1) / 2;
    if (i < early) return n - 2 * i - ((n & 1) == 0 || i == 0 ? 1 : 0);
    return (n & ~1) - 2 - 2 * (i - early);
}

// After a wait that ran out: the rows of the last passes and of the block that was taken over, of which it is not known which were written. (A function of
// its own: in the kernel's lines it cost launches of one page 0.3 us; 16 heads of 128, 40 tokens: 9.2 and 8.8.)
template <bool PAIR>
__device__ __noinline__ void mark_rows(bf16* out, int64_t ld_out, const int4* tiles, int n_tiles, int hgs, int cols, const int* items, int* status) {
    for (int k = 0; k < ITEMS; k++) {
        const int item = items[k];
        if (item < 0) continue;
        const int last = tile_of<PAIR>(item / hgs, n_tiles);
        for (int t = PAIR ? last & ~1 : last; t <= last; t++) {
            const int4 r = tiles[t];
            for (int i = threadIdx.x; i < r.y * cols; i += THREADS)
                out[(size_t)(r.x + i / cols) * ld_out + (size_t)(item % hgs) * cols + i % cols] = __float2bfloat16_rn(__int_as_float(0x7fc00000));
        }
    }
    if (threadIdx.x == 0) set_status(status);
}

__device__ __forceinline__ uint32_t at_cta(uint32_t addr, int cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}

// PAIR: neighbouring records of a sequence share a pass. SPLIT: the CTAs of a cluster share the pages of a pass, n_split of them. Every CTA tells the others
// its rows' reference maxima and sums, then sends each row's O, at the common maximum, to the CTA that adds up and writes that row.
template <bool PEN, bool SIG, bool PAIR, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 2)
attn_window_prefill_tc_kernel(p3_attn_window_args a, int n_hc, int n_split, int* status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(16) Pass pass_s[2];
    __shared__ __align__(16) uint4 next_s;
    __shared__ __align__(8) uint64_t bars_s[BARS];
    __shared__ int fail_s, items_s[ITEMS];
    __shared__ uint32_t tmem_s;
    volatile int* fail = &fail_s;
    const int d = a.dim, dv = a.vdim, kb = (d + 63) / 64, vb = (dv + 63) / 64, rep = a.n_heads / a.n_kv;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    const uint32_t sQ = base, sK = sQ + kb * 2 * BOX, sV = sK + ST * kb * BOX;
    const uint32_t pen_off = sV + ST * vb * BOX - raw, turn = raw + pen_off + 4 * 4 * PEN_LD * 4, bars = smem_u32(bars_s);
    // pages are counted through all passes of the CTA
    const uint32_t q_full = bars + 8u * Q_FULL;
    auto k_full = [&](int p) { return bars + 8u * (K_FULL + (p & 1)); };
    auto k_empty = [&](int p) { return bars + 8u * (K_EMPTY + (p & 1)); };
    auto v_full = [&](int p) { return bars + 8u * (V_FULL + (p & 1)); };
    auto v_empty = [&](int p) { return bars + 8u * (V_EMPTY + (p & 1)); };
    auto s_full = [&](int p) { return bars + 8u * (S_FULL + (p & 1)); };
    auto sm_done = [&](int p) { return bars + 8u * (SM_DONE + (p & 1)); };
    auto o_done = [&](int p) { return bars + 8u * (O_DONE + (p & 1)); };
    auto pass_full = [&](int i) { return bars + 8u * (PASS_FULL + (i & 1)); };
    auto pass_empty = [&](int i) { return bars + 8u * (PASS_EMPTY + (i & 1)); };
    const uint32_t next_full = bars + 8u * NEXT_FULL, drained = bars + 8u * DRAINED;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // split: every CTA's rows' {reference maximum, sum}, where the blocks of outputs are otherwise
    auto state = [&](int cta, int row) -> float2& { return reinterpret_cast<float2*>(smem_raw + (turn - raw))[cta * 128 + row]; };
    const int rank = SPLIT ? (int)(blockIdx.x % n_split) : 0;
    float run_at = -INFINITY, run_l = 0.f;                   // those of this thread's row, of a CTA with pages
    auto tell = [&](int row, float m, float l) {             // to all CTAs, of which it is known that they run
#pragma unroll 1
        for (int c = 0; c < n_split; c++)
            asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(at_cta(turn + 8 * (rank * 128 + row), c)), "f"(m), "f"(l) : "memory");
    };
    if (warp == W_MMA) {
        if (lane == 0) {
            mbar_init(q_full, 32);
            for (int p = 0; p < 2; p++) {
                mbar_init(k_full(p), 32); mbar_init(k_empty(p), 1); mbar_init(v_full(p), 32); mbar_init(v_empty(p), 1);
                mbar_init(s_full(p), 1); mbar_init(o_done(p), 1); mbar_init(sm_done(p), 4);
                mbar_init(pass_full(p), 1); mbar_init(pass_empty(p), 5);
            }
            mbar_init(next_full, 1); mbar_init(drained, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            fail_s = 0;
            for (int k = 0; k < ITEMS; k++) items_s[k] = -1;
        }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "n"(TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (SPLIT) cluster_arrive();                             // this CTA runs: the others may write to its shared memory once all have said so
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_s);
    pdl_trigger();
    pdl_wait();                                              // q, the pools, the tile records and `out` belong to earlier kernels until here

    if (warp == W_LOAD) {
        // A page of one K/V head is one block of memory: lane l of copy i brings its 16-byte piece 32 i + l. The place of a piece in the boxes
        // (64 columns, pieces swizzled as the UMMA reads them) repeats, 8 or 16 rows on, after `per` copies: a copy costs its instruction
        // alone (with the place formed for each one the copies of a page took 850 instructions).
        const int v_ld = a.v_ld > 0 ? a.v_ld : dv;
        // whole rows, also where a value is the leading part of its key (what comes in behind it is not read)
        const bool v_whole = v_ld == dv || (a.v_pool == a.k_pool && v_ld == d && kb == vb);
        auto period = [](int cols) { return cols % 32 == 0 ? cols / 32 : cols / 16; };
        auto places = [&](uint32_t (&at)[8], int cols) {
            const int pr = cols / 8, dr = 32 / pr, dc = 32 - dr * pr;        // pieces per row; rows and pieces from one copy to the next
            int rr = lane / pr, c = lane - rr * pr;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                at[u] = (c >> 3) * BOX + rr * 128 + (((c & 7) ^ (rr & 7)) << 4);
                rr += dr; c += dc;
                if (c >= pr) { c -= pr; rr++; }
            }
        };
        uint32_t k_at[8], v_at[8];
        places(k_at, d);
        places(v_at, v_whole ? v_ld : dv);
        auto copy = [&](uint32_t dst, const bf16* src, const uint32_t (&at)[8], int cols, auto per) {
            constexpr int P = decltype(per)::value;
            const char* s = reinterpret_cast<const char*>(src) + 16 * lane;
            const int n_c = cols / 4, step = 256 * P / cols * 128;
            for (int i = 0; i < n_c; i += P, dst += step, s += 512 * P)
#pragma unroll
                for (int u = 0; u < P; u++) cp_async16(dst + at[u], s + 512 * u);
        };
        // `bar` hears from every lane when its copies have landed
        auto stage = [&](uint32_t dst, const bf16* src, const uint32_t (&at)[8], int cols, int per, uint32_t bar) {
            if (per == 4) copy(dst, src, at, cols, std::integral_constant<int, 4>{});
            else if (per == 3) copy(dst, src, at, cols, std::integral_constant<int, 3>{});
            else if (per == 2) copy(dst, src, at, cols, std::integral_constant<int, 2>{});
            else if (per == 1) copy(dst, src, at, cols, std::integral_constant<int, 1>{});
            else if (per == 5) copy(dst, src, at, cols, std::integral_constant<int, 5>{});
            else copy(dst, src, at, cols, std::integral_constant<int, 7>{});
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
        };
        const int k_per = period(d), v_cols = v_whole ? v_ld : dv, v_per = period(v_cols);
        const int4* recs = reinterpret_cast<const int4*>(a.tiles);
        const int hgs = a.n_heads / n_hc, keep_pg = (a.keep_first + 63) / 64;
        int page_0 = 0, passes = 0, taken = 0;           // pages before this pass, passes, CTAs taken over
        bool all_done = false;
        for (int item = SPLIT ? blockIdx.x / n_split : blockIdx.x; item >= 0; taken++) {
            // The grid's next CTA that has not started is taken over after this one: its rows' pages are on the way while these outputs are written. Where
            // blocks may turn out to be without a pass it is asked for once the pages of this one are on the way, so that none waits behind a
            // long pass while other CTAs find nothing to do.
            auto take_over = [&]() {
                if (lane == 0) {
                    mbar_expect_tx(next_full, 16);
                    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(&next_s)), "r"(next_full) : "memory");
                }
            };
            if (!PAIR && !SPLIT) take_over();
            const int t = tile_of<PAIR>(item / hgs, a.n_tiles), h0 = item % hgs * n_hc, g = h0 / rep;
            const int4 r0 = recs[PAIR ? t & ~1 : t], r1 = PAIR ? recs[min(t | 1, a.n_tiles - 1)] : r0, own = PAIR && (t & 1) ? r1 : r0;
            const bool both = PAIR && (t | 1) < a.n_tiles && r1.z == r0.z && r0.y > 0 && r1.y > 0;
            if (both ? (t & 1) != 0 : own.y > 0) {       // a pass, unless the block of the next record takes this one too, or there are no rows
                const int first = both ? min(first_key(a, r0.w), first_key(a, r1.w)) : first_key(a, own.w);
                const int last = both ? max(r0.w + r0.y, r1.w + r1.y) - 1 : own.w + own.y - 1;
                // pages: those of the kept first tokens before the window's pages, then from the first visible key to the last row's position
                const int lo_pg = first / 64, n_keep = min(keep_pg, lo_pg), n_all = n_keep + last / 64 - lo_pg + 1;
                const int from = SPLIT ? n_all * rank / n_split : 0, n = SPLIT ? n_all * (rank + 1) / n_split - from : n_all;
                auto page_at = [&](int it) { it += from; return it < n_keep ? it : lo_pg + it - n_keep; };
                const int32_t* bt = a.block_table + (size_t)own.z * a.bt_stride;
                int page = 0, page1 = n > 0 ? bt[page_at(0)] : 0;    // ids of pages it, it + 1
                const int mine = both ? 3 : PAIR && (t & 1) ? 2 : 1;
                if (lane == 0) {
                    items_s[passes % ITEMS] = item;
                    mbar_wait_lim<false>(pass_empty(passes), ph(passes) ^ 1u, fail);
                    if (SPLIT || !*fail) {               // else the place may be in use (split: the only pass, which the CTA's end goes by whatever ran out)
                        Pass& ps = pass_s[passes & 1];
                        ps.rec[0] = r0; ps.rec[1] = r1; ps.n = n; ps.lo_pg = lo_pg; ps.n_keep = n_keep; ps.h0 = h0; ps.mine = mine; ps.first = from; ps.n_all = n_all;
                        mbar_arrive(pass_full(passes));
                    }
                }
                __syncwarp();
                for (int it = n > 0 ? -1 : 0; it < n; it++) {        // K one page ahead of V: its stage comes free earlier
                    const int page2 = it + 2 < n ? bt[page_at(it + 2)] : 0, p = page_0 + it;
                    if (it + 1 < n) {
                        mbar_wait_lim<false>(k_empty(p + 1), ph(p + 1) ^ 1u, fail);
                        stage(sK + ((p + 1) & 1) * kb * BOX, (const bf16*)a.k_pool + ((size_t)page1 * a.n_kv + g) * 64 * d, k_at, d, k_per, k_full(p + 1));
                    }
                    if (it < 0) {                        // the queries, once the scores of the pass before are there
                        if (p >= 0) mbar_wait_lim<false>(k_empty(p), ph(p), fail);
                        auto copy_q = [&](auto lanes) {  // lanes per row
                            constexpr int LPR = decltype(lanes)::value, PER = 32 / LPR;
                            const int c = lane % LPR, hi = lane / LPR;
#pragma unroll 1
                            for (int u = 0; u < 2; u++) {        // a half: one record, one head; rows that it does not have are zeros
                                const int4 r = u / n_hc ? r1 : r0;
                                const int left = (8 * c < d && (mine >> (u / n_hc) & 1) ? r.y : 0) - hi;
                                const bf16* src = (const bf16*)a.q + (size_t)(r.x + hi) * a.ld_q + (size_t)(h0 + u % n_hc) * d + 8 * c;
                                const uint32_t dst = sQ + (c >> 3) * 2 * BOX + (u * 64 + hi) * 128 + (((c & 7) ^ hi) << 4);
#pragma unroll
                                for (int k = 0; k < 2 * LPR; k++, src += (size_t)PER * a.ld_q)
                                    cp_async16((dst ^ ((k * PER & 7) << 4)) + k * PER * 128, k * PER < left ? src : (const bf16*)a.q, k * PER < left ? 16 : 0);
                            }
                        };
                        if (kb == 2) copy_q(std::integral_constant<int, 16>{}); else copy_q(std::integral_constant<int, 8>{});
                        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(q_full) : "memory");
                    } else {
                        mbar_wait_lim<false>(v_empty(p), ph(p) ^ 1u, fail);
                        const uint32_t dst = sV + (p & 1) * vb * BOX;
                        const bf16* src = (const bf16*)a.v_pool + ((size_t)page * a.n_kv + g) * 64 * v_ld;
                        if (v_whole) stage(dst, src, v_at, v_cols, v_per, v_full(p));
                        else {                           // the leading numbers of longer rows
                            for (int i = lane; i < 8 * dv; i += 32) {
                                const int rr = i / (dv / 8), c = i - rr * (dv / 8);
                                cp_async16(dst + (c >> 3) * BOX + rr * 128 + (((c & 7) ^ (rr & 7)) << 4), src + (size_t)rr * v_ld + 8 * c);
                            }
                            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(v_full(p)) : "memory");
                        }
                    }
                    page = page1; page1 = page2;
                }
                page_0 += n;
                passes++;
                if (SPLIT && n == 0) all_done = true;    // that was the end of the work as well
            }
            if (SPLIT) break;
            if (PAIR) take_over();
            const bool came = __all_sync(0xffffffffu, mbar_drain<false>(next_full, taken & 1u));       // in flight: waited for even where nothing else is
            if (!came) *fail = 1;
            uint32_t more, x = 0;
            asm volatile("{\n.reg .pred p;\n.reg .b128 h;\nld.shared.b128 h, [%2];\nclusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n"
                         "selp.u32 %0, 1, 0, p;\nmov.u32 %1, 0;\n@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n}"
                         : "=r"(more), "=r"(x) : "r"(smem_u32(&next_s)) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            item = came && more ? (int)x : -1;
            if (__any_sync(0xffffffffu, *fail)) {
                if (lane == 0) items_s[passes % ITEMS] = item;
                break;
            }
        }
        if (lane == 0 && !all_done) {
            mbar_wait_lim<false>(pass_empty(passes), ph(passes) ^ 1u, fail);
            if (SPLIT && passes == 0) pass_s[0].mine = pass_s[0].n_all = 0;
            if (!*fail) {
                pass_s[passes & 1].n = 0;
                mbar_arrive(pass_full(passes));
            }
        }
        cp_async_wait<0>();
        for (int p = max(0, page_0 - ST); p < page_0; p++) {       // nothing is in flight when the CTA ends
            mbar_wait_lim<false>(k_empty(p), ph(p), fail);
            mbar_wait_lim<false>(v_empty(p), ph(p), fail);
        }
    } else if (warp == W_MMA) {
        // MMA issuer: one thread, its products at constant distances from what a page starts from
        constexpr uint32_t ID = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
        const uint32_t id_qk = ID | ((64u >> 3) << 17), id_pv = ID | (1u << 16) | ((uint32_t)(dv >> 3) << 17);
        // operand descriptors; what changes is added to their address fields (16-byte units)
        const uint64_t qd = umma_desc_sw128(sQ), kd0 = umma_desc_sw128(sK), vd0 = umma_desc_mn_sw128(sV, BOX, 1024);
        auto issue = [&](auto steps) {                   // steps of 16 numbers of a key; 0: a number that is not one of the usual
            constexpr int KS = decltype(steps)::value;
            const int ks = KS ? KS : d / 16;
            for (int i = 0, page_0 = 0;; i++) {
                mbar_wait_lim<false>(pass_full(i), ph(i), fail);
                const int n = *reinterpret_cast<volatile int*>(&pass_s[i & 1].n);
                mbar_arrive(pass_empty(i));
                if (n <= 0 || *fail) break;
                mbar_wait_lim<false>(q_full, i & 1, fail);
                for (int t = 0; t < n + 2; t++) {
                    const int p = page_0 + t, j = p - 2;
                    if (t >= 2) mbar_wait_lim<false>(v_full(j), ph(j), fail);
                    if (t < n) mbar_wait_lim<false>(k_full(p), ph(p), fail);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the copies, for the tensor cores
                    if (t >= 2) {                        // O += P(j) V(j)
                        mbar_wait_lim<false>(sm_done(j), ph(j), fail);
                        tc_fence_after();
                        const uint32_t o = tmem + O_COL, pc = tmem + (j & 1) * 64;
                        const uint64_t vd = vd0 + (uint32_t)((j & 1) * vb * (BOX >> 4));
#pragma unroll
                        for (int kk = 0; kk < 8; kk++)   // P of keys 0-31 in columns 0-15, of keys 32-63 in columns 32-47; the rest 16 columns on
                            tc_mma_bf16_ts(o, pc + 16 * (kk >> 2) + 32 * ((kk >> 1) & 1) + 8 * (kk & 1), vd + (kk & 3) * (16 * 128 >> 4), id_pv,
                                           kk ? 1u : (uint32_t)(t - 2));
                        tc_commit(o_done(j));
                        tc_commit(v_empty(j));
                    }
                    if (t < n) {                         // S(t) = Q K(t)^T, behind the P.V that reads the same columns
                        tc_fence_after();
                        const uint32_t sc = tmem + (p & 1) * 64;
                        const uint64_t kd = kd0 + (uint32_t)((p & 1) * kb * (BOX >> 4));
#pragma unroll
                        for (int kk = 0; kk < 8; kk++)
                            if (kk < ks) tc_mma_bf16(sc, qd + ((kk >> 2) * (2 * BOX >> 4) + 2 * (kk & 3)), kd + ((kk >> 2) * (BOX >> 4) + 2 * (kk & 3)), id_qk, kk ? 1u : 0u);
                        tc_commit(s_full(p));
                        tc_commit(k_empty(p));
                    }
                }
                page_0 += n;
            }
            if (*fail) { tc_commit(drained); mbar_drain<false>(drained, 0); }               // products that nothing waited for
        };
        if (elect_one()) {
            if (d == 128) issue(std::integral_constant<int, 8>{});
            else if (d == 96) issue(std::integral_constant<int, 6>{});
            else if (d == 64) issue(std::integral_constant<int, 4>{});
            else issue(std::integral_constant<int, 0>{});
        }
        __syncwarp();
    } else {
        // ---- softmax: 32 rows of one half (one record, one head) per warp, a row per thread
        const int u = warp >> 1, r0 = (warp & 1) * 32, i = r0 + lane;
        const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16), t_o = t_lane + O_COL;
        for (int pass = 0, page_0 = 0;; pass++) {
            mbar_wait_lim<false>(pass_full(pass), ph(pass), fail);
            const Pass& now = pass_s[pass & 1];
            const int n = now.n, n_keep = now.n_keep, past_keep = now.lo_pg - now.n_keep, h = now.h0 + u % n_hc, from = SPLIT ? now.first : 0;
            const bool mine = now.mine >> (u / n_hc) & 1, shared = PAIR && now.mine == 3;
            const int4 rec = now.rec[u / n_hc];
            const int lo_pg = now.lo_pg;
            __syncwarp();
            if (lane == 0) mbar_arrive(pass_empty(pass));
            if (n <= 0 || __any_sync(0xffffffffu, *fail)) break;
            auto page_at = [&](int it) { it += from; return it < n_keep ? it : past_keep + it; };
            const int nq = mine ? rec.y : 0, pos = rec.w + i;
            const bool row_ok = i < nq;
            // without penalties a key that is not seen is `gone` before the scale is multiplied in, -infinity behind it whatever the scale's sign; a scale
            // of zero is the smallest number instead (a score of 3e38 becomes 5e-7)
            const float scale2 = PEN || a.scale != 0.f ? a.scale * LOG2E : __int_as_float(1), gone = PEN || scale2 > 0.f ? -INFINITY : INFINITY;
            const float sb2 = SIG ? a.sig_bias[h] * LOG2E : 0.f;
            const f2 scale22 = SIG && !PEN ? pack2(-scale2, -scale2) : pack2(scale2, scale2), sbias22 = pack2(-sb2, -sb2), one2 = pack2(1.f, 1.f);
            const bool sink = a.sink && rank == 0;
            float m = sink ? a.sink[h] * LOG2E : -INFINITY, l = sink ? 1.f : 0.f, pend = 1.f, at = m;     // pend: what O and l, which are at the reference `at`, are to be multiplied by
            const int lo = first_key(a, pos), warp_lo = rec.w + r0, warp_hi = rec.w + min(nq - 1, r0 + 31), lo_hi = first_key(a, max(warp_hi, 0));
            const bool any_rows = r0 < nq, all_rows = r0 + 32 <= nq;
            if (SPLIT && a.elem_gate && row_ok && (warp * 32 + lane) / ((128 + n_split - 1) / n_split) == rank)      // the gates of the rows that this CTA will write
                for (int c = 0; c < dv; c += 32)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(a.elem_gate + ((size_t)rec.x + i) * a.ld_elem_gate + (size_t)h * dv + c));
            float* ps = reinterpret_cast<float*>(smem_raw + pen_off) + warp * 4 * PEN_LD;
            const float* pl = ps + ((31 - lane) & 3) * PEN_LD + ((31 - lane) & ~3);          // this lane's copy, column 0
            float pn[3];
            auto pen_fetch = [&](int it) {
                const float* p = a.penalty + (size_t)h * a.n_penalty;
                const int dist = warp_lo + 31 - page_at(it) * 64 - lane;
#pragma unroll
                for (int k = 0; k < 3; k++) pn[k] = p[min(max(dist - 32 * k, 0), a.n_penalty - 1)];
            };
            // a record's own pages are two runs of the pass's: kept ones from 0 to x, and from y to `end`
            int x = 0, y = 0, end = n;
            if (shared) {
                const int lo_own = first_key(a, rec.w) / 64, keep_own = min((a.keep_first + 63) / 64, lo_own);
                if (lo_own > lo_pg) { x = n_keep + max(0, keep_own - lo_pg); y = n_keep + lo_own - lo_pg; }
                end = n_keep + (rec.w + nq - 1) / 64 - lo_pg + 1;
                if (SPLIT) { x = min(max(x - from, 0), n); y = min(max(y - from, 0), n); end = min(max(end - from, 0), n); }
            }
            for (int run = PAIR ? 0 : 1; run < 2; run++) {
                int it = run ? y : 0;
                const int stop = run ? end : x;
                if (PEN && it < stop) pen_fetch(it);
                for (; it < stop; it++) {
                    const int j0 = page_at(it) * 64;
                    const int p = page_0 + it;
                    const uint32_t t_s = t_lane + (p & 1) * 64;
                    if (PEN) {
                        __syncwarp();                            // the page before is read
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            const float v = -LOG2E * pn[k];
#pragma unroll
                            for (int c = 0; c < 4; c++)
                                if (k || lane >= c) ps[c * PEN_LD + lane + 32 * k - c] = v;
                        }
                        __syncwarp();
                        if (it + 1 < stop) pen_fetch(it + 1);
                    }
                    mbar_wait_lim<false>(s_full(p), ph(p), fail);
                    tc_fence_after();
                    auto scale_o = [&](float cf) { scale_o_far(t_o, dv, o_done(p - 1), ph(p - 1), it > 0, fail, cf); };
                    // every key of the page is visible to every row of the warp: behind its first row, and its last row still sees it
                    const bool full = all_rows && j0 + 63 <= warp_lo && (j0 >= lo_hi || j0 + 63 < a.keep_first);
                    const bool none = !any_rows || j0 > warp_hi;
                    const bool whole = __all_sync(0xffffffffu, full);
                    float top = -INFINITY;                       // the page's maximum
                    if (!SIG && __builtin_expect(__any_sync(0xffffffffu, pend != 1.f), 0)) { scale_o(pend); l *= pend; }
                    // 32 keys at a time: a page of 64 scores, penalties and weights did not fit the registers. Once in the program, twice run, and what
                    // is rarely done in functions of its own: in lines of 64 keys with all of it a warp waited for instructions more than for anything
                    // else (4 x 1000 tokens behind 100, 32 heads of 96 over 8, window 512: 78 us, 66 so; 16 keys at a time 72).
#pragma unroll 1
                    for (int hf = 0; hf < 2; hf++) {
                        uint32_t pk[32];                         // their weights: upper 16 bits, then what they leave
                        if (__builtin_expect(none, 0)) {
#pragma unroll
                            for (int k = 0; k < 32; k++) pk[k] = 0u;
                        } else {
                            f2 v[16];
                            ld32(t_s + 32 * hf, v);
                            if (PEN) {
#pragma unroll
                                for (int k = 0; k < 16; k += 2) {
                                    const ulonglong2 pv = *reinterpret_cast<const ulonglong2*>(pl + 32 * hf + 2 * k);
                                    v[k] = fma2(v[k], scale22, pv.x);
                                    v[k + 1] = fma2(v[k + 1], scale22, pv.y);
                                }
                            }
                            if (!whole) {                        // a branch, so that whole pages do without the tests of every key
                                auto below = [](int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; };
                                const int j = j0 + 32 * hf;
                                const uint32_t seen = row_ok ? below(pos - j + 1) & (~below(lo - j) | below(a.keep_first - j)) : 0u;
#pragma unroll
                                for (int k = 0; k < 16; k++) {
                                    const float2 x = unpack2(v[k]);
                                    v[k] = pack2(seen >> (2 * k) & 1u ? x.x : gone, seen >> (2 * k + 1) & 1u ? x.y : gone);
                                }
                            }
                            if (!SIG) {
                                float mx[2] = {top, -INFINITY};
#pragma unroll
                                for (int k = 0; k < 16; k++) { const float2 x = unpack2(v[k]); mx[k & 1] = max3(mx[k & 1], PEN ? x.x : x.x * scale2, PEN ? x.y : x.y * scale2); }
                                top = fmaxf(mx[0], mx[1]);
                            }
                            float ls;
                            for (;;) {                           // a second time only for a reference that was none, or 2^64 behind
                                const float mu = SIG || m == -INFINITY ? 0.f : m;
                                const f2 mu2 = pack2(-mu, -mu);
                                f2 sA = 0, sB = 0;
#pragma unroll
                                for (int k = 0; k < 16; k++) {
                                    const f2 x = v[k];
                                    float2 q;
                                    f2 pp;
                                    if (SIG) {                   // 1 / (1 + 2^-(score + bias)); a masked key gives 1 / inf = 0
                                        q = unpack2(PEN ? sub2(sbias22, x) : fma2(x, scale22, sbias22));
                                        q = unpack2(add2(pack2(ex2f(q.x), ex2f(q.y)), one2));
                                        pp = pack2(rcpf(q.x), rcpf(q.y));
                                    } else {
                                        q = unpack2(PEN ? add2(x, mu2) : fma2(x, scale22, mu2));
                                        pp = pack2(ex2f(q.x), ex2f(q.y));
                                        if (k & 1) sA = add2(sA, pp); else sB = add2(sB, pp);
                                    }
                                    q = unpack2(pp);
                                    pk[k] = __byte_perm(__float_as_uint(q.x), __float_as_uint(q.y), 0x7632);
                                    const float2 r = unpack2(sub2(pp, pp & 0xffff0000ffff0000ull));
                                    pk[16 + k] = pack_bf16(r.x, r.y);
                                }
                                const float2 x = unpack2(add2(sA, sB));
                                ls = x.x + x.y;
                                if (SIG) break;
                                const bool redo = m == -INFINITY ? top != -INFINITY : top - m > 64.f;
                                if (__builtin_expect(!__any_sync(0xffffffffu, redo), 1)) break;
                                const float corr = !redo ? 1.f : m == -INFINITY ? 0.f : ex2f(m - top);
                                if (redo) m = top;
                                l *= corr;
                                if (it > 0) scale_o(corr);
                                if (hf) scale_p_far(t_s, corr);
                            }
                            l += ls;
                        }
                        tc_st32_nowait(t_s + 32 * hf, pk);
                    }
                    if (!SIG) {
                        const float grow = top - m;              // not a number (no key yet) compares false
                        at = m;
                        if (grow > 8.f) { pend = ex2f(-grow); m = top; } else pend = 1.f;
                    }
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sm_done(p));
                }
                if (PAIR)
#pragma unroll 1
                    for (; it < (run ? n : y); it++) other_page(bars, page_0 + it, it == 0, t_lane, sV + ((page_0 + it) & 1) * vb * BOX, dv, fail);
            }
            // ---- epilogue: O / l, gates
            page_0 += n;
            if (n > 1) mbar_wait_lim<false>(o_done(page_0 - 2), ph(page_0 - 2), fail);
            mbar_wait_lim<false>(o_done(page_0 - 1), ph(page_0 - 1), fail);
            tc_fence_after();
            if constexpr (SPLIT) {
                if (row_ok) { run_at = at; run_l = l; }
                continue;
            }
            if (mine && any_rows) {
                float inv = (a.gate && row_ok ? a.gate[((size_t)rec.x + i) * a.n_heads + h] : 1.f) * (a.out_scale != 0.f ? a.out_scale : 1.f);
                if (!SIG) inv = l > 0.f ? inv / l : 0.f;
                // row-wise out of TMEM into the warp's block, and from there in pieces of 64 bytes of a row (32 with gates: four lanes a row, eight
                // rows an instruction) to memory; a lane writing its own row took an instruction of the load-store unit per row and 16 bytes.
                // 16-byte pieces are swizzled: no bank conflicts either way. Without element-wise gates 32 columns go as bf16, else 16 as fp32.
                const uint32_t tb = turn + warp * TURN;
                const int sub = lane >> 2, part = lane & 3, left = nq - r0 - sub;        // rows from this lane's first on
                auto piece = [&](int row, int pc) { return tb + row * 64 + ((pc ^ ((row >> 1) & 3)) << 4); };
                const size_t row = (size_t)rec.x + r0 + sub, col = (size_t)h * dv;
                const f2 inv2 = pack2(inv, inv);
                auto put = [&](const uint32_t* w) {          // 16 words of the lane's row
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(piece(lane, k)), "r"(w[4 * k]), "r"(w[4 * k + 1]), "r"(w[4 * k + 2]), "r"(w[4 * k + 3]) : "memory");
                    __syncwarp();
                };
                auto get = [&](int k) {                      // this lane's piece of row 8 k + sub
                    uint4 y;
                    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(y.x), "=r"(y.y), "=r"(y.z), "=r"(y.w) : "r"(piece(8 * k + sub, part)));
                    return y;
                };
                if (!a.elem_gate) {
                    bf16* o = (bf16*)a.out + row * a.ld_out + col + 8 * part;
#pragma unroll 1
                    for (int c0 = 0; c0 < dv; c0 += 32) {
                        uint32_t w[16];
#pragma unroll
                        for (int hf = 0; hf < 2; hf++) {
                            if (c0 + 16 * hf >= dv) break;
                            uint32_t v[16];
                            ld16(t_o + c0 + 16 * hf, v);
#pragma unroll
                            for (int k = 0; k < 8; k++) {
                                const float2 x = unpack2(mul2(pack2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1])), inv2));
                                w[8 * hf + k] = pack_bf16(x.x, x.y);
                            }
                        }
                        put(w);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const uint4 y = get(k);
                            if (8 * k < left && c0 + 8 * part < dv) *reinterpret_cast<uint4*>(o + (size_t)(8 * k) * a.ld_out + c0) = y;
                        }
                    }
                } else {
                    bf16* o = (bf16*)a.out + row * a.ld_out + col + 4 * part;
                    const float* eg = a.elem_gate + row * a.ld_elem_gate + col + 4 * part;
                    const bool quads = a.ld_elem_gate % 4 == 0 && ((uintptr_t)a.elem_gate & 15) == 0;
                    float4 t[4], t1[4];                      // gates of these 16 columns, and of the next
                    auto gates = [&](float4* to, int c0) {
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const float* q = eg + (size_t)(8 * k) * a.ld_elem_gate + c0;
                            to[k] = 8 * k >= left || c0 >= dv ? make_float4(0.f, 0.f, 0.f, 0.f) : quads ? *reinterpret_cast<const float4*>(q) : make_float4(q[0], q[1], q[2], q[3]);
                        }
                    };
                    gates(t1, 0);
#pragma unroll 1
                    for (int c0 = 0; c0 < dv; c0 += 16) {
#pragma unroll
                        for (int k = 0; k < 4; k++) t[k] = t1[k];
                        gates(t1, c0 + 16);
                        uint32_t v[16];
                        ld16(t_o + c0, v);
#pragma unroll
                        for (int k = 0; k < 16; k++) v[k] = __float_as_uint(__uint_as_float(v[k]) * inv);
                        put(v);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const uint4 y = get(k);
                            const float y0 = __uint_as_float(y.x) * rcpf(1.0f + ex2f(-LOG2E * t[k].x)), y1 = __uint_as_float(y.y) * rcpf(1.0f + ex2f(-LOG2E * t[k].y));
                            const float y2 = __uint_as_float(y.z) * rcpf(1.0f + ex2f(-LOG2E * t[k].z)), y3 = __uint_as_float(y.w) * rcpf(1.0f + ex2f(-LOG2E * t[k].w));
                            if (8 * k < left) *reinterpret_cast<uint2*>(o + (size_t)(8 * k) * a.ld_out + c0) = make_uint2(pack_bf16(y0, y1), pack_bf16(y2, y3));
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();                                         // nothing is in flight, O is read
    tc_fence_after();
    if constexpr (SPLIT) {
        const Pass& now = pass_s[0];
        const int pitch = 4 * (dv + 4), row = threadIdx.x, share = (128 + n_split - 1) / n_split;      // rows that a CTA writes
        const bool work = now.n_all > 0 && now.mine;
        auto pages = [&](int c) { return now.n_all * (c + 1) / n_split - now.n_all * c / n_split; };
        auto rows = [&](int r) { return work && now.mine >> (r / 64 / n_hc) & 1 ? now.rec[r / 64 / n_hc].y - r % 64 : 0; };     // above 0: the row exists
        cluster_wait();                                      // every CTA runs; this one said so at its start
        if (row < 128) {
            if (*fail) tell(row, __int_as_float(0x7fc00000), 0.f);         // every CTA's rows become what is not a number
            else if (pages(rank) > 0) tell(row, run_at, run_l);
            else {                                           // no page of the CTA's own: the sink, which the first one counts, or nothing
                const bool sink = !SIG && a.sink && rank == 0 && rows(row) > 0;
                tell(row, sink ? a.sink[now.h0 + row / 64 % n_hc] * LOG2E : -INFINITY, sink ? 1.f : 0.f);
            }
        }
        __syncwarp();
        cluster_sync();
        if (row < 128 && work) {
            float top = -INFINITY, l = 0.f;
            bool bad = false;
#pragma unroll 1
            for (int c = 0; c < n_split; c++) { const float m = state(c, row).x; top = fmaxf(top, m); bad = bad || m != m; }
#pragma unroll 1
            for (int c = 0; c < n_split; c++) { const float2 t = state(c, row); l += t.y > 0.f ? t.y * ex2f(t.x - top) : 0.f; }
            const float own = state(rank, row).x, f = SIG ? 1.f : own == -INFINITY ? 0.f : ex2f(own - top);
            const int u = row / 64;
            float inv = a.out_scale != 0.f ? a.out_scale : 1.f;
            if (a.gate && rows(row) > 0) inv *= a.gate[((size_t)now.rec[u / n_hc].x + row % 64) * a.n_heads + now.h0 + u % n_hc];
            if (!SIG) inv = l > 0.f ? inv / l : 0.f;
            state(0, row).x = bad ? __int_as_float(0x7fc00000) : inv;       // (the row's own thread read it)
            if (pages(rank) > 0) {
                const uint32_t t_o = tmem + ((uint32_t)(warp * 32) << 16) + O_COL;
                const uint32_t to = at_cta(base, row / share) + (rank * share + row % share) * pitch;
#pragma unroll 1
                for (int c0 = 0; c0 < dv; c0 += 16) {
                    uint32_t v[16];
                    ld16(t_o + c0, v);
#pragma unroll
                    for (int k = 0; k < 16; k += 4)
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + 4 * (c0 + k)), "f"(__uint_as_float(v[k]) * f),
                                     "f"(__uint_as_float(v[k + 1]) * f), "f"(__uint_as_float(v[k + 2]) * f), "f"(__uint_as_float(v[k + 3]) * f) : "memory");
                }
            }
        }
        __syncwarp();
        cluster_sync();                                      // nothing is sent to a CTA behind this
        if (work) {
            const int q4 = dv / 4, r_lo = share * rank, n_r = min(share, 128 - r_lo);
            const bool quads = a.ld_elem_gate % 4 == 0 && ((uintptr_t)a.elem_gate & 15) == 0;
#pragma unroll 1
            for (int i = threadIdx.x; i < n_r * q4; i += THREADS) {
                const int r = r_lo + i / q4, c = i % q4 * 4, u = r / 64;
                if (rows(r) <= 0) continue;
                const size_t at = (size_t)now.rec[u / n_hc].x + r % 64, col = (size_t)(now.h0 + u % n_hc) * dv + c;
                float4 g = make_float4(0.f, 0.f, 0.f, 0.f), y = g;
                if (a.elem_gate) {
                    const float* q = a.elem_gate + at * a.ld_elem_gate + col;
                    g = quads ? *reinterpret_cast<const float4*>(q) : make_float4(q[0], q[1], q[2], q[3]);
                }
#pragma unroll 1
                for (int k = 0; k < n_split; k++) {
                    if (pages(k) == 0) continue;
                    const float4 t = *reinterpret_cast<const float4*>(smem_raw + (base - raw) + (k * share + r - r_lo) * pitch + 4 * c);
                    y.x += t.x; y.y += t.y; y.z += t.z; y.w += t.w;
                }
                const float inv = state(0, r).x;
                y.x *= inv; y.y *= inv; y.z *= inv; y.w *= inv;
                if (a.elem_gate) {
                    y.x *= rcpf(1.0f + ex2f(-LOG2E * g.x)); y.y *= rcpf(1.0f + ex2f(-LOG2E * g.y));
                    y.z *= rcpf(1.0f + ex2f(-LOG2E * g.z)); y.w *= rcpf(1.0f + ex2f(-LOG2E * g.w));
                }
                *reinterpret_cast<uint2*>((bf16*)a.out + at * a.ld_out + col) = make_uint2(pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
            }
        }
        if (*fail && threadIdx.x == 0) set_status(status);
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    } else if (*fail) mark_rows<PAIR>((bf16*)a.out, a.ld_out, reinterpret_cast<const int4*>(a.tiles), a.n_tiles, a.n_heads / n_hc, n_hc * dv, items_s, status);
    if (warp == W_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM) : "memory");
}

template <bool PEN, bool SIG, bool PAIR, bool SPLIT>
int launch_as(const p3_attn_window_args* a, int n_hc, int n_split, cudaStream_t st) {
    const auto kernel = attn_window_prefill_tc_kernel<PEN, SIG, PAIR, SPLIT>;
    const size_t bytes = win_smem((a->dim + 63) / 64, (a->vdim + 63) / 64);
    static P3DevFlags flags; bool& set = flags.cur();
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)win_smem(2, 2));
        P3_CHECK_ARG(e == cudaSuccess, "attn_window_prefill: shared memory attribute: %s", cudaGetErrorString(e));
        set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((int64_t)a->n_tiles * (a->n_heads / n_hc) * n_split)); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = bytes; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (SPLIT) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = n_split; attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        n++;
    }
    if (p3_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr; cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, kernel, *a, n_hc, n_split, p3_status_word());
    return 0;
}
template <bool PEN, bool SIG, bool PAIR>
int launch(const p3_attn_window_args* a, int n_hc, int n_split, cudaStream_t st) {
    return n_split > 1 ? launch_as<PEN, SIG, PAIR, true>(a, n_hc, n_split, st) : launch_as<PEN, SIG, PAIR, false>(a, n_hc, 1, st);
}
}  // namespace

// Where this kernel is the faster one, measured both ways at 8 to 32 heads and 1 to 128 tiles of rows (us, here and mma.sync). A CTA takes longer until
// its first outputs, a page less. Above 64 numbers nearly always (1 x 40 tokens, 16 heads of 96: 8.9 and 9.0; 1 x 130: 11.5 and 15.1; 4 x 2048: 143 and
// 343). mma.sync has three CTAs an SM up to 64 numbers: there with sigmoid weights (two sums a key, no maximum) from the second tile of rows on (16
// heads of 64, 1 x 64 tokens: 7.1 and 6.8; 1 x 130: 9.8 and 12.7); else once the work, in tiles x heads, fills the SMs well: for 64 numbers from 192 on
// with two heads of a group a CTA (32 heads over 8, 1 x 333 tokens behind 704: 27.9 and 32.3), from 448 with penalties (192: 15.1 and 14.2, 704: 24.7
// and 27.4) or two records a CTA (16 heads, 256: 21.7 and 21.8, 480: 30.7 and 33.6, 2048: 112 and 182); not with both (480: 23.3 and 19.9, 2048: 74 and
// 66); below 64 numbers from 1536 on (48 numbers, 48: 10.7 and 7.0, 960: 52.7 and 50.2, 1536: 91 and 104, 4096: 265 and 307).
static bool tc_wins(const p3_attn_window_args* a) {
    const int size = a->dim > a->vdim ? a->dim : a->vdim;
    const int64_t work = (int64_t)a->n_tiles * a->n_heads;
    const bool even = (a->n_heads / a->n_kv) % 2 == 0;
    if (size > 64) return true;
    if (a->sig_bias) return a->n_tiles > 1;
    if (a->penalty && !even) return false;
    return work >= (size <= 48 ? 1536 : even && !a->penalty ? 192 : 448);
}
// whole 16-byte pieces everywhere
bool attn_window_tc_ok(const p3_attn_window_args* a) {
    return tc_wins(a) && !a->act_f32 && a->dim % 16 == 0 && a->vdim % 16 == 0 && a->dim <= 128 && a->vdim <= 128 && a->ld_q % 8 == 0 && a->ld_out % 8 == 0 &&
           a->v_ld % 8 == 0 && (((uintptr_t)a->q | (uintptr_t)a->out | (uintptr_t)a->k_pool | (uintptr_t)a->v_pool) & 15) == 0;
}

int launch_attn_window_tc(const p3_attn_window_args* a, cudaStream_t st) {
    const bool even = (a->n_heads / a->n_kv) % 2 == 0;
    const int64_t full = even ? (int64_t)a->n_tiles * (a->n_heads / 2) : (int64_t)((a->n_tiles + 1) / 2) * a->n_heads;      // passes with both halves in use
    // Passes that leave half of the places (two CTAs an SM) empty share their pages among the CTAs of a cluster, up to eight. A page takes a CTA about 1.6
    // us (1.2 with sigmoid weights), the cluster's launch, exchange and sums about 11 and 0.6 a CTA, and clusters do not fill an SM's last places (64 passes
    // in fours took 23 us or 36, as the clusters fell; 96 in threes 37, in twos 25). In groups of odd size a sequence's last record has no partner, nor its first
    // where it stands second: half a pass more a sequence (records of ten sequences, 8 heads of 128: 24.9 us whole and 40 in threes). 64 rows of 16 heads of
    // 128 over 4 behind 1500: 44 -> 21 us in eights; 333 rows of 32 x 96 behind 704 37 -> 32 in twos; 500 rows of 16 over 4 stay whole (23.0; in twos
    // 25.6, in fours 24.0). Over 400 steps of 1 to 16 sequences, each timed with 1 to 8 CTAs a pass, this takes 0.966 of the time of whole passes, 1.07 at the
    // most, the best of all eight 0.951.
    const int seqs = a->n_seqs > 0 && a->n_seqs < a->n_tiles ? a->n_seqs : a->n_tiles, page = a->sig_bias ? 12 : 16;
    const int64_t passes = even ? full : (int64_t)((a->n_tiles + seqs + (seqs > 1)) / 2) * a->n_heads;
    int64_t n_split = 1, least = page * (int64_t)a->max_pages;
    for (int k = 2; k <= 8 && k * passes <= 224; k++) {
        const int64_t cost = page * (((int64_t)a->max_pages + k - 1) / k) + 110 + 6 * k;
        if (cost < least) { least = cost; n_split = k; }
    }
    // Both halves of a CTA in use, unless that would leave half of the SMs without one (a half alone takes about as long as two): 333 rows of
    // 32 heads of 96 on 96 CTAs 39 us, on 192 half empty ones 42.
    const bool two = full >= 74 || n_split > 1;
    const int n_hc = two && even ? 2 : 1, ns = (int)n_split;
    if (two && !even) {
        if (a->sig_bias) return a->penalty ? launch<true, true, true>(a, 1, ns, st) : launch<false, true, true>(a, 1, ns, st);
        return a->penalty ? launch<true, false, true>(a, 1, ns, st) : launch<false, false, true>(a, 1, ns, st);
    }
    if (a->sig_bias) return a->penalty ? launch<true, true, false>(a, n_hc, ns, st) : launch<false, true, false>(a, n_hc, ns, st);
    return a->penalty ? launch<true, false, false>(a, n_hc, ns, st) : launch<false, false, false>(a, n_hc, ns, st);
}
