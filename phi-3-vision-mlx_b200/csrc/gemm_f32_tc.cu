// fp32 products of p3_gemm_any on the 5th-gen tensor cores, without giving up fp32: an operand x is the sum of three bf16 numbers that hold its
// 24 bits exactly (the nearest to x, to what that leaves, and the rest), and of the nine products of such parts all but that of the third parts are
// formed: a product is exact to 2^-32 of itself. The tensor cores cut off where fp32 rounds, so TMEM does not sum all of K: the products of first parts
// (16 bits each) are summed over 64 numbers of k and then added to the output's running sum in fp32 registers; the others, below 2^-7 of
// them, have a sum of their own over up to 2048 numbers, smallest products of a block first.
// Relative error against 64 bits, and that of one FMA chain over K = 512 | 3072 | 8192: dense rows of N(0, 1) 9e-8 | 1.5e-7 | 2.2e-7 (chain 4.1e-7 |
// 9.9e-7 | 1.6e-6), all positive 1.0e-7 | 1.2e-7 | 2.0e-7 (3.5e-7 | 7.4e-7 | 1.4e-6), one number a row 2.5e-8 (2.5e-8), four 2.6e-8 | 3.8e-8 | 4.5e-8
// (4.0e-8). Above the chain's only where a few products are all there is: 1.1 times with two or four among 8192 numbers, 1.4 times with four of very
// different size side by side (5e-8: four cut off a block).
//
// One CTA per SM walks output tiles of 128 x BN:
//   warps 0-15:  a block of 64 numbers of k, read one block ahead into registers, is split and goes to TMEM (X: a row is a TMEM lane) and to shared
//                memory (W: K-major, 128B swizzle); three stages. With X in TMEM a product reads only W from shared memory: with both operands
//                there, the MMAs and the split's stores ask for more than its 128 bytes a clock.
//   warps 16-23: the sums of first parts are read back while the other products of the block are formed (one buffer), the others' every 32 blocks, and
//                added in registers; epilogue
//   warp 24:     issues the 32 MMAs of a block. A warp that also splits cannot: that takes some 1300 clocks.
// Bound by the split (five instructions a number, every CTA its own rows of X and W) and the MMAs, about 40 clocks each. With six products
// (24 MMAs, exact to 2^-24 at worst) 512 x 3072 x 1024 (rows, columns, K) took 27.2 us instead of 29.7 (FMA kernel 102). 1200 x 4096 x 3072: 238 us
// (725), 64 x 1024 x 3072: 41 (86), 17 x 1024 x 512: 10.9 (16.4).
// What has no parts is one FMA chain, as on the FMA pipes: rows of X and W with numbers below 2^-110 (their lower parts are below every bf16), above the
// largest bf16 or not finite, sums that are not finite, and sums below 2^-112, where TMEM cuts off more than fp32 does.
// A wait that runs out sets the status word; every tile that the CTA writes from then on is not a number (roles walk the tiles alike, so that none waits for
// another beyond that).
#include <type_traits>
#include "tc_common.cuh"
#include "gemm_any.cuh"
#include "../../include/phi3_b200.h"

namespace {
constexpr int TM_ROWS = 128, KB = 64, STAGES = 3, FLUSH = 32;   // FLUSH: blocks whose small products are summed in TMEM
constexpr int SPLIT = 16, ADD = 8, W_ADD = SPLIT, W_MMA = SPLIT + ADD, THREADS = 32 * (W_MMA + 1);
constexpr int A_COLS = 96;                                   // TMEM columns of one stage of X: three parts of 64 bf16
constexpr int ACC_COL = STAGES * A_COLS;
constexpr int TMEM = 512;                                    // 3 x 96 for X, BN sums of products of first parts, BN of the others
constexpr size_t f32tc_smem(int bn) { return (size_t)STAGES * 3 * bn * KB * 2 + 1024; }

// 16 TMEM lanes x 8 columns: thread t holds columns 2 (t % 4), + 1 of lane t / 4 in a and of lane t / 4 + 8 in b
__device__ __forceinline__ void st_16x256b(uint32_t t, const uint32_t (&a)[2], const uint32_t (&b)[2]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(t), "r"(a[0]), "r"(a[1]), "r"(b[0]), "r"(b[1]) : "memory");
}
__device__ __forceinline__ void ld_32x32b_x8(uint32_t t, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(t));
}
// a - b, two at a time
__device__ __forceinline__ void sub2(float (&d)[2], const float (&a)[2], const float (&b)[2]) {
    asm("{\n.reg .b64 x, y, z;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nsub.rn.f32x2 z, x, y;\nmov.b64 {%0, %1}, z;\n}"
        : "=f"(d[0]), "=f"(d[1]) : "f"(a[0]), "f"(a[1]), "f"(b[0]), "f"(b[1]));
}
__device__ __forceinline__ void add2(float& c0, float& c1, float a0, float a1) {
    asm("{\n.reg .b64 x, y;\nmov.b64 x, {%0, %1};\nmov.b64 y, {%2, %3};\nadd.rn.f32x2 x, x, y;\nmov.b64 {%0, %1}, x;\n}" : "+f"(c0), "+f"(c1) : "f"(a0), "f"(a1));
}
// the nearest bf16 numbers, packed, and what they leave
__device__ __forceinline__ uint32_t part(const float (&x)[2], float (&rest)[2]) {
    const uint32_t p = pack_bf16(x[0], x[1]);
    const float h[2] = {__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u)};
    sub2(rest, x, h);
    return p;
}
// four numbers -> three parts of two words each. Two parts leave at most eight bits, which are the third's; numbers below 2^-110, above the largest
// bf16 and those that are none leave more, in the lower half of their word: `more` collects these bits.
__device__ __forceinline__ void split4(const float4& f, uint32_t (&p0)[2], uint32_t (&p1)[2], uint32_t (&p2)[2], uint32_t& more) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float x[2] = {i ? f.z : f.x, i ? f.w : f.y};
        float r[2], s[2];
        p0[i] = part(x, r);
        p1[i] = part(r, s);
        const uint32_t s0 = __float_as_uint(s[0]), s1 = __float_as_uint(s[1]);
        p2[i] = __byte_perm(s0, s1, 0x7632);
        more |= s0 | s1;
    }
}

template <typename OT, int BN>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tc_kernel(AnyP p, int m_tiles, int n_tiles, int* status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars_s[2 * STAGES + 7];
    __shared__ uint32_t rows_s[2][1 + TM_ROWS + BN];          // of two tiles: the last that had such a row anywhere, in row i of X, in row i of W
    __shared__ uint32_t tmem_s;
    __shared__ int fail_s;
    volatile int* fail = &fail_s;
    constexpr int PART = BN * KB * 2, STAGE = 3 * PART;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = smem_u32(bars_s);
    auto full = [&](uint32_t s) { return bars + 8 * s; };                            // a stage is split
    auto empty = [&](uint32_t s) { return bars + 8 * (STAGES + s); };                // ... and multiplied
    auto sums = [&](uint32_t s) { return bars + 8 * (2 * STAGES + s); };             // sums are there (0: of a block's first parts, 1: of the others)
    auto taken = [&](uint32_t s) { return bars + 8 * (2 * STAGES + 2 + s); };        // ... and read
    auto rows_known = [&](uint32_t s) { return bars + 8 * (2 * STAGES + 4 + s); };   // a tile is split: rows_s[s] is written
    const uint32_t drained = bars + 8 * (2 * STAGES + 6);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        fail_s = 0;
        for (int s = 0; s < STAGES; s++) { mbar_init(full(s), SPLIT); mbar_init(empty(s), 1); }
        for (int s = 0; s < 2; s++) { mbar_init(sums(s), 1); mbar_init(taken(s), ADD); mbar_init(rows_known(s), SPLIT); }
        mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < 2 * (1 + TM_ROWS + BN); i += THREADS) (&rows_s[0][0])[i] = 0;
    if (warp == W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "n"(TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_s);
    pdl_trigger();
    pdl_wait();                                              // memory is touched only after the predecessors are done

    const int tiles = m_tiles * n_tiles, blocks = (p.K + KB - 1) / KB;
    // rows fastest: the CTAs in flight share columns of W
    auto find = [&](int tile, int& bz, int& g, int& m0, int& m1) {
        const int mt = tile % m_tiles;
        int64_t a, b;
        bz = mt % p.nb;
        const bool ok = find_tile<TM_ROWS>(p, mt / p.nb, g, a, b);
        m0 = (int)a; m1 = (int)b;
        return ok;
    };
    if (warp < SPLIT) {
        // ---- X: 16 rows and 32 of a block's numbers per warp; W: rows wr, wr + 32, ...
        const int xr = 32 * (warp & 3) + 16 * ((warp >> 2) & 1) + (lane >> 2), xk = 32 * (warp >> 3) + 4 * (lane & 3);
        const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3) + 16 * ((warp >> 2) & 1)) << 16) + 16 * (warp >> 3);
        constexpr int NB = BN / 32;
        const int wr = threadIdx.x >> 4, wk = 4 * (threadIdx.x & 15);
        const uint32_t ws = base + wr * 128 + ((((wk >> 3) ^ (wr & 7)) << 4) | ((wk & 4) << 1));
        const size_t w_step = (size_t)32 * p.ldw;
        const int whole = p.K / KB;                          // blocks without an end of K inside
        uint32_t stage = 0, phase = 1, count = 0;            // count: tiles of this CTA
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            int bz, g, m0, m1;
            if (!find(tile, bz, g, m0, m1)) continue;
            const float *xp[2], *wp;                         // rows of the tile, at this thread's numbers of the block to be read next
            float4 fx[4], fw[NB];
            const int n0 = tile / m_tiles * BN, n = n0 + wr < p.N ? n0 + wr : n0, w_left = p.N - n;
            const float* X = (const float*)p.X + (size_t)bz * p.x_bs + xk;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int m = m0 + xr + 8 * i < m1 ? m0 + xr + 8 * i : m0;
                xp[i] = X + (size_t)(p.x_rows ? p.x_rows[m] / p.x_row_div : m) * p.ldx;
            }
            wp = (const float*)p.W + (size_t)g * p.w_gstride + (size_t)bz * p.w_bs + wk + (size_t)n * p.ldw;
            // Rows that do not exist are read as the first one: their outputs are not written. Numbers behind K are zeros (`left`: numbers from
            // the block's first on; K % 4 == 0: four are inside or outside together).
            auto fetch_x = [&](int i, int left) {            // row xr + 8 (i & 1), numbers 16 (i >> 1) on
                fx[i] = xk + 16 * (i >> 1) < left ? __ldg(reinterpret_cast<const float4*>(xp[i & 1] + 16 * (i >> 1))) : make_float4(0.f, 0.f, 0.f, 0.f);
            };
            auto fetch_w = [&](int i, int left) {
                fw[i] = wk < left ? __ldg(reinterpret_cast<const float4*>(32 * i < w_left ? wp + i * w_step : wp)) : make_float4(0.f, 0.f, 0.f, 0.f);
            };
            auto next = [&]() { xp[0] += KB; xp[1] += KB; wp += KB; };
#pragma unroll
            for (int i = 0; i < 4; i++) fetch_x(i, p.K);
#pragma unroll
            for (int i = 0; i < NB; i++) fetch_w(i, p.K);
            next();
            uint32_t more_x[2] = {0, 0}, more_w[NB];
#pragma unroll
            for (int i = 0; i < NB; i++) more_w[i] = 0;
            count++;
            // block b is split, and block b + 1 read (mode 0: there is none, 1: whole, 2: it may end at K): what is split is read anew at once, so
            // that the loads of a block have the time of a block
            auto block = [&](int b, auto mode) {
                constexpr int MODE = decltype(mode)::value;
                const int left = MODE == 1 ? KB : p.K - (b + 1) * KB;
                mbar_wait_lim(empty(stage), phase, fail);
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    uint32_t a0[2], a1[2], a2[2], b0[2], b1[2], b2[2];
                    split4(fx[i], a0, a1, a2, more_x[0]);
                    if (MODE) fetch_x(i, left);
                    split4(fx[i + 1], b0, b1, b2, more_x[1]);
                    if (MODE) fetch_x(i + 1, left);
                    const uint32_t t = ta + stage * A_COLS + 4 * i;
                    st_16x256b(t, a0, b0); st_16x256b(t + 32, a1, b1); st_16x256b(t + 64, a2, b2);
                }
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    uint32_t p0[2], p1[2], p2[2];
                    split4(fw[i], p0, p1, p2, more_w[i]);
                    if (MODE) fetch_w(i, left);
                    const uint32_t dst = ws + stage * STAGE + i * 32 * 128;
                    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst), "r"(p0[0]), "r"(p0[1]) : "memory");
                    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst + PART), "r"(p1[0]), "r"(p1[1]) : "memory");
                    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst + 2 * PART), "r"(p2[0]), "r"(p2[1]) : "memory");
                }
                if (MODE) next();
                tc_wait_st();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(full(stage));
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            };
            for (int b = 0; b + 1 < blocks; b++) {
                if (b + 1 < whole) block(b, std::integral_constant<int, 1>{});
                else block(b, std::integral_constant<int, 2>{});
            }
            block(blocks - 1, std::integral_constant<int, 0>{});
            uint32_t* mark = rows_s[count & 1];
            uint32_t any = 0;
#pragma unroll
            for (int i = 0; i < 2; i++) if (more_x[i] & 0xffffu) any = mark[1 + xr + 8 * i] = count;
#pragma unroll
            for (int i = 0; i < NB; i++) if (more_w[i] & 0xffffu) any = mark[1 + TM_ROWS + wr + 32 * i] = count;
            if (any) mark[0] = count;
            __syncwarp();
            if (lane == 0) mbar_arrive(rows_known(count & 1));
        }
    } else if (warp == W_MMA) {
        constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TM_ROWS >> 4) << 24);
        const uint64_t wd = umma_desc_sw128(base);
        uint32_t it = 0, stage = 0, phase = 0, flush = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            int bz, g, m0, m1;
            if (!find(tile, bz, g, m0, m1)) continue;
            for (int b = 0; b < blocks; b++, it++) {
                mbar_wait_lim(taken(0), (it & 1u) ^ 1u, fail);
                mbar_wait_lim(full(stage), phase, fail);
                tc_fence_after();
                const uint32_t a = tmem + stage * A_COLS, hi = tmem + ACC_COL, lo = hi + BN;
                const uint64_t w = wd + stage * (STAGE >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int i = 0; i < 4; i++) tc_mma_bf16_ts(hi, a + 8 * i, w + 2 * i, IDESC, i ? 1u : 0u);
                    tc_commit(sums(0));                      // read back while the other products are formed: one buffer is enough
                }
                __syncwarp();
                if (b % FLUSH == 0) {
                    mbar_wait_lim(taken(1), (flush++ & 1u) ^ 1u, fail);
                    tc_fence_after();
                }
                if (elect_one()) {
#pragma unroll
                    for (int i = 0; i < 28; i++) {           // parts (of X, of W), smallest products first, in four steps of 16 numbers each
                        constexpr int PX[7] = {2, 1, 2, 0, 1, 1, 0}, PW[7] = {1, 2, 0, 2, 1, 0, 1};
                        tc_mma_bf16_ts(lo, a + 32 * PX[i / 4] + 8 * (i % 4), w + (PW[i / 4] * (PART >> 4) + 2 * (i % 4)), IDESC, i ? 1u : (uint32_t)(b % FLUSH));
                    }
                    tc_commit(empty(stage));
                    if (b % FLUSH == FLUSH - 1 || b == blocks - 1) tc_commit(sums(1));
                }
                __syncwarp();
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
        if (__any_sync(0xffffffffu, *fail)) {                // products that nothing waited for
            if (elect_one()) { tc_commit(drained); mbar_drain(drained, 0); }
            __syncwarp();
        }
    } else {
        // ---- sums: TMEM lanes 32 q .., half of the columns of a tile
        constexpr int NC = BN / 2;
        const int q = warp & 3, half = (warp - W_ADD) >> 2;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16) + ACC_COL + NC * half;
        uint32_t it = 0, flush = 0, count = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            int bz, g, m0, m1;
            if (!find(tile, bz, g, m0, m1)) continue;
            float acc[NC];
#pragma unroll
            for (int c = 0; c < NC; c++) acc[c] = 0.f;
            count++;
            auto add = [&](int which) {
                tc_fence_after();
#pragma unroll
                for (int c0 = 0; c0 < NC; c0 += 8) {
                    uint32_t v[8];
                    ld_32x32b_x8(tl + which * BN + c0, v);
                    tc_wait_ld();
#pragma unroll
                    for (int c = 0; c < 8; c++) asm volatile("" : "+r"(v[c]));
#pragma unroll
                    for (int c = 0; c < 8; c += 2) add2(acc[c0 + c], acc[c0 + c + 1], __uint_as_float(v[c]), __uint_as_float(v[c + 1]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(taken(which));
            };
            for (int b = 0; b < blocks; b++, it++) {
                mbar_wait_lim(sums(0), it & 1u, fail);
                add(0);
                if (b % FLUSH == FLUSH - 1 || b == blocks - 1) {
                    mbar_wait_lim(sums(1), flush++ & 1u, fail);
                    add(1);
                }
            }
            const int row0 = m0 + 32 * q, n0 = tile / m_tiles * BN + NC * half;
            // what is not a finite number, what is so small that TMEM cut off more than fp32 does, and what has a row of numbers without parts is summed
            // again, behind the others, as one FMA chain
            constexpr uint32_t SMALL = 15u << 23, NOT_FINITE = 255u << 23;                  // 2^-112
            uint64_t again = 0;
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const uint32_t u = __float_as_uint(acc[c]) & 0x7fffffffu;
                if (u - SMALL >= NOT_FINITE - SMALL && u) again |= 1ull << c;
            }
            mbar_wait_lim(rows_known(count & 1), ((count - 1) >> 1) & 1u, fail);
            const volatile uint32_t* no_parts = rows_s[count & 1];
            if (no_parts[0] == count) {
                if (no_parts[1 + 32 * q + lane] == count) again = ~0ull;
#pragma unroll 1
                for (int c = 0; c < NC; c++) if (no_parts[1 + TM_ROWS + NC * half + c] == count) again |= 1ull << c;
            }
            again = n0 < p.N ? again & (~0ull >> (64 - min(NC, p.N - n0))) : 0;
            if (row0 + lane >= m1 || *fail) again = 0;
            if (*fail) {
#pragma unroll
                for (int c = 0; c < NC; c++) acc[c] = __int_as_float(0x7fc00000);
            }
            const float* bias = p.bias ? p.bias + (size_t)g * p.bias_gstride : nullptr;
            OT* out = (OT*)p.out + (size_t)bz * p.o_bs;
            const float* gate = p.gate ? p.gate + (size_t)bz * p.o_bs : nullptr;
            const bool quads = p.ldo % 4 == 0 && p.o_bs % 4 == 0 && ((uintptr_t)p.out) % (4 * sizeof(OT)) == 0;
            // two neighbouring lanes trade four of eight columns: a store writes 32 bytes of each of 16 rows instead of 16 bytes of 32
            const bool odd = lane & 1;
#pragma unroll
            for (int c = 0; c < NC; c += 8) {
                float give[4], keep[2][4];
#pragma unroll
                for (int e = 0; e < 4; e++) give[e] = __shfl_xor_sync(0xffffffffu, odd ? acc[c + e] : acc[c + 4 + e], 1);
#pragma unroll
                for (int e = 0; e < 4; e++) { keep[0][e] = odd ? give[e] : acc[c + e]; keep[1][e] = odd ? acc[c + 4 + e] : give[e]; }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int m = row0 + (lane & ~1) + h;
                    const int n = n0 + c + (odd ? 4 : 0);
                    if (m >= m1 || n >= p.N) continue;
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        v[e] = keep[h][e];
                        if (n + e >= p.N) continue;
                        v[e] += bias ? bias[n + e] : 0.f;
                        if (gate) v[e] *= 1.0f / (1.0f + expf(-gate[(size_t)m * p.ld_gate + n + e]));
                    }
                    OT* o = out + (size_t)m * p.ldo + n;
                    if (quads && n + 3 < p.N) {
                        if constexpr (sizeof(OT) == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
                        else *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; e++) if (n + e < p.N) stf(o + e, v[e]);
                    }
                }
            }
            if (__any_sync(0xffffffffu, again != 0)) {
                __syncwarp();                                // the stores above are other lanes'
                auto chain = [&](int m, int n) {
                    const float4* x = reinterpret_cast<const float4*>((const float*)p.X + (size_t)bz * p.x_bs + (size_t)(p.x_rows ? p.x_rows[m] / p.x_row_div : m) * p.ldx);
                    const float4* w = reinterpret_cast<const float4*>((const float*)p.W + (size_t)g * p.w_gstride + (size_t)bz * p.w_bs + (size_t)n * p.ldw);
                    float v = 0.f;
#pragma unroll 4
                    for (int k = 0; k < p.K / 4; k++) {
                        const float4 a = __ldg(x + k), b = __ldg(w + k);
                        v = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, v))));
                    }
                    v += bias ? bias[n] : 0.f;
                    if (gate) v *= 1.0f / (1.0f + expf(-gate[(size_t)m * p.ld_gate + n]));
                    stf(out + (size_t)m * p.ldo + n, v);
                };
                // a lane the sums of its row, or all lanes those of a row after the other, whichever takes fewer rounds
                const int mine = __popcll(again);
                if (__reduce_max_sync(0xffffffffu, mine) <= __reduce_add_sync(0xffffffffu, (mine + 31) / 32)) {
                    for (; again; again &= again - 1) chain(row0 + lane, n0 + __ffsll(again) - 1);
                } else {
                    for (uint32_t rows = __ballot_sync(0xffffffffu, mine > 0); rows; rows &= rows - 1) {
                        const int src = __ffs(rows) - 1;
                        const uint64_t cols = __shfl_sync(0xffffffffu, again, src);
                        for (int c = lane; c < NC; c += 32) if (cols >> c & 1) chain(row0 + src, n0 + c);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();                                         // nothing is in flight: every block's sums are read
    tc_fence_after();
    if (threadIdx.x == 0 && *fail) set_status(status);
    if (warp == W_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM) : "memory");
}

template <typename OT, int BN>
int launch(const AnyP& p, cudaStream_t st) {
    static P3DevFlags flags; bool& set = flags.cur();
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<OT, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f32tc_smem(BN));
        P3_CHECK_ARG(e == cudaSuccess, "gemm_any: shared memory attribute: %s", cudaGetErrorString(e));
        set = true;
    }
    const int64_t m_tiles = ((p.M + TM_ROWS - 1) / TM_ROWS + (p.seg ? p.n_groups : 0)) * p.nb, n_tiles = (p.N + BN - 1) / BN;
    const int64_t tiles = m_tiles * n_tiles;
    p3_launch_pdl(gemm_f32_tc_kernel<OT, BN>, dim3((unsigned)(tiles < 148 ? tiles : 148)), dim3(THREADS), f32tc_smem(BN), st, p, (int)m_tiles, (int)n_tiles, p3_status_word());
    return 0;
}
template <typename OT>
int launch_width(const AnyP& p, int bn, cudaStream_t st) {
    return bn == 32 ? launch<OT, 32>(p, st) : bn == 64 ? launch<OT, 64>(p, st) : launch<OT, 96>(p, st);
}
}  // namespace

// Columns of a tile: the width whose busiest SM is done first. Nanoseconds of a block of 64 numbers of k by width (128 rows, a tile an SM, K from 4096 to
// 8192), and about those of a tile beside its blocks. 128 columns took longer than 96 at every size: of 72 registers a thread the 96-wide
// kernel spills 128 bytes already.
int gemm_f32_tc_width(const void* any_p) {
    const AnyP& p = *static_cast<const AnyP*>(any_p);
    static const int width[3] = {96, 64, 32}, block[3] = {1450, 1090, 790};
    const int64_t m_tiles = ((p.M + TM_ROWS - 1) / TM_ROWS + (p.seg ? p.n_groups / 2 : 0)) * p.nb, blocks = (p.K + KB - 1) / KB;
    int best = 96;
    int64_t best_cost = INT64_MAX;
    for (int i = 0; i < 3; i++) {
        const int64_t waves = (m_tiles * ((p.N + width[i] - 1) / width[i]) + 147) / 148, cost = waves * (blocks * block[i] + 1500);
        if (cost < best_cost) { best = width[i]; best_cost = cost; }
    }
    return best;
}
int launch_gemm_f32_tc(const void* any_p, int out_f32, cudaStream_t st) {
    const AnyP& p = *static_cast<const AnyP*>(any_p);
    return out_f32 ? launch_width<float>(p, gemm_f32_tc_width(any_p), st) : launch_width<bf16>(p, gemm_f32_tc_width(any_p), st);
}
