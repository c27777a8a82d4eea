// p3_gemm_any: out[M,N] = X[M,K] * W[N,K]^T (+ bias) for ANY sizes, strides and alignments, operands fp32 or bf16, fp32
// accumulation. Two extras make it the mixture-of-experts workhorse: the rows of X can be gathered through an index list, and
// the rows can be cut into segments that each multiply with their own weight matrix (device-side segment offsets, so the host
// never learns how many tokens an expert received). A launch can also hold a batch of independent products over column blocks of
// X and out (one per attention head), with an optional sigmoid gate on the result.
//
// fp32 operands keep their 24 bits (no TF32): at most 16 rows as a stream of W, more in register tiles on the FMA pipes, each output one FMA chain
// in ascending k whatever the tile and the other rows; from 17 rows, 256 columns and K = 512 on as splits into bf16 parts on the tensor cores
// (gemm_f32_tc.cu: sums as near to 64 bits as the chain's or nearer, and one row's bits whatever the tile and the other rows there, but not the
// chain's: a row of a launch of 16 and of 17 rows differs in the last bits); a plain kernel for rows that are not 16-byte aligned. bf16 operands of aligned shapes run on the
// tensor cores through mma.sync m16n8k16 (fp32 accumulators); the dense bf16 projections with K % 8 == 0 go to the tcgen05
// kernel (p3_gemm) instead — this file is what is left: grouped expert products, fp32, and shapes p3_gemm does not take.
#include "gemm_any.cuh"
#include "../../include/phi3_b200.h"

namespace {
constexpr int BM = 64, BN = 64, BK = 16;

template <typename XT, typename WT, typename OT>
__global__ void __launch_bounds__(256) gemm_any_fma_kernel(AnyP p) {
    pdl_trigger();                                           // the next kernel may set up while this one runs ...
    pdl_wait();                                              // ... and this one touches memory only after its predecessors are done
    __shared__ __align__(16) float As[BK][BM + 4];
    __shared__ __align__(16) float Bs[BK][BN + 4];
    int g; int64_t m0, m1;
    const int bz = blockIdx.x % p.nb;
    if (!find_tile<BM>(p, blockIdx.x / p.nb, g, m0, m1)) return;
    const int n0 = blockIdx.y * BN, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const XT* X = (const XT*)p.X + (size_t)bz * p.x_bs;
    const WT* W = (const WT*)p.W + (size_t)g * p.w_gstride + (size_t)bz * p.w_bs;
    // this thread stages row (tid / 4) of each tile, k = (tid % 4) * 4 .. + 3
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    const int64_t am = m0 + lr;
    const XT* arow = nullptr;
    if (am < m1) arow = X + (size_t)(p.x_rows ? p.x_rows[am] / p.x_row_div : am) * p.ldx;
    const WT* brow = (n0 + lr < p.N) ? W + (size_t)(n0 + lr) * p.ldw : nullptr;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < p.K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = k0 + lk + j;
            As[lk + j][lr] = (arow && k < p.K) ? ldf(arow + k) : 0.f;
            Bs[lk + j][lr] = (brow && k < p.K) ? ldf(brow + k) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; k++) {
            const float4 a = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Bs[k][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    const float* bias = p.bias ? p.bias + (size_t)g * p.bias_gstride : nullptr;
    OT* out = (OT*)p.out + (size_t)bz * p.o_bs;
    const float* gate = p.gate ? p.gate + (size_t)bz * p.o_bs : nullptr;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int64_t m = m0 + ty * 4 + i;
        if (m >= m1) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx * 4 + j;
            if (n >= p.N) continue;
            float v = acc[i][j] + (bias ? bias[n] : 0.f);
            if (gate) v *= 1.0f / (1.0f + expf(-gate[(size_t)m * p.ld_gate + n]));
            stf(out + (size_t)m * p.ldo + n, v);
        }
    }
}

// fp32 operands with 16-byte aligned rows (K, pitches multiples of 4). Tile RM x RN, a thread owns TM x TN outputs; k-slabs of 16 travel
// global -> registers -> shared memory (transposed, two buffers), the next slab's loads in flight while this one is multiplied. The sum of
// an output is ONE FMA chain in ascending k like in gemm_any_fma_kernel (same bits), whatever the tile. The packed FMA takes two
// neighbouring columns per instruction, which halves the instructions to issue (1100 x 4096 x 2048: 477 us, 495 us with scalar FMAs, before
// the read-ahead). Bound by the FMA pipes (74 TFLOP/s): 46 TFLOP/s at 1100 x 4096 x 2048, 32 at 512 x 3072 x 1024 (2.6 tiles of 64 x 64 per
// SM), where the kernel for any alignment reached 11 (299 us -> 102 us).
__device__ __forceinline__ void fma2(float2& c, float a, float2 b) {
    uint64_t cc = *reinterpret_cast<uint64_t*>(&c), bb = *reinterpret_cast<uint64_t*>(&b), aa;
    asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(aa), "l"(bb));
    c = *reinterpret_cast<float2*>(&cc);
}
template <typename OT, int RM, int RN, int TM, int TN>
__global__ void __launch_bounds__((RM / TM) * (RN / TN)) gemm_f32_kernel(AnyP p) {
    pdl_wait();                                              // memory is touched only after the predecessors are done
    constexpr int NT = (RM / TM) * (RN / TN), TK = 16, GX = RN / TN;
    constexpr int LA = RM * TK / 4 / NT, LB = RN * TK / 4 / NT;      // 16-byte loads per thread and slab
    static_assert(LA * NT * 4 == RM * TK && LB * NT * 4 == RN * TK && TM % 4 == 0 && TN % 4 == 0, "tile shape");
    __shared__ __align__(16) float As[2][TK][RM + 4];
    __shared__ __align__(16) float Bs[2][TK][RN + 4];
    int g; int64_t m0, m1;
    const int bz = blockIdx.x % p.nb;
    if (!find_tile<RM>(p, blockIdx.x / p.nb, g, m0, m1)) return;
    const int n0 = blockIdx.y * RN, tid = threadIdx.x, tx = tid % GX, ty = tid / GX;
    const float* X = (const float*)p.X + (size_t)bz * p.x_bs;
    const float* W = (const float*)p.W + (size_t)g * p.w_gstride + (size_t)bz * p.w_bs;
    const int lr = tid >> 2, lk = (tid & 3) * 4;             // staging: rows lr, lr + NT / 4, ...; numbers lk .. lk + 3 of the slab
    const float* ap[LA]; const float* bp[LB];
#pragma unroll
    for (int i = 0; i < LA; i++) {
        const int64_t m = m0 + lr + i * (NT / 4);
        ap[i] = m < m1 ? X + (size_t)(p.x_rows ? p.x_rows[m] / p.x_row_div : m) * p.ldx + lk : nullptr;
    }
#pragma unroll
    for (int i = 0; i < LB; i++) {
        const int n = n0 + lr + i * (NT / 4);
        bp[i] = n < p.N ? W + (size_t)n * p.ldw + lk : nullptr;
    }
    float4 ra[LA], rb[LB];
    auto fetch = [&](int k0) {
        const bool in = k0 + lk < p.K;                       // K % 4 == 0: four numbers are inside or outside together
#pragma unroll
        for (int i = 0; i < LA; i++) ra[i] = ap[i] && in ? __ldg(reinterpret_cast<const float4*>(ap[i] + k0)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < LB; i++) rb[i] = bp[i] && in ? __ldg(reinterpret_cast<const float4*>(bp[i] + k0)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int i = 0; i < LA; i++) {
            const int r = lr + i * (NT / 4);
            As[buf][lk][r] = ra[i].x; As[buf][lk + 1][r] = ra[i].y; As[buf][lk + 2][r] = ra[i].z; As[buf][lk + 3][r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < LB; i++) {
            const int r = lr + i * (NT / 4);
            Bs[buf][lk][r] = rb[i].x; Bs[buf][lk + 1][r] = rb[i].y; Bs[buf][lk + 2][r] = rb[i].z; Bs[buf][lk + 3][r] = rb[i].w;
        }
    };
    // a thread's rows come in groups of four, RM / (TM / 4) apart (columns alike): the 16-byte reads of a warp are then neighbours
    constexpr int GM = RM / (TM / 4), GN = RN / (TN / 4);
    float2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = make_float2(0.f, 0.f);
    fetch(0);
    put(0);
    __syncthreads();
    for (int k0 = 0, buf = 0; k0 < p.K; k0 += TK, buf ^= 1) {
        const bool more = k0 + TK < p.K;
        if (more) fetch(k0 + TK);
        // with 64 sums per thread (one CTA per SM at most shapes) the operands of number k + 1 are read while those of k are multiplied:
        // 719 -> 595 us at 1024 x 3072 x 3072; the small tiles lose by it (99 -> 121 us at 200 x 1024 x 3072)
        constexpr int AHEAD = TM * TN >= 64 ? 1 : 0;
        float a[AHEAD + 1][TM]; float2 b[AHEAD + 1][TN / 2];
        auto read = [&](int k) {
#pragma unroll
            for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(a[k & AHEAD] + i) = *reinterpret_cast<const float4*>(&As[buf][k][(i / 4) * GM + ty * 4]);
#pragma unroll
            for (int j = 0; j < TN; j += 4) *reinterpret_cast<float4*>(b[k & AHEAD] + j / 2) = *reinterpret_cast<const float4*>(&Bs[buf][k][(j / 4) * GN + tx * 4]);
        };
        if (AHEAD) read(0);
#pragma unroll
        for (int k = 0; k < TK; k++) {
            if (!AHEAD) read(k);
            else if (k + 1 < TK) read(k + 1);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN / 2; j++) fma2(acc[i][j], a[k & AHEAD][i], b[k & AHEAD][j]);
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
    pdl_trigger();                                           // not before: the next kernel's waiting CTAs would take this one's places
    const float* bias = p.bias ? p.bias + (size_t)g * p.bias_gstride : nullptr;
    OT* out = (OT*)p.out + (size_t)bz * p.o_bs;
    const float* gate = p.gate ? p.gate + (size_t)bz * p.o_bs : nullptr;
    const bool quads = p.ldo % 4 == 0 && p.o_bs % 4 == 0 && ((uintptr_t)p.out) % (4 * sizeof(OT)) == 0;
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int64_t m = m0 + (i / 4) * GM + ty * 4 + i % 4;
        if (m >= m1) continue;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int n = n0 + (j / 4) * GN + tx * 4;
            if (n >= p.N) continue;
            float v[4] = {acc[i][j / 2].x, acc[i][j / 2].y, acc[i][j / 2 + 1].x, acc[i][j / 2 + 1].y};
#pragma unroll
            for (int e = 0; e < 4; e++) {
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
}

// fp32, at most 16 rows: a stream of W. A CTA owns 16 columns and the whole K; thread (column, row group) sums its outputs in one FMA chain
// (ascending k, the bits of the other fp32 kernels). W and X travel through a ring of 128-wide k-slabs by async copies. Bound by the
// chain (K x 4 cycles: 6.4 us at K = 3072) and, at 16 rows, by the shared-memory reads: 13 us for 1 x 1024 x 3072, 39 us for 16 x 3072 x
// 3072, where the tiles need 86 and 125 us.
constexpr int SF_COLS = 16, SF_K = 128, SF_ST = 6, SF_LD = SF_K + 4;
template <typename OT, int ROWS>                             // ROWS: rows of X, rounded up to 1, 2, 4, 8 or 16
__global__ void __launch_bounds__(128) gemm_f32_rows_kernel(AnyP p) {
    pdl_trigger();                                           // the next kernel may set up while this one runs ...
    pdl_wait();                                              // ... and this one touches memory only after its predecessors are done
    extern __shared__ __align__(16) float ring[];            // [SF_ST][16 rows of W | ROWS rows of X][SF_LD]
    constexpr int STAGE = (SF_COLS + ROWS) * SF_LD, PER = ROWS > 8 ? 2 : 1;
    const int bz = blockIdx.x % p.nb, n0 = (blockIdx.x / p.nb) * SF_COLS, tid = threadIdx.x, col = tid & 15, row = tid >> 4;
    const float* X = (const float*)p.X + (size_t)bz * p.x_bs;
    const float* W = (const float*)p.W + (size_t)bz * p.w_bs;
    const int slabs = (p.K + SF_K - 1) / SF_K;
    // staging: warp w brings rows w, w + 4, ... of the stage (16 of W, then those of X); rows and numbers that do not exist become zeros
    constexpr int RJ = (SF_COLS + ROWS + 3) / 4;
    const int lane4 = (tid & 31) * 4;
    const float* src[RJ];
#pragma unroll
    for (int j = 0; j < RJ; j++) {
        const int r = (tid >> 5) + 4 * j, m = r - SF_COLS;
        src[j] = nullptr;
        if (r < SF_COLS) { if (n0 + r < p.N) src[j] = W + (size_t)(n0 + r) * p.ldw + lane4; }
        else if (m < p.M) src[j] = X + (size_t)(p.x_rows ? p.x_rows[m] / p.x_row_div : m) * p.ldx + lane4;
    }
    auto stage = [&](int s) {
        float* dst = ring + (s % SF_ST) * STAGE + lane4;
#pragma unroll
        for (int j = 0; j < RJ; j++) {
            const int r = (tid >> 5) + 4 * j;
            const bool in = src[j] && s * SF_K + lane4 < p.K;
            if (r < SF_COLS + ROWS) cp_async16(smem_u32(dst + r * SF_LD), in ? src[j] + s * SF_K : W, in ? 16 : 0);
        }
    };
    for (int s = 0; s < SF_ST - 1; s++) { if (s < slabs) stage(s); cp_async_commit(); }
    float acc[PER] = {};
    for (int s = 0; s < slabs; s++) {
        cp_async_wait<SF_ST - 2>();
        __syncthreads();                                     // slab s is there for everyone, slab s - 1 is read
        if (s + SF_ST - 1 < slabs) stage(s + SF_ST - 1);
        cp_async_commit();
        if (row < ROWS) {
            const float* w = ring + (s % SF_ST) * STAGE + col * SF_LD;
            const float* x = ring + (s % SF_ST) * STAGE + (SF_COLS + row) * SF_LD;
#pragma unroll
            for (int k = 0; k < SF_K; k += 4) {
                const float4 b = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
                for (int i = 0; i < PER; i++) {
                    const float4 a = *reinterpret_cast<const float4*>(x + i * 8 * SF_LD + k);
                    acc[i] = fmaf(a.x, b.x, acc[i]); acc[i] = fmaf(a.y, b.y, acc[i]); acc[i] = fmaf(a.z, b.z, acc[i]); acc[i] = fmaf(a.w, b.w, acc[i]);
                }
            }
        }
    }
    cp_async_wait<0>();
    const int n = n0 + col;
    const float* gate = p.gate ? p.gate + (size_t)bz * p.o_bs : nullptr;
    if (row >= ROWS || n >= p.N) return;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int m = row + 8 * i;
        if (m >= p.M) continue;
        float v = acc[i] + (p.bias ? p.bias[n] : 0.f);
        if (gate) v *= 1.0f / (1.0f + expf(-gate[(size_t)m * p.ld_gate + n]));
        stf((OT*)p.out + (size_t)bz * p.o_bs + (size_t)m * p.ldo + n, v);
    }
}

template <typename OT, int RM, int RN, int TM, int TN>
void launch_f32(const AnyP& p, cudaStream_t st) {
    const unsigned mt = (unsigned)((p.M + RM - 1) / RM) + (p.seg ? (unsigned)p.n_groups : 0u);
    p3_launch_pdl(gemm_f32_kernel<OT, RM, RN, TM, TN>, dim3(mt * (unsigned)p.nb, (unsigned)((p.N + RN - 1) / RN)),
                  dim3((RM / TM) * (RN / TN)), (size_t)0, st, p);
}
template <typename OT, int ROWS>
int launch_f32_rows(const AnyP& p, cudaStream_t st) {
    constexpr size_t bytes = sizeof(float) * SF_ST * (SF_COLS + ROWS) * SF_LD;
    static P3DevFlags flags; bool& set = flags.cur();
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<OT, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        P3_CHECK_ARG(e == cudaSuccess, "gemm_any: shared memory attribute: %s", cudaGetErrorString(e));
        set = true;
    }
    p3_launch_pdl(gemm_f32_rows_kernel<OT, ROWS>, dim3((unsigned)((p.N + SF_COLS - 1) / SF_COLS * p.nb)), dim3(128), bytes, st, p);
    return 0;
}
// Which tile? Times of one k-step on B200 in ns, lone CTA on an SM | per CTA when several share one: 128 x 128 94 | 105, 64 x 64 47 | 29,
// 32 x 32 41 | 11 (measured from 64 x 4096 x 3072 to 1100 x 4096 x 2048); the busiest SM decides. 64 x 128, 64 x 64 with 4 x 4 outputs per
// thread and 32 x 64 were behind one of these three at every size tried.
int f32_tile(const AnyP& p) {
    if (!p.seg && p.M <= 16) return 16;
    auto cost = [&](int r, int64_t alone, int64_t shared) -> int64_t {
        if (((int64_t)p.N + r - 1) / r > 65535) return INT64_MAX;        // more column tiles than the grid's second dimension holds
        const int64_t tiles = ((p.M + r - 1) / r + (p.seg ? p.n_groups / 2 : 0)) * ((p.N + r - 1) / r) * p.nb, per_sm = (tiles + 147) / 148;
        return alone > per_sm * shared ? alone : per_sm * shared;
    };
    const int64_t c128 = cost(128, 94, 105), c64 = cost(64, 47, 29), c32 = cost(32, 41, 11);
    return c128 <= c64 && c128 <= c32 ? 128 : c64 <= c32 ? 64 : 32;
}
template <typename OT>
int dispatch_f32(const AnyP& p, cudaStream_t st) {
    const int tile = f32_tile(p);
    if (tile == 16) {
        if (p.M <= 1) return launch_f32_rows<OT, 1>(p, st);
        if (p.M <= 2) return launch_f32_rows<OT, 2>(p, st);
        if (p.M <= 4) return launch_f32_rows<OT, 4>(p, st);
        if (p.M <= 8) return launch_f32_rows<OT, 8>(p, st);
        return launch_f32_rows<OT, 16>(p, st);
    }
    if (tile == 128) launch_f32<OT, 128, 128, 8, 8>(p, st);
    else if (tile == 64) launch_f32<OT, 64, 64, 8, 4>(p, st);
    else launch_f32<OT, 32, 32, 4, 4>(p, st);
    return 0;
}

// bf16 x bf16 on the tensor cores: 64 x 64 tile, 4 warps (2 x 2), each warp 32 x 32 = 2 x 4 MMAs of m16n8k16 per 16-wide k
// step; operands staged through shared memory as bf16 (row-major [row][k], 16-byte chunks, K % 8 == 0 and 16-byte aligned rows
// required by the launcher). Same tile walk, gather and segment logic as the FMA kernel. A k-slab is 128 elements: 16 lanes read
// the 256 contiguous bytes of one row, so that with few rows, where the kernel is a stream of W, DRAM sees bursts instead of
// 64-byte pieces of 64 rows; the next slab's loads are in flight while this one is multiplied.
// TK = k elements per stage: 128, or 64 for products with K <= 64 (the per-head products of an attention mixer), which would
// otherwise multiply a half-empty slab and hold twice the staging registers.
template <typename OT, int TK>
__global__ void __launch_bounds__(128) gemm_any_mma_kernel(AnyP p) {
    pdl_trigger();                                           // the next kernel may set up while this one runs ...
    pdl_wait();                                              // ... and this one touches memory only after its predecessors are done
    __shared__ __align__(16) bf16 As[BM][TK + 8];
    __shared__ __align__(16) bf16 Bs[BN][TK + 8];
    int g; int64_t m0, m1;
    const int bz = blockIdx.x % p.nb;
    if (!find_tile<BM>(p, blockIdx.x / p.nb, g, m0, m1)) return;
    const int n0 = blockIdx.y * BN, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const bf16* X = (const bf16*)p.X + (size_t)bz * p.x_bs;
    const bf16* W = (const bf16*)p.W + (size_t)g * p.w_gstride + (size_t)bz * p.w_bs;
    // staging: 64 rows x TK / 8 chunks of 8 elements per operand; LPR lanes per row, RPR rows per round of the CTA, NR rounds;
    // round j: row RPR j + (32 / LPR) warp + lane / LPR, chunk lane % LPR
    constexpr int LPR = TK / 8, RPR = 128 / LPR, NR = BM / RPR;
    const int srow0 = (32 / LPR) * warp + lane / LPR, schunk = (lane % LPR) * 8;
    int64_t aoff[NR];                                       // element offset of this thread's A row in round j, -1: no such row
#pragma unroll
    for (int j = 0; j < NR; j++) {
        const int64_t am = m0 + srow0 + RPR * j;
        aoff[j] = (am < m1) ? (int64_t)(p.x_rows ? p.x_rows[am] / p.x_row_div : am) * p.ldx : -1;
    }
    const bf16* brow0 = W + (size_t)(n0 + srow0) * p.ldw;
    float acc[2][4][4] = {};
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 ra[NR], rb[NR];
    auto fetch = [&](int k0) {
        const int k = k0 + schunk;
        const bool in = k < p.K;                           // K % 8 == 0: a chunk is inside or outside as a whole
#pragma unroll
        for (int j = 0; j < NR; j++) {
            ra[j] = (aoff[j] >= 0 && in) ? __ldg(reinterpret_cast<const uint4*>(X + aoff[j] + k)) : zero;
            rb[j] = (n0 + srow0 + RPR * j < p.N && in) ? ldg_nc_v4(brow0 + (size_t)(RPR * j) * p.ldw + k) : zero;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < p.K; k0 += TK) {
#pragma unroll
        for (int j = 0; j < NR; j++) {
            *reinterpret_cast<uint4*>(&As[srow0 + RPR * j][schunk]) = ra[j];
            *reinterpret_cast<uint4*>(&Bs[srow0 + RPR * j][schunk]) = rb[j];
        }
        __syncthreads();
        if (k0 + TK < p.K) fetch(k0 + TK);
#pragma unroll
        for (int kk = 0; kk < TK; kk += 16) {
            uint32_t a[2][4], b[4][2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int r = wm + i * 16 + (lane >> 2), c = kk + (lane & 3) * 2;
                a[i][0] = *reinterpret_cast<const uint32_t*>(&As[r][c]);
                a[i][1] = *reinterpret_cast<const uint32_t*>(&As[r + 8][c]);
                a[i][2] = *reinterpret_cast<const uint32_t*>(&As[r][c + 8]);
                a[i][3] = *reinterpret_cast<const uint32_t*>(&As[r + 8][c + 8]);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int r = wn + j * 8 + (lane >> 2), c = kk + (lane & 3) * 2;
                b[j][0] = *reinterpret_cast<const uint32_t*>(&Bs[r][c]);
                b[j][1] = *reinterpret_cast<const uint32_t*>(&Bs[r][c + 8]);
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma_bf16_16816(acc[i][j], a[i], b[j][0], b[j][1]);
        }
        __syncthreads();
    }
    const float* bias = p.bias ? p.bias + (size_t)g * p.bias_gstride : nullptr;
    OT* out = (OT*)p.out + (size_t)bz * p.o_bs;
    const float* gate = p.gate ? p.gate + (size_t)bz * p.o_bs : nullptr;
    // a thread holds pairs of neighbouring columns: one 4- or 8-byte store per pair where the pair is aligned
    const bool pair_ok = (p.ldo % 2 == 0) && (p.o_bs % 2 == 0) && (((uintptr_t)p.out) % (2 * sizeof(OT)) == 0);
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int hlf = 0; hlf < 2; hlf++) {
                const int64_t m = m0 + wm + i * 16 + (lane >> 2) + hlf * 8;
                const int n = n0 + wn + j * 8 + (lane & 3) * 2;
                if (m >= m1 || n >= p.N) continue;
                float v0 = acc[i][j][hlf * 2] + (bias ? bias[n] : 0.f);
                float v1 = (n + 1 < p.N) ? acc[i][j][hlf * 2 + 1] + (bias ? bias[n + 1] : 0.f) : 0.f;
                if (gate) {
                    v0 *= 1.0f / (1.0f + expf(-gate[(size_t)m * p.ld_gate + n]));
                    if (n + 1 < p.N) v1 *= 1.0f / (1.0f + expf(-gate[(size_t)m * p.ld_gate + n + 1]));
                }
                OT* o = out + (size_t)m * p.ldo + n;
                if (pair_ok && n + 1 < p.N) {
                    if constexpr (sizeof(OT) == 4) *reinterpret_cast<float2*>(o) = make_float2(v0, v1);
                    else *reinterpret_cast<uint32_t*>(o) = pack_bf16(v0, v1);
                } else {
                    stf(o, v0);
                    if (n + 1 < p.N) stf(o + 1, v1);
                }
            }
}
}  // namespace

bool gemm_grouped_ok(const p3_gemm_any_args* a);               // gemm_tc.cu
int launch_gemm_grouped(const p3_gemm_any_args* a, cudaStream_t st);
int gemm_f32_tc_width(const void* any_p);                      // gemm_f32_tc.cu
int launch_gemm_f32_tc(const void* any_p, int out_f32, cudaStream_t st);

static AnyP any_params(const p3_gemm_any_args* a) {
    AnyP p{a->X, a->ldx, a->x_rows, a->x_row_div, a->W, a->ldw, a->w_group_stride, a->bias, a->bias_group_stride,
           a->out, a->ldo, a->M, a->N, a->K, a->seg_offsets, a->seg_offsets ? a->n_groups : 1,
           a->n_batch > 1 ? a->n_batch : 1, a->x_batch_stride, a->w_batch_stride, a->out_batch_stride, a->gate, a->ld_gate};
    if (p.nb == 1) p.x_bs = p.w_bs = p.o_bs = 0;
    return p;
}
static bool aligned_f32(const p3_gemm_any_args* a, int nb) {
    return a->x_f32 && a->K % 4 == 0 && a->ldx % 4 == 0 && a->ldw % 4 == 0 && a->w_group_stride % 4 == 0 &&
           (nb == 1 || (a->x_batch_stride % 4 == 0 && a->w_batch_stride % 4 == 0)) && (((uintptr_t)a->X | (uintptr_t)a->W) & 15) == 0;
}
// fp32 on the tensor cores (gemm_f32_tc.cu): dense products from 17 rows on at every size timed (rows, columns, K: 17 x 1024 x 512 10.9 us, 16.4 on the
// FMA tiles; 17 x 256 x 3072 41 and 86; 512 x 3072 x 1024 29.7 and 102). Below 512 numbers of k or 256 columns a product stays one FMA chain, the bits of the kernel for any alignment: gates, routers,
// low ranks, products per head.
// Segments of few rows fill a small part of 128-row tiles: where that makes more tiles than the SMs take at once, FMA tiles of 32 rows are faster for short
// products (64 segments, 512 columns, FMA and tensor cores: K = 512, 16 rows a segment 51 and 63 us, 64 rows 78 and 76; K = 768, 16 rows 77 and 77;
// K = 1024, 4 rows 87 and 93, 16 rows 101 and 89; K = 2048, 4 rows 167 and 156). With few tiles the tensor cores were faster at every size (8
// segments of 512 columns, K = 1024, 17 to 512 rows: 31 .. 41 and 18 .. 33).
static bool few_rows_a_segment(const p3_gemm_any_args* a) {
    const int64_t rows = a->K < 768 ? 32 : a->K < 1024 ? 16 : a->K < 1536 ? 8 : 0;
    return a->seg_offsets && (int64_t)a->n_groups * (((int64_t)a->N + 63) / 64) > 96 && a->M <= a->n_groups * rows;
}
static bool f32_tc(const p3_gemm_any_args* a, const AnyP& p) {
    const int64_t tiles = ((a->M + 127) / 128 + (a->seg_offsets ? a->n_groups : 0)) * p.nb * (((int64_t)a->N + 31) / 32);
    return !a->force_fma && a->M > 16 && a->N >= 256 && a->K >= 512 && tiles < (1ll << 30) && !few_rows_a_segment(a);
}
extern "C" int p3_gemm_any_tile(const p3_gemm_any_args* a) {
    const AnyP p = any_params(a);
    return !aligned_f32(a, p.nb) ? 0 : f32_tc(a, p) ? -gemm_f32_tc_width(&p) : f32_tile(p);
}

extern "C" int p3_gemm_any(const p3_gemm_any_args* a, cudaStream_t st) {
    P3_CHECK_ARG(a && a->X && a->W && a->out, "gemm_any: null operand");
    P3_CHECK_ARG(a->M >= 0 && a->N >= 1 && a->K >= 1 && a->M < (1ll << 30), "gemm_any: bad sizes");
    P3_CHECK_ARG(!a->seg_offsets || a->n_groups >= 1, "gemm_any: segments need n_groups >= 1");
    P3_CHECK_ARG(!a->x_rows || a->x_row_div >= 1, "gemm_any: gather needs x_row_div >= 1");
    P3_CHECK_ARG(a->x_f32 == a->w_f32, "gemm_any: X and W must have the same element type");
    if (a->M == 0) return 0;
    if (gemm_grouped_ok(a)) return launch_gemm_grouped(a, st);
    const AnyP p = any_params(a);
    const int nb = p.nb;
    P3_CHECK_ARG(nb <= 65535, "gemm_any: too many products in a batch");
    const unsigned mt = (unsigned)((a->M + BM - 1) / BM) + (a->seg_offsets ? (unsigned)a->n_groups : 0u);
    const dim3 grid(mt * (unsigned)nb, (unsigned)((a->N + BN - 1) / BN));
    const bool vec = aligned_f32(a, nb);
    if (vec && f32_tc(a, p)) {
        if (launch_gemm_f32_tc(&p, a->out_f32, st)) return -1;
    } else if (vec) {
        const int rc = a->out_f32 ? dispatch_f32<float>(p, st) : dispatch_f32<bf16>(p, st);
        if (rc) return rc;
    } else if (a->x_f32) {
        if (a->out_f32) p3_launch_pdl(gemm_any_fma_kernel<float, float, float>, dim3(grid), dim3(256), (size_t)(0), st, p);
        else p3_launch_pdl(gemm_any_fma_kernel<float, float, bf16>, dim3(grid), dim3(256), (size_t)(0), st, p);
    } else {
        const bool tc = a->K % 8 == 0 && a->ldx % 8 == 0 && a->ldw % 8 == 0 && a->w_group_stride % 8 == 0 &&
                        (nb == 1 || (a->x_batch_stride % 8 == 0 && a->w_batch_stride % 8 == 0)) &&
                        ((uintptr_t)a->X & 15) == 0 && ((uintptr_t)a->W & 15) == 0 && (!a->force_fma || a->force_fma == 2);
        if (tc) {
            if (a->K <= 64) {
                if (a->out_f32) p3_launch_pdl(gemm_any_mma_kernel<float, 64>, dim3(grid), dim3(128), (size_t)(0), st, p);
                else p3_launch_pdl(gemm_any_mma_kernel<bf16, 64>, dim3(grid), dim3(128), (size_t)(0), st, p);
            } else if (a->out_f32) p3_launch_pdl(gemm_any_mma_kernel<float, 128>, dim3(grid), dim3(128), (size_t)(0), st, p);
            else p3_launch_pdl(gemm_any_mma_kernel<bf16, 128>, dim3(grid), dim3(128), (size_t)(0), st, p);
        } else {
            if (a->out_f32) p3_launch_pdl(gemm_any_fma_kernel<bf16, bf16, float>, dim3(grid), dim3(256), (size_t)(0), st, p);
            else p3_launch_pdl(gemm_any_fma_kernel<bf16, bf16, bf16>, dim3(grid), dim3(256), (size_t)(0), st, p);
        }
    }
    P3_CHECK_LAUNCH("gemm_any");
    return 0;
}
