// Dense bf16 GEMM on 5th-gen tensor cores: out[M,N] = X[M,K] . W[N,K]^T (+ fused epilogue).
// Replaces every prefill / ViT / projector nn.Linear and the patch-embed conv of the reference
// (phi.py:140-143,155-156,186-192,391,437-438,465-466,604).
//
// Structure (one CTA per SM, persistent over output tiles, 128 x BN tile, BK = 64):
//   warp 0   : TMA producer  — cp.async.bulk.tensor 2D, 128B swizzle, STAGES-deep mbarrier ring
//   warp 1   : MMA issuer    — one elected lane issues tcgen05.mma.cta_group::1.kind::f16
//                              (UMMA 128 x BN x 16), accumulators in TMEM (2 x BN columns, double buffered)
//   warp 2   : TMEM allocator
//   warps 4-11: epilogue     — tcgen05.ld 32x32b (two warps per TMEM lane quarter, half the columns each),
//                              fused bias / GELU / residual / SwiGLU / fp32 / row scatter
// Both operands are K-major (activations [M,K] and nn.Linear weights [N,K]), so no transposes.
#include "tc_common.cuh"
#include "../../include/phi3_b200.h"
#include <cstdlib>
#include <cstring>

struct GemmEpi {
    const bf16* bias;
    void* out;
    int64_t ldo;
    const void* resid;
    const int32_t* row_map;
    int kind;
    // fused RMSNorm (phi.py:478-479) of the INPUT rows: the gain is folded into W at load time, the per-row scale
    // rsqrt(sum_c ss_in[row][c] / K + eps) multiplies the accumulators; ss_in = sum-of-squares partials of the rows of X
    const float* ss_in; int n_ss_in; float eps;
    // RESIDUAL: sum of squares of every 32-column chunk written, ss_out[row][N/32] (feeds the next GEMM's ss_in)
    float* ss_out;
    // P3_EPI_ROPE_KV: SuRoPE (phi.py:418-423,487-507) + paged KV write (phi.py:542-548) on the qkv projection. W rows are
    // permuted per head so that every 32-column chunk holds 16 dims [16j,16j+16) and their rotary partners [half+16j, +16).
    const float *cosT, *sinT; int64_t tab_bstride;
    int L, n_heads, n_kv, hd, past, row_div, write_cache;
    const int32_t* past_dev;
    bf16* pool; const int32_t* block_table; int bt_stride;
    // split-K (small M: few output tiles, the GEMM is a weight stream and one SM ingests only ~1/148 of HBM bandwidth, so every
    // SM must stream): `ksplit` CTAs share an output tile, each accumulates a K slice, dumps fp32 partials to `ws`
    // [tile][ksplit][128][BN]; the last one to arrive (per-tile counter) sums them in slice order and runs the epilogue.
    int ksplit; float* ws; int* counters; int64_t ws_bytes;
    // outputs larger than the L2 can keep (batched prefill): store with the streaming (evict-first) policy so that the
    // write-allocated lines do not push the resident W band / X rows out of L2 (ncu: 2.7-3.1x DRAM over-read without it)
    int stream_out;
    int band_mb;                                           // rasterisation band (MB of W kept L2-resident); 0 = default
    // grouped product (mixture of experts): rows [seg[g], seg[g + 1]) of X multiply with the N rows of W that begin at g * w_rows
    const int32_t* seg; int n_groups, w_rows;
    // gated unit of [gate | up] weights, glu_f rows each (P3_EPI_GLU, pair kernel only)
    int glu_f, glu_act; float glu_limit, glu_alpha;
};
__device__ __forceinline__ void st_out16(void* p, const uint4& v, int stream) {
    if (stream) __stcs(reinterpret_cast<uint4*>(p), v); else *reinterpret_cast<uint4*>(p) = v;
}
#define P3_SPLITK_COUNTER_BYTES 4096
#define P3_EPI_ROPE_KV 8

__device__ __forceinline__ float epi_act(int kind, float x) {
    // CLIP fc1 and the projector run in fp32 in the reference (fp32 activations x bf16 weights
    // promote to fp32), so the activation is applied to the unrounded accumulator.
    if (kind == P3_EPI_QGELU) return __fdividef(x, 1.f + __expf(-1.702f * x));
    if (kind == P3_EPI_GELU) return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
    return x;
}

// Tile rasterisation: n-fastest inside bands of `nb` n-tiles so the band's W tiles (nb * BN * K * 2 B) stay
// L2-resident while A streams through once per band. (m-fastest order re-read A once per n-tile: ncu showed
// 2.1 GB of DRAM reads for a 157 MB problem.) Band size, ncu DRAM reads in the batched prefill (M = 16384):
// 48 MB bands -> qkv 727 MB, gate_up 733 MB; 32 MB -> 359 / 557 MB (a 48 MB band does not survive next to the X
// stream and the write-allocated output); for K = 8192 (4 MB per W tile, 74 concurrent tiles stream 72 MB per wave)
// nothing is retained across waves whatever the band, and the widest band that covers N (48 MB) reads least.
__device__ __forceinline__ void tile_coords(int tile, int m_tiles, int n_tiles, int nb, int& mt, int& nt) {
    const int band_tiles = nb * m_tiles;
    const int band = tile / band_tiles, rem = tile - band * band_tiles;
    const int nb_this = min(nb, n_tiles - band * nb);
    mt = rem / nb_this;
    nt = band * nb + rem - mt * nb_this;
}
__host__ __device__ __forceinline__ int band_width(int K, int BN, int n_tiles, int band_mb = 0) {
    long long per = (long long)BN * K * 2;
    int nb = (int)(((long long)(band_mb > 0 ? band_mb : (per <= (2ll << 20) ? 32 : 48)) << 20) / (per > 0 ? per : 1));
    return nb < 1 ? 1 : (nb > n_tiles ? n_tiles : nb);
}

// Grouped products: which rows a CTA multiplies is known on the device only. Every CTA forms the running count of row tiles of the groups (in
// shared memory, behind the dependency wait) and finds the group of a tile by bisection; tiles of one group follow one another, column tiles
// fastest, so that the CTAs in flight share rows of X and stream W.
constexpr int GROUPS_MAX = 1024;
struct GroupTable { int tiles[GROUPS_MAX + 1], row[GROUPS_MAX + 1]; };     // row tiles before group g; first row of group g
struct GroupTile { int m, m_end, w, n; };                                  // rows [m, m_end) of X, rows of W from w + n on
__device__ __forceinline__ void group_table(GroupTable& t, const int32_t* seg, int n_groups, int M, int bm) {    // one warp; rows from M on are nobody's
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int g0 = 0; g0 <= n_groups; g0 += 32) {
        const int g = g0 + lane, a = g <= n_groups ? min(seg[g], M) : 0, b = g < n_groups ? min(seg[g + 1], M) : a;
        int c = (b - a + bm - 1) / bm;
        const int own = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, c, o); if (lane >= o) c += v; }
        if (g <= n_groups) { t.tiles[g] = before + c - own; t.row[g] = a; }
        before += __shfl_sync(0xffffffffu, c, 31);
    }
}
__device__ __forceinline__ GroupTile group_tile(const GroupTable& t, int n_groups, int w_rows, int tile, int n_tiles, int bm, int bn) {
    const int mt = tile / n_tiles;
    int lo = 0, hi = n_groups;                             // tiles[lo] <= mt < tiles[hi]
    while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (t.tiles[mid] <= mt) lo = mid; else hi = mid; }
    return {t.row[lo] + (mt - t.tiles[lo]) * bm, t.row[lo + 1], lo * w_rows, (tile - mt * n_tiles) * bn};
}

constexpr int EPI_SMEM = 8 * 2048;                           // the epilogue warps' blocks of output
template <int BN>
struct TcCfg {
    static constexpr int BM = 128, BK = 64;
    static constexpr int STAGES = (BN == 256) ? 4 : (BN == 128 ? 6 : 8);
    static constexpr int A_BYTES = BM * BK * 2;
    static constexpr int B_BYTES = BN * BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int TMEM_COLS = 2 * BN;
    static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256 + EPI_SMEM;
    // kind::f16 instruction descriptor: D=f32 (1<<4), A=B=bf16 (1<<7, 1<<10), K-major both, N>>3 @17, M>>4 @24
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
};

// per-row RMSNorm scale from the producer's partial sums; 1 when the GEMM is not normed. A row's lane adds the sums of its quadruples in
// ascending order, whatever the tile: one row has one scale. Four lanes bring 64 bytes of a row, eight
// rows at a time, and hand the quadruples over through the warp's block of shared memory: reads of whole sectors (a lane reading its own row:
// 781 x 16384 x 3072 with 96 partial sums a row took 95 us, 81 without).
__device__ __forceinline__ float epi_row_scale(const GemmEpi& ep, uint8_t* sb, int row0, int m_end, int K) {
    if (!ep.ss_in) return 1.f;
    const int lane = threadIdx.x & 31, sub = lane >> 2, part = lane & 3, n = ep.n_ss_in;
    float s = 0.f;
    if ((n & 3) == 0) {
        const float* p = ep.ss_in + (size_t)(row0 + sub) * n + 4 * part;
        float* q = reinterpret_cast<float*>(sb);               // [block of 16 numbers][row][4]
        for (int c0 = 0; c0 < n; c0 += 32) {
            float4 f[2][4];
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    f[h][i] = c0 + 16 * h + 4 * part < n && row0 + 8 * i + sub < m_end
                                  ? __ldcg(reinterpret_cast<const float4*>(p + (size_t)8 * i * n + c0 + 16 * h)) : make_float4(0.f, 0.f, 0.f, 0.f);
            __syncwarp();                                      // the block before is read
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int i = 0; i < 4; i++) q[h * 128 + (8 * i + sub) * 4 + part] = (f[h][i].x + f[h][i].y) + (f[h][i].z + f[h][i].w);
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float4 t = *reinterpret_cast<const float4*>(q + h * 128 + lane * 4);      // zeros behind the last
                s += t.x; s += t.y; s += t.z; s += t.w;
            }
        }
    } else if (row0 + lane < m_end) {
        const float* p = ep.ss_in + (size_t)(row0 + lane) * n;
        for (int c = 0; c < n; c++) s += __ldcg(p + c);
    }
    return rsqrtf(s / (float)K + ep.eps);
}

// P3_EPI_ROPE_KV, per output row (token): everything that does not depend on the column chunk — computed once per tile,
// not once per 32-column chunk (the integer divisions by run-time L / page / hd cost more than the rotation itself)
struct RopeRow {
    bf16 *qrow, *kd, *vd;
    const float *cr, *sr;                                      // cos / sin rows of this token's position
};
__device__ __forceinline__ RopeRow epi_rope_row(const GemmEpi& ep, int row) {
    RopeRow r;
    const int hd = ep.hd, half = hd / 2;
    const int b = row / ep.L, pos = (ep.past_dev ? *ep.past_dev : ep.past) + (row - b * ep.L);
    const int crow = b / ep.row_div;
    r.qrow = reinterpret_cast<bf16*>(ep.out) + (size_t)row * ep.ldo;
    r.kd = r.vd = nullptr;
    if (ep.write_cache) {
        const int pg = pos / P3_PAGE;
        const int page = ep.block_table[(size_t)crow * ep.bt_stride + pg];
        r.kd = ep.pool + (size_t)page * kv_page_elems(ep.n_kv, hd) + (size_t)(pos - pg * P3_PAGE) * hd;
        r.vd = r.kd + (size_t)ep.n_kv * P3_PAGE * hd;
    }
    r.cr = ep.cosT + (size_t)crow * ep.tab_bstride + (size_t)pos * half;
    r.sr = ep.sinT + (size_t)crow * ep.tab_bstride + (size_t)pos * half;
    // the rows are read chunk by chunk after the accumulators arrive: have them in L1 by then (each miss is ~1 us of
    // exposed epilogue when a CTA has only one or two tiles)
    for (int o = 0; o < half * 4; o += 128) {
        asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(r.cr) + o));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(r.sr) + o));
    }
    return r;
}
// one 32-column chunk of the (row-permuted) qkv projection
__device__ __forceinline__ void epi_rope32(const GemmEpi& ep, const RopeRow& rr, int n0, float rs, const uint32_t* acc) {
    const int hd = ep.hd, half = hd / 2;
    const int head = n0 / hd, j = (n0 - head * hd) / 32;
    uint4 o1[2], o2[2];
    uint32_t* u1 = reinterpret_cast<uint32_t*>(o1);
    uint32_t* u2 = reinterpret_cast<uint32_t*>(o2);
    if (head < ep.n_heads + ep.n_kv) {                        // q or k head: rotate
        const float* cr = rr.cr + 16 * j;
        const float* sr = rr.sr + 16 * j;
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            const float4 c4 = __ldg(reinterpret_cast<const float4*>(cr + i)), s4 = __ldg(reinterpret_cast<const float4*>(sr + i));
            const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
            float a1[4], a2[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {                     // the projection output is bf16 in the reference flow, rope runs in fp32
                const float x1 = bf16_round(__uint_as_float(acc[i + e]) * rs), x2 = bf16_round(__uint_as_float(acc[16 + i + e]) * rs);
                a1[e] = x1 * cs[e] - x2 * sn[e];
                a2[e] = x2 * cs[e] + x1 * sn[e];
            }
            u1[i / 2] = pack_bf16(a1[0], a1[1]); u1[i / 2 + 1] = pack_bf16(a1[2], a1[3]);
            u2[i / 2] = pack_bf16(a2[0], a2[1]); u2[i / 2 + 1] = pack_bf16(a2[2], a2[3]);
        }
        bf16* d1 = rr.qrow + head * hd + 16 * j;
        st_out16(d1, o1[0], ep.stream_out); st_out16(d1 + 8, o1[1], ep.stream_out);
        st_out16(d1 + half, o2[0], ep.stream_out); st_out16(d1 + half + 8, o2[1], ep.stream_out);
        if (rr.kd && head >= ep.n_heads) {
            bf16* k = rr.kd + (size_t)(head - ep.n_heads) * P3_PAGE * hd + 16 * j;
            reinterpret_cast<uint4*>(k)[0] = o1[0]; reinterpret_cast<uint4*>(k)[1] = o1[1];
            reinterpret_cast<uint4*>(k + half)[0] = o2[0]; reinterpret_cast<uint4*>(k + half)[1] = o2[1];
        }
    } else {                                                   // v head: 32 plain columns
#pragma unroll
        for (int i = 0; i < 8; i++) {
            u1[i] = pack_bf16(__uint_as_float(acc[2 * i]) * rs, __uint_as_float(acc[2 * i + 1]) * rs);
            u2[i] = pack_bf16(__uint_as_float(acc[16 + 2 * i]) * rs, __uint_as_float(acc[17 + 2 * i]) * rs);
        }
        bf16* d = rr.qrow + n0;
        st_out16(d, o1[0], ep.stream_out); st_out16(d + 8, o1[1], ep.stream_out);
        st_out16(d + 16, o2[0], ep.stream_out); st_out16(d + 24, o2[1], ep.stream_out);
        if (rr.vd) {
            bf16* v = rr.vd + (size_t)(head - ep.n_heads - ep.n_kv) * P3_PAGE * hd + 32 * j;
            reinterpret_cast<uint4*>(v)[0] = o1[0]; reinterpret_cast<uint4*>(v)[1] = o1[1];
            reinterpret_cast<uint4*>(v)[2] = o2[0]; reinterpret_cast<uint4*>(v)[3] = o2[1];
        }
    }
}

// A warp's 32 rows x 64 bytes of output, turned in its own 2 KB of shared memory: a lane puts its row, and gets a quarter of every eighth row, so
// that a store instruction writes 8 x 64 contiguous bytes. Straight from the accumulators' layout a lane writes 16 bytes of its own row and
// every 32-byte sector takes two instructions (1024 x 9216 x 512, fp32 / bf16 results: 23.7 / 15.1 us, turned 16.2 / 13.3). 16-byte pieces are swizzled: no bank
// conflicts either way.
template <typename T> __device__ __forceinline__ T& rows_at(uint8_t* sb, int row, int piece) {
    return *reinterpret_cast<T*>(sb + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4));
}
__device__ __forceinline__ void rows_put(uint8_t* sb, int lane, const uint4* v) {
    __syncwarp();                                          // the block before is read
#pragma unroll
    for (int j = 0; j < 4; j++) rows_at<uint4>(sb, lane, j) = v[j];
    __syncwarp();
}
__device__ __forceinline__ uint4 rows_get(uint8_t* sb, int lane, int i) { return rows_at<uint4>(sb, 8 * i + (lane >> 2), lane & 3); }   // of row 8 i + lane / 4
__device__ __forceinline__ int64_t epi_out_row(const GemmEpi& ep, int row) { return ep.row_map ? (int64_t)ep.row_map[row] : (int64_t)row; }
// 32 bf16 columns of 32 rows (row0: the warp's first; rows from m_end on are not written)
__device__ __forceinline__ void epi_put_bf16(const GemmEpi& ep, uint8_t* sb, int row0, int m_end, int n0, const uint4* v) {
    const int lane = threadIdx.x & 31;
    rows_put(sb, lane, v);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = row0 + 8 * i + (lane >> 2);
        if (row < m_end) st_out16(reinterpret_cast<bf16*>(ep.out) + epi_out_row(ep, row) * ep.ldo + n0 + 8 * (lane & 3), rows_get(sb, lane, i), ep.stream_out);
    }
}

// 32 outputs of a gated unit from its gate and up accumulators, in the arithmetic of the separate activation kernels
template <int ACT> __device__ __forceinline__ void glu32(const GemmEpi& ep, const float* g, const float* u, uint32_t* o) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        float y[2];
#pragma unroll
        for (int e = 0; e < 2; e++)
            y[e] = ACT == P3_GLU_CLAMPED ? glu_clamped(g[i + e], u[i + e], ep.glu_limit, ep.glu_alpha) : glu_act<ACT>(g[i + e]) * u[i + e];
        o[i / 2] = pack_bf16(y[0], y[1]);
    }
}
__device__ __forceinline__ void epi_glu32(const GemmEpi& ep, uint8_t* sb, int row0, int m_end, int n0, const uint32_t* ga, const uint32_t* ua) {
    float g[32], u[32];
#pragma unroll
    for (int i = 0; i < 32; i++) { g[i] = __uint_as_float(ga[i]); u[i] = __uint_as_float(ua[i]); }
    if (ep.bias) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(ep.bias + n0 + i)), b = __ldg(reinterpret_cast<const uint4*>(ep.bias + ep.glu_f + n0 + i));
            const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 x = unpack_bf16(av[e]), y = unpack_bf16(bv[e]);
                g[i + 2 * e] += x.x; g[i + 2 * e + 1] += x.y; u[i + 2 * e] += y.x; u[i + 2 * e + 1] += y.y;
            }
        }
    }
    uint4 o[4];
    uint32_t* w = reinterpret_cast<uint32_t*>(o);
    if (row0 + (int)(threadIdx.x & 31) < m_end) {                // as in the SwiGLU epilogue: the units divide
        if (ep.glu_act == P3_GLU_CLAMPED) glu32<P3_GLU_CLAMPED>(ep, g, u, w);
        else if (ep.glu_act == 0) glu32<0>(ep, g, u, w);
        else if (ep.glu_act == 1) glu32<1>(ep, g, u, w);
        else glu32<2>(ep, g, u, w);
    }
    epi_put_bf16(ep, sb, row0, m_end, n0, o);
}

// 32 lanes' columns turned into rows: a lane brings column `lane` of 32 rows and leaves with its row of 32 columns, through 4 KB of the warp's own
// (16-byte pieces swizzled by the row: no bank conflicts either way)
__device__ __forceinline__ void turn32(uint8_t* sb, int lane, uint32_t* v) {
    __syncwarp();                                          // the block before is read
#pragma unroll
    for (int i = 0; i < 32; i++) *reinterpret_cast<uint32_t*>(sb + i * 128 + (((lane >> 2) ^ (i & 7)) << 4) + (lane & 3) * 4) = v[i];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const uint4 t = *reinterpret_cast<const uint4*>(sb + lane * 128 + ((j ^ (lane & 7)) << 4));
        v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
    }
}
// epilogue for 32 consecutive accumulator columns of a warp's 32 rows (row0: its first; rows from m_end on are not written; rs: RMSNorm scale of
// the lane's row, 1 when not normed). Columns that end inside the 32, and row pitches that split 16-byte pieces, go element by element.
// A residual's pieces of 64 bytes a row are read one ahead: `r` holds the first of this chunk on entry, of the chunk at (row1, n1) (none: n1 >= N) on
// exit.
__device__ __forceinline__ bool epi_whole(const GemmEpi& ep, int n0, int N) {
    return n0 + 32 <= N && (ep.ldo & (ep.kind == P3_EPI_F32 || ep.kind == P3_EPI_RESIDUAL_F32 ? 3 : 7)) == 0;
}
__device__ __forceinline__ void epi_resid(const GemmEpi& ep, int row0, int m_end, int n0, int N, int bytes, uint4* r) {
    if ((ep.kind != P3_EPI_RESIDUAL && ep.kind != P3_EPI_RESIDUAL_F32) || !epi_whole(ep, n0, N)) return;
    const int lane = threadIdx.x & 31, esz = ep.kind == P3_EPI_RESIDUAL_F32 ? 4 : 2;
    const char* p = reinterpret_cast<const char*>(ep.resid) + (int64_t)n0 * esz + bytes + 16 * (lane & 3);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = row0 + 8 * i + (lane >> 2);
        if (row < m_end) r[i] = *reinterpret_cast<const uint4*>(p + epi_out_row(ep, row) * ep.ldo * esz);
    }
}
__device__ __forceinline__ void epi_rows32(const GemmEpi& ep, uint8_t* sb, int row0, int m_end, int n0, int row1, int n1, int N, const uint32_t* acc, float rs,
                                           uint4 (&r)[4]) {
    const int lane = threadIdx.x & 31, own = row0 + lane, sub = lane >> 2, part = lane & 3;
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(acc[i]) * rs;
    if (ep.bias) {
        if (n0 + 32 <= N) {
            uint4 bv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) bv[i] = __ldg(reinterpret_cast<const uint4*>(ep.bias + n0) + i);
            const uint32_t* bu = reinterpret_cast<const uint32_t*>(bv);
#pragma unroll
            for (int i = 0; i < 16; i++) { float2 f = unpack_bf16(bu[i]); v[2 * i] += f.x; v[2 * i + 1] += f.y; }
        } else {
            for (int i = 0; i < 32; i++) if (n0 + i < N) v[i] += __bfloat162float(ep.bias[n0 + i]);
        }
    }
    if (ep.kind == P3_EPI_F32 || ep.kind == P3_EPI_RESIDUAL_F32) {
        const float* resid = ep.kind == P3_EPI_RESIDUAL_F32 ? reinterpret_cast<const float*>(ep.resid) : nullptr;
        float* out = reinterpret_cast<float*>(ep.out);
        if (epi_whole(ep, n0, N)) {
#pragma unroll
            for (int h = 0; h < 2; h++) {                      // 16 columns each
                uint4 w[4], next[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    w[j] = make_uint4(__float_as_uint(v[16 * h + 4 * j]), __float_as_uint(v[16 * h + 4 * j + 1]), __float_as_uint(v[16 * h + 4 * j + 2]),
                                      __float_as_uint(v[16 * h + 4 * j + 3]));
                if (resid) epi_resid(ep, h ? row1 : row0, m_end, h ? n1 : n0, N, h ? 0 : 64, next);
                rows_put(sb, lane, w);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int row = row0 + 8 * i + sub;
                    const uint4 g = rows_get(sb, lane, i);
                    float4 f = make_float4(__uint_as_float(g.x), __uint_as_float(g.y), __uint_as_float(g.z), __uint_as_float(g.w));
                    if (resid) { f.x += __uint_as_float(r[i].x); f.y += __uint_as_float(r[i].y); f.z += __uint_as_float(r[i].z); f.w += __uint_as_float(r[i].w); }
                    if (row < m_end) *reinterpret_cast<float4*>(out + epi_out_row(ep, row) * ep.ldo + n0 + 16 * h + 4 * part) = f;
                }
                if (resid) {
#pragma unroll
                    for (int i = 0; i < 4; i++) r[i] = next[i];
                }
            }
        } else if (own < m_end) {
            const int64_t at = epi_out_row(ep, own) * ep.ldo + n0;
#pragma unroll
            for (int i = 0; i < 32; i++) if (n0 + i < N) out[at + i] = resid ? v[i] + resid[at + i] : v[i];
        }
        return;
    }
    const bool full = epi_whole(ep, n0, N);
    const bf16* resid = ep.kind == P3_EPI_RESIDUAL ? reinterpret_cast<const bf16*>(ep.resid) : nullptr;
    bf16* out = reinterpret_cast<bf16*>(ep.out);
    if (ep.kind == P3_EPI_QGELU) {                            // one branch per chunk, not per element: with the kind test inside the
#pragma unroll                                                 // loop 23080 x 4096 x 1024 takes 270 us, like this 169
        for (int i = 0; i < 32; i++) v[i] = __fdividef(v[i], 1.f + __expf(-1.702f * v[i]));
    } else if (ep.kind == P3_EPI_GELU) {
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = 0.5f * v[i] * (1.f + erff(v[i] * 0.70710678118654752f));
    }
    if (full) {
        uint4 ov[4];
        uint32_t* ou = reinterpret_cast<uint32_t*>(ov);
#pragma unroll
        for (int i = 0; i < 16; i++) ou[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
        if (!resid && !ep.ss_out) { epi_put_bf16(ep, sb, row0, m_end, n0, ov); return; }
        uint4 next[4];
        if (resid) epi_resid(ep, row1, m_end, n1, N, 0, next);
        rows_put(sb, lane, ov);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = row0 + 8 * i + sub;
            const uint4 g = rows_get(sb, lane, i);
            uint32_t w[4] = {g.x, g.y, g.z, g.w};
            if (resid) {
                const uint32_t ru[4] = {r[i].x, r[i].y, r[i].z, r[i].w};
#pragma unroll
                for (int e = 0; e < 4; e++) { const float2 f = unpack_bf16(ru[e]), x = unpack_bf16(w[e]); w[e] = pack_bf16(f.x + x.x, f.y + x.y); }
            }
            if (row < m_end) st_out16(out + epi_out_row(ep, row) * ep.ldo + n0 + 8 * part, make_uint4(w[0], w[1], w[2], w[3]), ep.stream_out);
            if (ep.ss_out) {                                   // squares of the bf16 values just written, by pairs of columns, to the place just read ...
                float t[4];
#pragma unroll
                for (int e = 0; e < 4; e++) { const float2 f = unpack_bf16(w[e]); t[e] = f.x * f.x + f.y * f.y; }
                rows_at<float4>(sb, 8 * i + sub, part) = make_float4(t[0], t[1], t[2], t[3]);
            }
        }
        if (ep.ss_out) {                                       // ... and so back to the row's lane, which adds its 16 pairs from left to right
            __syncwarp();
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) { const float4 t = rows_at<float4>(sb, lane, j); s += t.x; s += t.y; s += t.z; s += t.w; }
            if (own < m_end) ep.ss_out[(size_t)epi_out_row(ep, own) * (N / 32) + n0 / 32] = s;
        }
        if (resid) {
#pragma unroll
            for (int i = 0; i < 4; i++) r[i] = next[i];
        }
    } else if (own < m_end) {
        const int64_t orow = epi_out_row(ep, own);
        bf16* o = out + orow * ep.ldo + n0;
        const bf16* r = resid ? resid + orow * ep.ldo + n0 : nullptr;
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            if (n0 + i >= N) continue;
            o[i] = __float2bfloat16_rn(r ? __bfloat162float(r[i]) + bf16_round(v[i]) : v[i]);
            const float f = __bfloat162float(o[i]);
            sq += f * f;
        }
        if (ep.ss_out) ep.ss_out[(size_t)orow * (N / 32) + n0 / 32] = sq;
    }
}

// GROUPED: tmA covers 128 rows per box, tmA32 32 (tiles of few rows: decode steps are a stream of W)
template <int BN, bool GROUPED>
__global__ void __launch_bounds__(384, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA32, GemmEpi ep,
               int M, int N, int K) {
    using C = TcCfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = smem_base + C::STAGES * C::STAGE_BYTES;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (C::STAGES + s); };
    auto tfull_bar = [&](int s) { return bars + 8u * (2 * C::STAGES + s); };
    auto tempty_bar = [&](int s) { return bars + 8u * (2 * C::STAGES + 2 + s); };
    const uint32_t tmem_slot = bars + 8u * (2 * C::STAGES + 4);
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(
        smem_raw + (tmem_slot - smem_u32(smem_raw)));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m_tiles = (M + C::BM - 1) / C::BM, n_tiles = (N + BN - 1) / BN;
    const int ksplit = ep.ksplit > 1 ? ep.ksplit : 1;
    int total = m_tiles * n_tiles * ksplit; const int kb_all = (K + C::BK - 1) / C::BK;   // work item = (tile, K slice)
    const int nb = band_width(K, BN, n_tiles, ep.band_mb);
    __shared__ int s_last;

    if (warp == 0 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
    }
    if (warp == 1 && lane == 0) {
        for (int s = 0; s < C::STAGES; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int s = 0; s < 2; s++) { mbar_init(tfull_bar(s), 1); mbar_init(tempty_bar(s), 256); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "n"(C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_ptr;
    // programmatic dependent launch: barrier init / TMEM allocation above overlap the previous kernel's tail; nothing
    // below (TMA loads of X, residual reads, output writes) may run before that kernel has completed
    pdl_trigger();
    pdl_wait();
    __shared__ GroupTable groups;                              // (not part of the other kernel's shared memory)
    if constexpr (GROUPED) {
        if (warp == 3) group_table(groups, ep.seg, ep.n_groups, M, C::BM);
        __syncthreads();
        total = groups.tiles[ep.n_groups] * n_tiles;
    }

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0; uint32_t phase = 0;
            for (int item = blockIdx.x; item < total; item += gridDim.x) {
                const int tile = item / ksplit, ks = item - tile * ksplit;
                int m_idx, n_idx;
                bool few = false;
                if constexpr (GROUPED) {
                    const GroupTile t = group_tile(groups, ep.n_groups, ep.w_rows, tile, n_tiles, C::BM, BN);
                    m_idx = t.m; n_idx = t.w + t.n; few = t.m_end - t.m <= 32;
                } else {
                    int mt_, nt_;
                    tile_coords(tile, m_tiles, n_tiles, nb, mt_, nt_);
                    m_idx = mt_ * C::BM; n_idx = nt_ * BN;
                }
                const int k0 = (int)((long long)kb_all * ks / ksplit), k1 = (int)((long long)kb_all * (ks + 1) / ksplit);
                for (int k = k0; k < k1; k++) {
                    mbar_wait(empty_bar(stage), phase ^ 1);
                    mbar_expect_tx(full_bar(stage), GROUPED && few ? C::A_BYTES / 4 + C::B_BYTES : C::STAGE_BYTES);
                    const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
                    tma_load_2d(sa, GROUPED && few ? &tmA32 : &tmA, full_bar(stage), k * C::BK, m_idx);
                    tma_load_2d(sa + C::A_BYTES, &tmB, full_bar(stage), k * C::BK, n_idx);
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // The whole warp stays converged and one elected lane issues: with the loop under `if (lane == 0)` the products of
        // 16384 rows took 4 to 10 % longer.
        int stage = 0; uint32_t phase = 0;
        int acc = 0; uint32_t acc_phase = 0;
        for (int item = blockIdx.x; item < total; item += gridDim.x) {
            const int ks = item % ksplit;
            const int k0 = (int)((long long)kb_all * ks / ksplit), k1 = (int)((long long)kb_all * (ks + 1) / ksplit);
            mbar_wait(tempty_bar(acc), acc_phase ^ 1);
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
            for (int k = k0; k < k1; k++) {
                mbar_wait(full_bar(stage), phase);
                tc_fence_after();
                const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
                const uint64_t adesc = umma_desc_sw128(sa), bdesc = umma_desc_sw128(sa + C::A_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < C::BK / 16; kk++)   // +32 bytes (>>4 = 2) per UMMA_K inside the swizzle atom
                        tc_mma_bf16(d_tmem, adesc + 2 * kk, bdesc + 2 * kk, C::IDESC, ((k - k0) | kk) ? 1u : 0u);
                    tc_commit(empty_bar(stage));
                    if (k == k1 - 1) tc_commit(tfull_bar(acc));
                }
                __syncwarp();
                if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
            }
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
    } else if (warp >= 4) {
        const int q = warp & 3, half = (warp - 4) >> 2;       // TMEM lane quarter, column half
        uint8_t* sb = smem_raw + (bars + 256 - smem_u32(smem_raw)) + (warp - 4) * 2048;
        int acc = 0; uint32_t acc_phase = 0;
        for (int item = blockIdx.x; item < total; item += gridDim.x) {
            const int tile = item / ksplit, ks = item - tile * ksplit;
            int m_idx, n_idx, m_end = M;
            if constexpr (GROUPED) {
                const GroupTile t = group_tile(groups, ep.n_groups, ep.w_rows, tile, n_tiles, C::BM, BN);
                m_idx = t.m; n_idx = t.n; m_end = t.m_end;
            } else {
                int mt_, nt_;
                tile_coords(tile, m_tiles, n_tiles, nb, mt_, nt_);
                m_idx = mt_ * C::BM; n_idx = nt_ * BN;
            }
            const int row = m_idx + q * 32 + lane;
            const bool row_ok = row < m_end;
            const int64_t orow = row_ok ? (ep.row_map ? (int64_t)ep.row_map[row] : (int64_t)row) : 0;
            const float rs = epi_row_scale(ep, sb, row - lane, m_end, K);  // summed while the tile's MMAs run
            RopeRow rr;                                          // likewise: page lookup + cos/sin rows pulled into L1
            if (ep.kind == P3_EPI_ROPE_KV && row_ok) rr = epi_rope_row(ep, (int)orow);
            uint4 r[4];
            epi_resid(ep, row - lane, m_end, n_idx + half * (BN / 2), N, 0, r);
            mbar_wait(tfull_bar(acc), acc_phase);
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN);
            if (!GROUPED && ksplit > 1) {
                // a tile's slices as [slice][4 columns][row]: a warp's 16-byte pieces are neighbours (row by row every sector takes two
                // instructions: 297 x 3072 x 8192, four slices: 39 us)
                float4* wsrow = reinterpret_cast<float4*>(ep.ws) + (size_t)tile * ksplit * C::BM * BN / 4 + q * 32 + lane;   // slice 0, this row
                float4* mine = wsrow + (size_t)ks * C::BM * BN / 4;
#pragma unroll 1
                for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
                    uint32_t v[32];
                    tc_ld32(taddr + c0, v);                                     // (warp-collective: every lane loads)
                    if (row_ok) {
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            mine[(c0 / 4 + i) * C::BM] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]),
                                                                     __uint_as_float(v[4 * i + 3]));
                    }
                    __syncwarp();
                }
                tc_fence_before();
                __threadfence();
                asm volatile("bar.sync 2, 256;" ::: "memory");                  // the 8 epilogue warps
                if (threadIdx.x == 128) s_last = (atomicAdd(ep.counters + tile, 1) == ksplit - 1);
                asm volatile("bar.sync 2, 256;" ::: "memory");
                if (!s_last) {
                    mbar_arrive(tempty_bar(acc));                               // the accumulator stage is free again
                    if (++acc == 2) { acc = 0; acc_phase ^= 1; }
                    continue;
                }
                __threadfence();
                tc_fence_after();
                if (threadIdx.x == 128) ep.counters[tile] = 0;                  // ready for the next launch
                // the last CTA of the tile: all slices' partials, in slice order, back into its accumulators
#pragma unroll 1
                for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
                    float4 f[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) f[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (row_ok) {
#pragma unroll 1
                        for (int s2 = 0; s2 < ksplit; s2++) {
                            const float4* src = wsrow + (size_t)s2 * C::BM * BN / 4 + c0 / 4 * C::BM;
#pragma unroll
                            for (int i = 0; i < 8; i++) { const float4 g = __ldcg(src + i * C::BM); f[i].x += g.x; f[i].y += g.y; f[i].z += g.z; f[i].w += g.w; }
                        }
                    }
                    __syncwarp();
                    tc_st32(taddr + c0, reinterpret_cast<const uint32_t*>(f));
                }
                tc_fence_before();
                asm volatile("bar.sync 2, 256;" ::: "memory");                  // SwiGLU reads columns that other warps summed
                tc_fence_after();
            }
            if (ep.kind == P3_EPI_SWIGLU) {
                // interleaved weights: columns [0,BN/2) gate, [BN/2,BN) matching up
#pragma unroll 1
                for (int c0 = half * (BN / 4); c0 < (half + 1) * (BN / 4); c0 += 32) {
                    uint32_t g[32], u[32];
                    tc_ld32(taddr + c0, g);
                    tc_ld32(taddr + BN / 2 + c0, u);
                    const int on0 = n_idx / 2 + c0;
                    if (on0 < N / 2) {
                        uint4 ov[4];
                        uint32_t* ou = reinterpret_cast<uint32_t*>(ov);
                        // rows that do not exist: their zeros would divide slowly (297 rows: 50 us, 41 so; as a branch around the units it cost
                        // the kernel's other epilogues 2 %)
#pragma unroll
                        for (int i = 0; i < 32; i++) g[i] = row_ok ? g[i] : __float_as_uint(1.f);
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            float g0 = bf16_round(__uint_as_float(g[2 * i]) * rs), g1 = bf16_round(__uint_as_float(g[2 * i + 1]) * rs);
                            float u0 = bf16_round(__uint_as_float(u[2 * i]) * rs), u1 = bf16_round(__uint_as_float(u[2 * i + 1]) * rs);
                            float a0 = bf16_round(g0 / (1.f + __expf(-g0))), a1 = bf16_round(g1 / (1.f + __expf(-g1)));
                            ou[i] = pack_bf16(a0 * u0, a1 * u1);
                        }
                        if (on0 + 32 <= N / 2 && (ep.ldo & 7) == 0) epi_put_bf16(ep, sb, row - lane, m_end, on0, ov);
                        else if (row_ok) {
                            bf16* o = reinterpret_cast<bf16*>(ep.out) + orow * ep.ldo + on0;
                            const bf16* ob = reinterpret_cast<const bf16*>(ov);
                            for (int i = 0; i < 32; i++) if (on0 + i < N / 2) o[i] = ob[i];
                        }
                    }
                }
            } else if (ep.kind == P3_EPI_ROPE_KV) {
                RopeRow rr;
                if (row_ok) rr = epi_rope_row(ep, (int)orow);
#pragma unroll 1
                for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
                    uint32_t v[32];
                    tc_ld32(taddr + c0, v);
                    if (row_ok && n_idx + c0 < N) epi_rope32(ep, rr, n_idx + c0, rs, v);
                }
            } else {
#pragma unroll 1
                for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
                    uint32_t v[32];
                    tc_ld32(taddr + c0, v);
                    if (n_idx + c0 < N) epi_rows32(ep, sb, row - lane, m_end, n_idx + c0, row - lane,
                                                      c0 + 32 < (half + 1) * (BN / 2) ? n_idx + c0 + 32 : N, N, v, rs, r);
                }
            }
            tc_fence_before();
            mbar_arrive(tempty_bar(acc));
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(C::TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------------------
// 2-CTA variant: a CTA pair (cluster 2x1, same TPC) computes a 256 x 256 tile with
// tcgen05.mma.cta_group::2 (UMMA 256 x 256 x 16). Each CTA TMA-loads its own 128 rows of A and only
// HALF of the W tile (128 rows); the tensor cores read the other half from the peer's shared
// memory, so L2->SM operand traffic per FLOP drops by a third (96 -> 64 B/cycle/SM at full rate) and
// the 6-stage ring holds 2x the K depth. The leader CTA (rank 0) issues every MMA; its commits are
// multicast to both CTAs' barriers; both CTAs' epilogue warps release the accumulator stage on the
// leader's barrier through the cluster shared window.
// ------------------------------------------------------------------------------------------
#define P3_PEER_MASK 0xFEFFFFFFu        // clears the CTA-rank bit of a shared::cluster address -> CTA 0 of the pair
__device__ __forceinline__ void tma_load_2d_2sm(uint32_t dst, const CUtensorMap* tm, uint32_t bar_cta0, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cta0), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tc_commit_2sm_mc(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc_mma_bf16_2sm(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

struct Tc2Cfg {
    static constexpr int BM = 128, BN_MAX = 256, BK = 64, STAGES = 6;
    static constexpr int A_BYTES = BM * BK * 2, B_BYTES = (BN_MAX / 2) * BK * 2;  // per CTA: own A rows + half of W rows
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int TMEM_COLS = 2 * BN_MAX;
    static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256 + EPI_SMEM;
    static constexpr int SMEM_TURN = SMEM + EPI_SMEM;          // 4 KB a warp
    static constexpr __host__ __device__ uint32_t idesc(int bn) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24); }
};

// GLU: out = act(gate) * up in the epilogue. A tile is 128 gate columns beside the matching 128 up columns: the leader CTA loads gate rows of W,
// its peer the up rows F further on, so the weights stay as they are and the fp32 [gate | up] rows never reach memory (5418 rows, K 2048,
// F 8192: product 291 us + activation 110 us before, 233 us as one).
//
// TURN: W is the 256-row side of a tile and X the side of BN rows, so that the rows of X are cut as finely as the columns of W otherwise (781 rows: 832
// are multiplied in tiles of 208, in tiles of 256 rows 1024). An accumulator lane is then a column of the output: the epilogue turns blocks of 32 x 32
// through shared memory and goes on as for the other side (781 x 9216 x 3072, fp32 out: 42.2 -> 38.7 us). What an epilogue forms for a
// row of X once per tile (row scales, rotary rows) it would form here for every 32 rows (the rotary product of 781 rows is level), and gated units want
// both halves of W in one row of accumulators (16 gate rows beside 16 up rows, in boxes of 16: 74 -> 107 us): these stay with X as the 256-row side.
template <bool GROUPED, bool GLU = false, bool TURN = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
gemm_tc2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmEpi ep,
                int M, int N, int K, int BN) {
    using C = Tc2Cfg;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = smem_base + C::STAGES * C::STAGE_BYTES;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (C::STAGES + s); };
    auto tfull_bar = [&](int s) { return bars + 8u * (2 * C::STAGES + s); };
    auto tempty_bar = [&](int s) { return bars + 8u * (2 * C::STAGES + 2 + s); };
    const uint32_t tmem_slot = bars + 8u * (2 * C::STAGES + 4);
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const bool leader = rank == 0;
    static_assert(!(TURN && (GROUPED || GLU)), "plain products only");
    const int tile_m = TURN ? BN : 2 * C::BM, tile_n = TURN ? 2 * C::BM : GLU ? 128 : BN;    // rows of X and W of a tile (gated: of a half of W)
    const int m_pairs = (M + tile_m - 1) / tile_m, n_tiles = GLU ? (ep.glu_f + 127) / 128 : (N + tile_n - 1) / tile_n;
    const uint32_t stage_tx = 2u * (C::A_BYTES + (uint32_t)BN * C::BK), idesc = Tc2Cfg::idesc(BN);   // a pair's bytes of one k block
    int total = m_pairs * n_tiles; const int kb = (K + C::BK - 1) / C::BK;
    const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    const int nb = band_width(K, TURN ? 2 * C::BM : BN, n_tiles, ep.band_mb);

    if (warp == 0 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
    }
    if (warp == 1 && lane == 0) {
        for (int s = 0; s < C::STAGES; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int s = 0; s < 2; s++) { mbar_init(tfull_bar(s), 1); mbar_init(tempty_bar(s), 512); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "n"(C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_ptr;
    // programmatic dependent launch: barrier init / TMEM allocation above overlap the previous kernel's tail; nothing
    // below (TMA loads of X, residual reads, output writes) may run before that kernel has completed
    pdl_trigger();
    pdl_wait();
    __shared__ GroupTable groups;
    if constexpr (GROUPED) {
        if (warp == 3) group_table(groups, ep.seg, ep.n_groups, M, 2 * C::BM);
        __syncthreads();
        total = groups.tiles[ep.n_groups] * n_tiles;
    }

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0; uint32_t phase = 0;
            for (int tile = cluster_id; tile < total; tile += n_clusters) {
                int m_idx, n_idx;
                if constexpr (GROUPED) {
                    const GroupTile t = group_tile(groups, ep.n_groups, ep.w_rows, tile, n_tiles, 2 * C::BM, BN);
                    m_idx = t.m; n_idx = t.w + t.n;
                } else {
                    int mt_, nt_;
                    tile_coords(tile, m_pairs, n_tiles, nb, mt_, nt_);
                    m_idx = mt_ * tile_m; n_idx = nt_ * tile_n;
                }
                if constexpr (TURN) {
                    m_idx += (int)rank * (BN / 2); n_idx += (int)rank * C::BM;
                } else {
                    m_idx += (int)rank * C::BM; n_idx += (int)rank * (GLU ? ep.glu_f : BN / 2);
                }
                for (int k = 0; k < kb; k++) {
                    mbar_wait(empty_bar(stage), phase ^ 1);
                    if (leader) mbar_expect_tx(full_bar(stage), stage_tx);   // both CTAs' bytes land on CTA 0's barrier
                    const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
                    const uint32_t fb0 = full_bar(stage) & P3_PEER_MASK;
                    tma_load_2d_2sm(sa, TURN ? &tmB : &tmA, fb0, k * C::BK, TURN ? n_idx : m_idx);
                    tma_load_2d_2sm(sa + C::A_BYTES, TURN ? &tmA : &tmB, fb0, k * C::BK, TURN ? m_idx : n_idx);
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (leader) {                                           // converged warp, elected issuing lane (see gemm_tc_kernel)
            int stage = 0; uint32_t phase = 0;
            int acc = 0; uint32_t acc_phase = 0;
            for (int tile = cluster_id; tile < total; tile += n_clusters) {
                mbar_wait(tempty_bar(acc), acc_phase ^ 1);
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * C::BN_MAX);
                for (int k = 0; k < kb; k++) {
                    mbar_wait(full_bar(stage), phase);
                    tc_fence_after();
                    const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
                    const uint64_t adesc = umma_desc_sw128(sa), bdesc = umma_desc_sw128(sa + C::A_BYTES);
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < C::BK / 16; kk++)
                            tc_mma_bf16_2sm(d_tmem, adesc + 2 * kk, bdesc + 2 * kk, idesc, (k | kk) ? 1u : 0u);
                        tc_commit_2sm_mc(empty_bar(stage));                             // frees the slot in both CTAs
                        if (k == kb - 1) tc_commit_2sm_mc(tfull_bar(acc));              // accumulators ready in both CTAs
                    }
                    __syncwarp();
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                }
                if (++acc == 2) { acc = 0; acc_phase ^= 1; }
            }
        }
    } else if (warp >= 4) {
        const int q = warp & 3, half = (warp - 4) >> 2;
        const int c_mid = ((BN + 31) / 32 + 1) / 2 * 32, c_lo = half ? c_mid : 0, c_hi = half ? BN : c_mid;   // this warp's columns
        uint8_t* sb = smem_raw + (bars + 256 - smem_u32(smem_raw)) + (warp - 4) * (TURN ? 4096 : 2048);
        int acc = 0; uint32_t acc_phase = 0;
        for (int tile = cluster_id; tile < total; tile += n_clusters) {
            int m_idx, n_idx, m_end = M;
            if constexpr (GROUPED) {
                const GroupTile t = group_tile(groups, ep.n_groups, ep.w_rows, tile, n_tiles, 2 * C::BM, BN);
                m_idx = t.m; n_idx = t.n; m_end = t.m_end;
            } else {
                int mt_, nt_;
                tile_coords(tile, m_pairs, n_tiles, nb, mt_, nt_);
                m_idx = mt_ * tile_m; n_idx = nt_ * tile_n;
            }
            if constexpr (TURN) {
                const int f0 = n_idx + (int)rank * C::BM + q * 32;                          // the warp's output columns
                m_end = min(M, m_idx + BN);
                uint4 r[4];
                epi_resid(ep, m_idx + c_lo, m_end, f0, N, 0, r);
                mbar_wait(tfull_bar(acc), acc_phase);
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * C::BN_MAX);
                for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
                    uint32_t v[32];
                    tc_ld32(taddr + c0, v);
                    const int row0 = m_idx + c0;
                    if (f0 >= N || row0 >= m_end) continue;
                    turn32(sb, lane, v);
                    epi_rows32(ep, sb, row0, m_end, f0, row0 + 32, c0 + 32 < c_hi ? f0 : N, N, v, 1.f, r);
                }
                tc_fence_before();
                mbar_arrive_cluster(tempty_bar(acc) & P3_PEER_MASK);
                if (++acc == 2) { acc = 0; acc_phase ^= 1; }
                continue;
            }
            m_idx += (int)rank * C::BM;
            const int row = m_idx + q * 32 + lane;
            const bool row_ok = row < m_end;
            const int64_t orow = row_ok ? (ep.row_map ? (int64_t)ep.row_map[row] : (int64_t)row) : 0;
            const float rs = epi_row_scale(ep, sb, row - lane, m_end, K);  // summed while the tile's MMAs run
            RopeRow rr;                                          // likewise: page lookup + cos/sin rows pulled into L1
            if (ep.kind == P3_EPI_ROPE_KV && row_ok) rr = epi_rope_row(ep, (int)orow);
            uint4 r[4];
            if (!GLU) epi_resid(ep, row - lane, m_end, n_idx + c_lo, N, 0, r);
            mbar_wait(tfull_bar(acc), acc_phase);
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * C::BN_MAX);
            if constexpr (GLU) {
                for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 32) {
                    uint32_t g[32], u[32];
                    tc_ld32(taddr + c0, g);
                    tc_ld32(taddr + 128 + c0, u);
                    if (n_idx + c0 < ep.glu_f) epi_glu32(ep, sb, row - lane, m_end, n_idx + c0, g, u);
                }
            } else if (ep.kind == P3_EPI_SWIGLU) {
                for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 32) {    // BN = 256
                    uint32_t g[32], u[32];
                    tc_ld32(taddr + c0, g);
                    tc_ld32(taddr + 128 + c0, u);
                    const int on0 = n_idx / 2 + c0;
                    if (on0 < N / 2) {
                        uint4 ov[4];
                        uint32_t* ou = reinterpret_cast<uint32_t*>(ov);
                        // rows that do not exist: their zeros would divide slowly (297 rows: 50 us, 41 so; as a branch around the units it cost
                        // the kernel's other epilogues 2 %)
#pragma unroll
                        for (int i = 0; i < 32; i++) g[i] = row_ok ? g[i] : __float_as_uint(1.f);
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            float g0 = bf16_round(__uint_as_float(g[2 * i]) * rs), g1 = bf16_round(__uint_as_float(g[2 * i + 1]) * rs);
                            float u0 = bf16_round(__uint_as_float(u[2 * i]) * rs), u1 = bf16_round(__uint_as_float(u[2 * i + 1]) * rs);
                            float a0 = bf16_round(g0 / (1.f + __expf(-g0))), a1 = bf16_round(g1 / (1.f + __expf(-g1)));
                            ou[i] = pack_bf16(a0 * u0, a1 * u1);
                        }
                        if (on0 + 32 <= N / 2 && (ep.ldo & 7) == 0) epi_put_bf16(ep, sb, row - lane, m_end, on0, ov);
                        else if (row_ok) {
                            bf16* o = reinterpret_cast<bf16*>(ep.out) + orow * ep.ldo + on0;
                            const bf16* ob = reinterpret_cast<const bf16*>(ov);
                            for (int i = 0; i < 32; i++) if (on0 + i < N / 2) o[i] = ob[i];
                        }
                    }
                }
            } else if (ep.kind == P3_EPI_ROPE_KV) {
                for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
                    uint32_t v[32];
                    tc_ld32(taddr + c0, v);
                    if (row_ok && n_idx + c0 < N) epi_rope32(ep, rr, n_idx + c0, rs, v);
                }
            } else {
                for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
                    uint32_t v[32];
                    tc_ld32(taddr + c0, v);
                    if (n_idx + c0 < N) epi_rows32(ep, sb, row - lane, m_end, n_idx + c0, row - lane, c0 + 32 < c_hi ? n_idx + c0 + 32 : N, N, v, rs, r);
                }
            }
            tc_fence_before();
            mbar_arrive_cluster(tempty_bar(acc) & P3_PEER_MASK);                        // the leader's MMA warp owns this barrier
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
    }
    tc_fence_before();
    cluster_sync();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(C::TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------------------
// mma.sync cross-check GEMM (tests / bring-up only; not the product path)
// ------------------------------------------------------------------------------------------
#define FB_BM 64
#define FB_BN 64
#define FB_BK 32
__global__ void __launch_bounds__(128) gemm_mma_kernel(const bf16* __restrict__ X, int64_t ldx, const bf16* __restrict__ W,
                                                       int64_t ldw, GemmEpi ep, int M, int N, int K) {
    __shared__ __align__(16) bf16 sA[FB_BM][FB_BK + 8];
    __shared__ __align__(16) bf16 sB[FB_BN][FB_BK + 8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int m0 = blockIdx.y * FB_BM;
    const bool swiglu = ep.kind == P3_EPI_SWIGLU;
    // SwiGLU: this CTA produces 64 output columns; gate rows then (second pass) the matching up rows
    const int o0 = blockIdx.x * FB_BN;
    const int passes = swiglu ? 2 : 1;
    float acc[2][2][4][4];
    for (int pass = 0; pass < passes; pass++) {
        const int nrow0 = swiglu ? ((o0 / 128) * 256 + (o0 % 128) + pass * 128) : o0;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[pass][i][j][c] = 0.f;
        for (int k0 = 0; k0 < K; k0 += FB_BK) {
            for (int i = tid; i < FB_BM * FB_BK / 8; i += 128) {
                int r = i / (FB_BK / 8), c = (i % (FB_BK / 8)) * 8;
                uint4 va = make_uint4(0, 0, 0, 0), vb = make_uint4(0, 0, 0, 0);
                if (m0 + r < M && k0 + c < K) va = *reinterpret_cast<const uint4*>(X + (size_t)(m0 + r) * ldx + k0 + c);
                if (nrow0 + r < N && k0 + c < K) vb = *reinterpret_cast<const uint4*>(W + (size_t)(nrow0 + r) * ldw + k0 + c);
                *reinterpret_cast<uint4*>(&sA[r][c]) = va;
                *reinterpret_cast<uint4*>(&sB[r][c]) = vb;
            }
            __syncthreads();
#pragma unroll
            for (int ks = 0; ks < FB_BK; ks += 16) {
                uint32_t a[2][4], b[4][2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    a[i][0] = *reinterpret_cast<const uint32_t*>(&sA[wm + i * 16 + g][ks + 2 * t]);
                    a[i][1] = *reinterpret_cast<const uint32_t*>(&sA[wm + i * 16 + g + 8][ks + 2 * t]);
                    a[i][2] = *reinterpret_cast<const uint32_t*>(&sA[wm + i * 16 + g][ks + 2 * t + 8]);
                    a[i][3] = *reinterpret_cast<const uint32_t*>(&sA[wm + i * 16 + g + 8][ks + 2 * t + 8]);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    b[j][0] = *reinterpret_cast<const uint32_t*>(&sB[wn + j * 8 + g][ks + 2 * t]);
                    b[j][1] = *reinterpret_cast<const uint32_t*>(&sB[wn + j * 8 + g][ks + 2 * t + 8]);
                }
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) mma_bf16_16816(acc[pass][i][j], a[i], b[j][0], b[j][1]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                int row = m0 + wm + i * 16 + g + (c >> 1) * 8;
                int col = o0 + wn + j * 8 + 2 * t + (c & 1);
                if (row >= M) continue;
                int64_t orow = ep.row_map ? ep.row_map[row] : row;
                if (swiglu) {
                    if (col >= N / 2) continue;
                    float gb = bf16_round(acc[0][i][j][c]), ub = bf16_round(acc[1][i][j][c]);
                    float a = bf16_round(gb / (1.f + __expf(-gb)));
                    reinterpret_cast<bf16*>(ep.out)[orow * ep.ldo + col] = __float2bfloat16_rn(a * ub);
                    continue;
                }
                if (col >= N) continue;
                float v = acc[0][i][j][c] + (ep.bias ? __bfloat162float(ep.bias[col]) : 0.f);
                if (ep.kind == P3_EPI_F32) { reinterpret_cast<float*>(ep.out)[orow * ep.ldo + col] = v; continue; }
                if (ep.kind == P3_EPI_RESIDUAL_F32) {
                    reinterpret_cast<float*>(ep.out)[orow * ep.ldo + col] = v + reinterpret_cast<const float*>(ep.resid)[orow * ep.ldo + col];
                    continue;
                }
                if (ep.kind == P3_EPI_RESIDUAL) v = __bfloat162float(reinterpret_cast<const bf16*>(ep.resid)[orow * ep.ldo + col]) + bf16_round(v);
                else if (ep.kind == P3_EPI_QGELU || ep.kind == P3_EPI_GELU) v = epi_act(ep.kind, v);
                reinterpret_cast<bf16*>(ep.out)[orow * ep.ldo + col] = __float2bfloat16_rn(v);
            }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
// Weight tensor maps are immutable for the life of a model: p3_gemm_plan_weights builds the three maps the kernels can ask
// for (box rows 256 / 128 for the single-CTA tiles, 128 = half a 256-wide tile for the CTA pair) ONCE into a caller-owned
// blob; p3_gemm_fused then skips cuTensorMapEncodeTiled for W (the X map still depends on the call's activation pointer).
struct GemmWPlan { uint64_t magic; const void* W; int64_t ldw; int32_t N, K; CUtensorMap t256, t128; };
static_assert(sizeof(GemmWPlan) <= P3_GEMM_WPLAN_BYTES, "p3_gemm weight plan blob too small");
#define P3_WPLAN_MAGIC 0x5033574D41505331ull

static int make_tmap(CUtensorMap* tm, const void* ptr, int64_t rows, int64_t K, int64_t ld, int box_rows) {
    CUresult r = tc_encode_2d(tm, ptr, rows, K, ld, box_rows);
    P3_CHECK_ARG(r == CUDA_SUCCESS, "gemm: cuTensorMapEncodeTiled failed (%d) rows=%lld K=%lld ld=%lld", (int)r,
                 (long long)rows, (long long)K, (long long)ld);
    return 0;
}

static int num_sms() {
    static int n = 0;
    if (!n) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev); }
    return n;
}

static int cur_dev() { int d = 0; cudaGetDevice(&d); return d < 0 || d >= 64 ? 0 : d; }

template <int BN>
static int launch_tc(const void* X, int64_t ldx, const void* W, int64_t ldw, const GemmEpi& ep, int64_t M, int N, int K,
                     cudaStream_t st, const GemmWPlan* wp = nullptr) {
    using C = TcCfg<BN>;
    CUtensorMap ta, tb;
    if (make_tmap(&ta, X, M, K, ldx, C::BM)) return -1;
    if (wp && BN >= 128) memcpy(&tb, (BN == 256) ? &wp->t256 : &wp->t128, sizeof(tb));
    else if (make_tmap(&tb, W, N, K, ldw, BN)) return -1;      // 64-row boxes are not part of the plan blob: encoded per call
    static bool attr_set[64] = {};                             // the attribute is per device
    if (!attr_set[cur_dev()]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<BN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        P3_CHECK_ARG(e == cudaSuccess, "gemm: cannot set %d B dynamic smem: %s", C::SMEM, cudaGetErrorString(e));
        attr_set[cur_dev()] = true;
    }
    int64_t tiles = ((M + C::BM - 1) / C::BM) * ((N + BN - 1) / BN);
    GemmEpi e2 = ep;
    e2.ksplit = 1;
    if (ep.ws && tiles * 2 < num_sms() && (int64_t)BN * K * 2 > (7ll << 18) * BN / 128) {
        // few output tiles AND a long K (each CTA would stream > 1.75 MB of W alone at ~45 KB/us, e.g. down_proj at M <= 320:
        // 24 tiles x 2 MB): split K so that tiles * ksplit ~ #SM (>= 4 k-blocks each). Measured: 43 -> 30 us
        // at M = 80, 40 -> 21 us at M = 16; for K = 3072 shapes the partial round trip costs more than it saves, so they stay unsplit.
        const int kb = (K + C::BK - 1) / C::BK;
        int ks = (int)(num_sms() / tiles);
        if (ks > 8) ks = 8;
        if (ks > kb / 4) ks = kb / 4;
        const int64_t need = P3_SPLITK_COUNTER_BYTES + tiles * ks * (int64_t)C::BM * BN * 4;
        if (ks >= 2 && tiles * 4 <= P3_SPLITK_COUNTER_BYTES && need <= ep.ws_bytes) {
            e2.ksplit = ks;
            e2.counters = reinterpret_cast<int*>(ep.ws);
            e2.ws = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ep.ws) + P3_SPLITK_COUNTER_BYTES);
        }
    }
    const int64_t items = tiles * e2.ksplit;
    unsigned grid = (unsigned)(items < num_sms() ? items : num_sms());
    p3_launch_pdl(gemm_tc_kernel<BN, false>, dim3(grid), dim3(384), (size_t)C::SMEM, st, ta, tb, ta, e2, (int)M, N, K);
    P3_CHECK_LAUNCH("gemm_tc");
    return 0;
}

static int gemm_2cta_mode() {                  // P3_GEMM_2CTA=0 forces the single-CTA kernel (A/B testing)
    static int v = -1;
    if (v < 0) { const char* e = getenv("P3_GEMM_2CTA"); v = (e && e[0] == '0') ? 0 : 1; }
    return v;
}

// waves over the CTA pairs times what one costs
static int64_t tile_cost(int64_t tiles, int width, int start, int percent) { return (tiles + num_sms() / 2 - 1) / (num_sms() / 2) * (width + start) * percent; }
// Columns of a pair's tile: the width whose waves over the CTA pairs cost least. A wave takes time in proportion to its columns plus its start
// and end (16 columns' worth), and narrow tiles re-read more of X per product: 5418 x 16384 x 3072 in 20 waves of 256 446 us, 22 of 224 447,
// 26 of 192 469, 31 of 160 501; 781 x 3072 x 8192 in one wave of 256 57.8, 224 53.1, 192 48.2. Over 138 products (300 - 5418 rows, N 1024 -
// 16384, K 1024 - 8192), each timed at every width, the widths chosen sum to 14.48 ms, the best ones to 14.41, 256 throughout to 14.90.
constexpr int plain_widths[4][2] = {{256, 100}, {224, 105}, {192, 105}, {160, 115}};
static int tile_width(int64_t M, int N) {
    const int64_t m = (M + 255) / 256;
    int best = 256; int64_t least = 0;
    for (const auto& c : plain_widths) {
        const int64_t t = tile_cost(m * ((N + c[0] - 1) / c[0]), c[0], 16, c[1]);
        if (!least || t < least) { least = t; best = c[0]; }
    }
    return best;
}
// Rows of X of a tile where W is its 256-row side; 0: X is. A wave on that side takes its rows plus 64 rows' worth (start, end and the turned epilogue).
// Over 79 products (200 - 5418 rows, N 2048 - 16384, K 1024 - 8192), each timed at nine widths, what this chooses takes 0.83 to 1.007 of the time of X as
// the 256-row side, 0.983 in the mean, the best of all widths 0.972: 300 x 9216 x 3072 25.4 -> 21.1 us with 160 rows, 781 rows 42.2 -> 38.7 with 208, 1100 x
// 3072 x 8192 46.9 -> 43.9 with 192. (From 224 rows on no choice of it: X as the 256-row side always costs less.) On 240 products of other sizes (130 - 6200 rows,
// N 1024 - 16384, K 1024 - 8192, fp32 and bf16 outputs) it takes 0.947, the best of all widths 0.934, and more than X as that side at two
// (1.002 and 1.04: 3407 x 3000 x 1024, 21.7 -> 22.6).
static int turned_rows(int64_t M, int N) {
    const int cost[6][2] = {{208, 99}, {192, 97}, {176, 97}, {160, 101}, {144, 106}, {128, 104}};
    int64_t least = INT64_MAX;
    for (const auto& c : plain_widths) {
        const int64_t t = tile_cost((M + 255) / 256 * ((N + c[0] - 1) / c[0]), c[0], 16, c[1]);
        if (t < least) least = t;
    }
    int best = 0;
    for (const auto& c : cost) {
        const int64_t t = tile_cost((M + c[0] - 1) / c[0] * ((N + 255) / 256), c[0], 64, c[1]);
        if (t < least) { least = t; best = c[0]; }
    }
    return best;
}
template <bool GLU, bool TURN>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmEpi& ep, int64_t M, int N, int K, int bn, int64_t tiles, cudaStream_t st) {
    constexpr int smem = TURN ? Tc2Cfg::SMEM_TURN : Tc2Cfg::SMEM;
    static bool attr_set[64] = {};
    if (!attr_set[cur_dev()]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc2_kernel<false, GLU, TURN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        P3_CHECK_ARG(e == cudaSuccess, "gemm: cannot set %d B dynamic smem: %s", smem, cudaGetErrorString(e));
        attr_set[cur_dev()] = true;
    }
    const int64_t clusters = tiles < num_sms() / 2 ? tiles : num_sms() / 2;
    p3_launch_pdl(gemm_tc2_kernel<false, GLU, TURN>, dim3((unsigned)(2 * clusters)), dim3(384), (size_t)smem, st, ta, tb, ep, (int)M, N, K, bn);
    P3_CHECK_LAUNCH("gemm_tc2");
    return 0;
}
static int launch_tc2(const void* X, int64_t ldx, const void* W, int64_t ldw, const GemmEpi& ep, int64_t M, int N, int K,
                      cudaStream_t st, const GemmWPlan* wp = nullptr) {
    const bool swiglu = ep.kind == P3_EPI_SWIGLU;
    const int rows = swiglu || ep.kind == P3_EPI_ROPE_KV || ep.ss_in ? 0 : turned_rows(M, N), bn = rows ? rows : swiglu ? 256 : tile_width(M, N), box = rows ? 128 : bn / 2;
    CUtensorMap ta, tb;
    if (make_tmap(&ta, X, M, K, ldx, rows ? rows / 2 : 128)) return -1;
    if (wp && box == 128) memcpy(&tb, &wp->t128, sizeof(tb));  // half of a 256-row W tile per CTA
    else if (make_tmap(&tb, W, N, K, ldw, box)) return -1;
    if (rows) return launch_pair<false, true>(ta, tb, ep, M, N, K, bn, ((M + bn - 1) / bn) * ((N + 255) / 256), st);
    return launch_pair<false, false>(ta, tb, ep, M, N, K, bn, ((M + 255) / 256) * ((N + bn - 1) / bn), st);
}

// the shared memory of a grouped launch holds the group table beside the ring
static bool smem_attr(const void* kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess; }

// out[M, N] (fp32, or bf16) = grouped product over rows already in group order; W [n_groups][w_rows][K] with row pitch ldw. Rows that overlap
// (one row for all, say) stay with the kernel that reads them by address: a tensor map wants rows that follow one another
bool gemm_grouped_ok(const p3_gemm_any_args* a) {
    return a->seg_offsets && !a->x_rows && !a->bias && !a->gate && a->n_batch <= 1 && !a->force_fma && !a->x_f32 && a->n_groups <= GROUPS_MAX && a->K % 8 == 0 &&
           a->ldx % 8 == 0 && a->ldw % 8 == 0 && a->ldx >= a->K && a->ldw >= a->K && a->w_group_stride % a->ldw == 0 && a->w_group_stride / a->ldw >= a->N &&
           a->w_group_stride / a->ldw * a->n_groups < (1ll << 31) && (((uintptr_t)a->X | (uintptr_t)a->W | (uintptr_t)a->out) & 15) == 0;
}
int launch_gemm_grouped(const p3_gemm_any_args* a, cudaStream_t st) {
    GemmEpi ep{};
    ep.out = a->out; ep.ldo = a->ldo; ep.kind = a->out_f32 ? P3_EPI_F32 : P3_EPI_NONE; ep.ksplit = 1;
    ep.seg = a->seg_offsets; ep.n_groups = a->n_groups; ep.w_rows = (int)(a->w_group_stride / a->ldw);
    const int64_t w_all = (int64_t)ep.w_rows * (a->n_groups - 1) + a->N, mean = a->M / a->n_groups;
    static bool attr_set[64] = {};
    if (!attr_set[cur_dev()]) {
        P3_CHECK_ARG(smem_attr((const void*)gemm_tc_kernel<128, true>, TcCfg<128>::SMEM) && smem_attr((const void*)gemm_tc2_kernel<true>, Tc2Cfg::SMEM),
                     "gemm_any: cannot set the shared memory of the grouped product");
        attr_set[cur_dev()] = true;
    }
    CUtensorMap ta, ta32, tb;
    const bool few = a->M <= 32;                               // then every tile takes the boxes of 32 rows
    if (make_tmap(&tb, a->W, w_all, a->K, a->ldw, 128) || (!few && make_tmap(&ta, a->X, a->M, a->K, a->ldx, 128))) return -1;
    if (mean >= 160 && gemm_2cta_mode()) {
        // CTA pairs on 256 x 256 tiles from a mean of 160 rows a group on: below it most of a pair's 256 rows would be padding, above it the pair
        // reads W half as often as 128 x 128 tiles do. More pairs than tiles only costs their launch.
        const int64_t most = (a->M / 256 + a->n_groups) * ((a->N + 255) / 256);
        const int64_t clusters = most < num_sms() / 2 ? most : num_sms() / 2;
        p3_launch_pdl(gemm_tc2_kernel<true>, dim3((unsigned)(2 * clusters)), dim3(384), (size_t)Tc2Cfg::SMEM, st, ta, tb, ep, (int)a->M, a->N, a->K, 256);
    } else {
        if (make_tmap(&ta32, a->X, a->M, a->K, a->ldx, 32)) return -1;
        if (few) ta = ta32;
        const int64_t most = (a->M / 128 + (a->M < a->n_groups ? a->M : a->n_groups)) * ((a->N + 127) / 128);
        p3_launch_pdl(gemm_tc_kernel<128, true>, dim3((unsigned)(most < num_sms() ? most : num_sms())), dim3(384), (size_t)TcCfg<128>::SMEM, st, ta, tb, ta32, ep,
                      (int)a->M, a->N, a->K);
    }
    P3_CHECK_LAUNCH("gemm_any");
    return 0;
}

// CTA pairs from a quarter of the SMs' worth of 256 x 256 tiles on: fewer rows leave a stream of W, which the kernels of smaller tiles spread
// over more CTAs
static bool pairs(int64_t M, int64_t N) { return gemm_2cta_mode() && M > 128 && ((M + 255) / 256) * ((N + 255) / 256) >= num_sms() / 4; }
// rows of X of a tile where W is its 256-row side (products without row scales, rotation and units), 0: X is, in tiles of p3_gemm_pair_width columns
extern "C" int p3_gemm_turned_rows(int64_t M, int64_t N) { return pairs(M, N) ? turned_rows(M, (int)N) : 0; }
extern "C" int p3_gemm_pair_width(int64_t M, int64_t N) {
    return pairs(M, N) ? tile_width(M, (int)N) : 0;
}

static int gemm_dispatch(const void* X, int64_t ldx, const void* W, int64_t ldw, const GemmEpi& ep, int64_t M, int N, int K,
                         int impl, cudaStream_t st, const GemmWPlan* wp) {
    if (impl == 1) {
        P3_CHECK_ARG(ep.kind != P3_EPI_ROPE_KV && !ep.ss_in && !ep.ss_out, "gemm: the mma.sync cross-check kernel has no fused norm / rope epilogue");
        int ncols = ep.kind == P3_EPI_SWIGLU ? N / 2 : N;
        dim3 grid((ncols + FB_BN - 1) / FB_BN, (unsigned)((M + FB_BM - 1) / FB_BM));
        gemm_mma_kernel<<<grid, 128, 0, st>>>((const bf16*)X, ldx, (const bf16*)W, ldw, ep, (int)M, N, K);
        P3_CHECK_LAUNCH("gemm_mma");
        return 0;
    }
    int64_t m_tiles = (M + 127) / 128;
    GemmEpi eps = ep;
    {
        static int mode = -1;                              // P3_GEMM_STREAM=0/1 forces the policy off/on (A/B only)
        if (mode < 0) { const char* e = getenv("P3_GEMM_STREAM"); mode = e ? (e[0] == '0' ? 0 : 1) : 2; }
        const int64_t out_bytes = M * (int64_t)(ep.kind == P3_EPI_SWIGLU ? N / 2 : N) * 2;
        eps.stream_out = mode == 2 ? (out_bytes >= (64ll << 20)) : mode;
        static int band = -1;                              // P3_GEMM_BAND_MB (A/B only)
        if (band < 0) { const char* e = getenv("P3_GEMM_BAND_MB"); band = e ? atoi(e) : 0; }
        eps.band_mb = band;
    }
    if (impl == 0 && p3_gemm_pair_width(M, N))
        return launch_tc2(X, ldx, W, ldw, eps, M, N, K, st, wp);
    bool small = m_tiles * ((N + 255) / 256) < 2 * num_sms();
    if (ep.kind == P3_EPI_SWIGLU || !small) return launch_tc<256>(X, ldx, W, ldw, eps, M, N, K, st, wp);
    // one row tile and fewer 128-wide column tiles than SMs (M <= 128 against the 3072..9216-row matrices: constrain steps): the GEMM
    // is a weight stream and a CTA only pulls what its TMA ring turns over per round trip -> 64-row W tiles put twice as many CTAs
    // on it (M = 80: qkv 18.9 -> 16.8 us, o_proj 19.3 -> 17.2, down_proj with split-K 28.6 -> 21.8). Not for
    // more row tiles: every CTA re-reads its X rows over the whole K, which outweighs the gain (M = 320 down_proj 36.6 -> 39.4 us).
    static int bn64 = -1;
    if (bn64 < 0) { const char* e = getenv("P3_GEMM_BN64"); bn64 = e ? atoi(e) : 1; }
    if (bn64 && m_tiles == 1 && (N + 127) / 128 < num_sms()) return launch_tc<64>(X, ldx, W, ldw, eps, M, N, K, st, wp);
    return launch_tc<128>(X, ldx, W, ldw, eps, M, N, K, st, wp);
}

extern "C" int p3_gemm(const void* X, int64_t ldx, const void* W, int64_t ldw, const void* bias, void* out, int64_t ldo,
                       const void* resid, const int32_t* row_map, int64_t M, int N, int K, int epi, int impl,
                       cudaStream_t st) {
    P3_CHECK_ARG(epi >= P3_EPI_NONE && epi <= P3_EPI_RESIDUAL_F32, "gemm: unknown epilogue %d", epi);
    P3_CHECK_ARG(ldx % 8 == 0 && ldw % 8 == 0, "gemm: ldx/ldw must be multiples of 8 elements (16 B)");
    P3_CHECK_ARG(((uintptr_t)X & 15) == 0 && ((uintptr_t)W & 15) == 0, "gemm: X/W must be 16-byte aligned");
    P3_CHECK_ARG((epi != P3_EPI_RESIDUAL && epi != P3_EPI_RESIDUAL_F32) || resid, "gemm: residual epilogue needs resid");
    P3_CHECK_ARG(epi != P3_EPI_SWIGLU || (N % 256 == 0 && !bias), "gemm: SwiGLU needs N %% 256 == 0 and no bias");
    P3_CHECK_ARG(M < (1ll << 31), "gemm: M too large");
    if (M == 0) return 0;
    GemmEpi ep{};
    ep.bias = (const bf16*)bias; ep.out = out; ep.ldo = ldo; ep.resid = resid; ep.row_map = row_map; ep.kind = epi;
    return gemm_dispatch(X, ldx, W, ldw, ep, M, N, K, impl, st, nullptr);
}

extern "C" int p3_gemm_glu(const void* X, int64_t ldx, const void* W, int64_t ldw, const void* bias, void* out, int64_t ldo, int64_t M, int F, int K,
                           int act, float limit, float alpha, cudaStream_t st) {
    P3_CHECK_ARG(X && W && out && act >= 0 && act <= P3_GLU_CLAMPED, "gemm_glu: bad arguments");
    P3_CHECK_ARG(ldx % 8 == 0 && ldw % 8 == 0 && ldo % 8 == 0, "gemm_glu: row pitches must be multiples of 8 elements (16 B)");
    P3_CHECK_ARG((((uintptr_t)X | (uintptr_t)W | (uintptr_t)out | (uintptr_t)bias) & 15) == 0, "gemm_glu: operands must be 16-byte aligned");
    P3_CHECK_ARG(M >= 0 && M < (1ll << 31) && F >= 32 && F % 32 == 0 && F < (1 << 30) && K >= 1, "gemm_glu: bad sizes");
    if (M == 0) return 0;
    GemmEpi ep{};
    ep.bias = (const bf16*)bias; ep.out = out; ep.ldo = ldo; ep.kind = P3_EPI_NONE; ep.ksplit = 1;
    ep.glu_f = F; ep.glu_act = act; ep.glu_limit = limit; ep.glu_alpha = alpha;
    ep.stream_out = M * (int64_t)F * 2 >= (64ll << 20);
    CUtensorMap ta, tb;
    if (make_tmap(&ta, X, M, K, ldx, 128) || make_tmap(&tb, W, 2 * (int64_t)F, K, ldw, 128)) return -1;
    return launch_pair<true, false>(ta, tb, ep, M, 2 * F, K, 256, ((M + 255) / 256) * ((F + 127) / 128), st);
}

extern "C" int p3_gemm_plan_weights(const void* W, int64_t ldw, int N, int K, void* plan) {
    P3_CHECK_ARG(W && plan && ldw % 8 == 0 && ((uintptr_t)W & 15) == 0, "gemm_plan_weights: bad arguments");
    P3_CHECK_ARG(((uintptr_t)plan & 63) == 0, "gemm_plan_weights: the plan blob must be 64-byte aligned");
    GemmWPlan* p = reinterpret_cast<GemmWPlan*>(plan);
    p->W = W; p->ldw = ldw; p->N = N; p->K = K;
    if (make_tmap(&p->t256, W, N, K, ldw, 256)) return -1;
    if (make_tmap(&p->t128, W, N, K, ldw, 128)) return -1;
    p->magic = P3_WPLAN_MAGIC;
    return 0;
}

// struct-argument entry: everything p3_gemm does + the fused prefill epilogues
extern "C" int p3_gemm_fused(const p3_gemm_args* a, cudaStream_t st) {
    P3_CHECK_ARG(a, "gemm_fused: null args");
    const int epi = a->epi;
    P3_CHECK_ARG((epi >= P3_EPI_NONE && epi <= P3_EPI_RESIDUAL_F32) || epi == P3_EPI_ROPE_KV, "gemm_fused: unknown epilogue %d", epi);
    P3_CHECK_ARG(a->ldx % 8 == 0 && a->ldw % 8 == 0, "gemm_fused: ldx/ldw must be multiples of 8 elements (16 B)");
    P3_CHECK_ARG(((uintptr_t)a->X & 15) == 0 && ((uintptr_t)a->W & 15) == 0, "gemm_fused: X/W must be 16-byte aligned");
    P3_CHECK_ARG((epi != P3_EPI_RESIDUAL && epi != P3_EPI_RESIDUAL_F32) || a->resid, "gemm_fused: residual epilogue needs resid");
    P3_CHECK_ARG(epi != P3_EPI_SWIGLU || (a->N % 256 == 0 && !a->bias), "gemm_fused: SwiGLU needs N %% 256 == 0 and no bias");
    P3_CHECK_ARG(!a->ss_out || (epi == P3_EPI_RESIDUAL && a->N % 32 == 0 && !a->row_map), "gemm_fused: ss_out needs the bf16 residual epilogue, N %% 32 == 0");
    P3_CHECK_ARG(!a->ss_in || (a->n_ss_in >= 1 && !a->row_map), "gemm_fused: ss_in needs n_ss_in >= 1 and no row map");
    P3_CHECK_ARG(a->M < (1ll << 31), "gemm_fused: M too large");
    if (a->M == 0) return 0;
    GemmEpi ep{};
    ep.bias = (const bf16*)a->bias; ep.out = a->out; ep.ldo = a->ldo; ep.resid = a->resid; ep.row_map = a->row_map; ep.kind = epi;
    ep.ss_in = a->ss_in; ep.n_ss_in = a->n_ss_in; ep.eps = a->eps; ep.ss_out = a->ss_out;
    if (epi == P3_EPI_ROPE_KV) {
        P3_CHECK_ARG(a->hd % 32 == 0 && a->N == (a->n_heads + 2 * a->n_kv) * a->hd && a->ldo % 8 == 0 && !a->bias && !a->row_map,
                     "gemm_fused: ROPE_KV needs head_dim %% 32 == 0, N = (n_heads + 2 n_kv) * head_dim, no bias / row map");
        P3_CHECK_ARG(a->cosT && a->sinT && a->L >= 1 && a->row_div >= 1 && a->M % a->L == 0, "gemm_fused: ROPE_KV needs rope tables and M = B * L");
        P3_CHECK_ARG(!a->write_cache || (a->pool && a->block_table), "gemm_fused: cache write needs pool and block table");
        ep.cosT = a->cosT; ep.sinT = a->sinT; ep.tab_bstride = a->tab_bstride; ep.L = a->L; ep.n_heads = a->n_heads; ep.n_kv = a->n_kv;
        ep.hd = a->hd; ep.past = a->past; ep.row_div = a->row_div; ep.write_cache = a->write_cache; ep.past_dev = a->past_dev;
        ep.pool = (bf16*)a->pool; ep.block_table = a->block_table; ep.bt_stride = a->bt_stride;
    }
    ep.ws = reinterpret_cast<float*>(a->splitk_ws); ep.ws_bytes = a->splitk_ws ? a->splitk_ws_bytes : 0;   // carved up by launch_tc
    const GemmWPlan* wp = reinterpret_cast<const GemmWPlan*>(a->w_plan);
    if (wp) P3_CHECK_ARG(wp->magic == P3_WPLAN_MAGIC && wp->W == a->W && wp->ldw == a->ldw && wp->N == a->N && wp->K == a->K,
                         "gemm_fused: weight plan does not describe this W");
    return gemm_dispatch(a->X, a->ldx, a->W, a->ldw, ep, a->M, a->N, a->K, a->impl, st, wp);
}
