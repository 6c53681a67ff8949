// bf16 q_len = 1 decode with the score and value products on the warp-level tensor cores.
//
// The streaming SIMT decode kernel issues ~120 warp instructions per (token, KV head) and is
// issue-bound at a third of HBM bandwidth.  Here one warp still owns one KV head of one
// (sequence, KV chunk) and still reads every K/V byte once with 16-byte loads, but the loaded
// registers are used directly as mma.sync.m16n8k16 fragments, about 8 instructions per token:
//
//   S^T[16 tokens x 8 heads] = K[16 tokens x D] * Q^T[D x 8 heads]
//       A = K: thread (g = lane/4, c = lane%4) loads 16 bytes (8 dims) of tokens g and g+8 per
//       32-dim chunk; a dot product does not care in which order dims are summed, so the 8
//       contiguous dims are assigned to the fragment's k-slots of two k-steps and Q^T uses the same
//       assignment.  Q^T (B operand) is built once: rotated at the query position in f32, scaled by
//       scale*log2(e), split into bf16 hi + lo so the rotation does not lose precision.
//   O^T[D x 8 heads] += V^T[D x 16 tokens] * P^T[16 tokens x 8 heads]
//       A = V^T: thread loads 16 dims of tokens 2c, 2c+1, 2c+8, 2c+9 and pairs the same dim of two
//       tokens with byte permutes; which dim lands in which output row is bookkeeping only.
//       B = P^T: the packed S^T accumulators transposed with movmatrix.
//
// Heads of the group sit on the n = 8 axis (group <= 8).  Softmax state (running max, partial sums)
// is per head; the max is made warp-consistent with three shuffles per tile, the sums are reduced
// once at the end.  Chunks of one sequence are merged by the same merge kernel as the SIMT path.
#include <cooperative_groups.h>

#include "common.h"

namespace flat {
namespace {

namespace cg = cooperative_groups;

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// K and V are read once.  Not through the read-only path (.nc): the kernel may be resident while the one before it in the
// stream still writes them (launch_dependent()), and .nc is for memory that nobody writes while the kernel runs.
__device__ __forceinline__ uint4 ld_stream(const void *p) {
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
}

__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The page table of a launch: in device memory, or (a single short sequence) among the kernel's arguments.  A type and not
// a pointer that could be either: through a generic pointer every page lookup of a long context is slower (decode of 64
// sequences of 512 to 8192 tokens 194 -> 218 us).
struct DeviceTable {
    __device__ __forceinline__ int page(const DecodeParams &p, int seq, int i) const {
        return p.page_table[(int64_t)seq * p.max_pages + i];
    }
};
struct InlineTable {
    int32_t pages[kInlinePages];
    __device__ __forceinline__ int page(const DecodeParams &, int, int i) const { return pages[i]; }
};

// Q^T fragments of a warp: head g of the group, dims 32j + 8c .. +7, rotated, scaled, split hi/lo.
// The rotation angle depends on (position, pair) only, so the warp evaluates each of the D/2 pairs once
// (lane l takes pairs l and l + 32; at long-context positions sincosf runs its slow argument reduction)
// and the fragments fetch their (cos, sin) with shuffles: pair 16j + 4c + e sits in lane
// 16 (j mod 2) + 4c + e, slot j / 2.
template <int D>
__device__ __forceinline__ void build_q(const DecodeParams &p, int seq, int kv_head, uint32_t (&qhi)[D / 32][4], uint32_t (&qlo)[D / 32][4]) {
    constexpr int kChunks = D / 32;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, c = lane & 3;
    const int G = p.group;
    const int64_t q_pos = p.q_rope_positions ? (int64_t)p.q_rope_positions[seq] : p.uniform_q_pos;
    const float fold = p.scale * kLog2e;
    constexpr int kSlots = D / 64;
    float cs_c[kSlots], cs_s[kSlots];
#pragma unroll
    for (int sl = 0; sl < kSlots; ++sl) {
        cs_c[sl] = 1.f;
        cs_s[sl] = 0.f;
        if (p.rope_q) sincosf(__fmul_rn((float)q_pos, p.inv_freq[lane + 32 * sl]), &cs_s[sl], &cs_c[sl]);
    }
#pragma unroll
    for (int j = 0; j < kChunks; ++j) {
        uint4 raw = make_uint4(0, 0, 0, 0);
        if (g < G)
            raw = *reinterpret_cast<const uint4 *>((const __nv_bfloat16 *)p.q +
                                                   ((int64_t)seq * p.q_heads + kv_head * G + g) * D + 32 * j + 8 * c);
        const uint32_t rr[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int src = 16 * (j & 1) + 4 * c + e;
            const float co = __shfl_sync(0xffffffffu, cs_c[j >> 1], src), s = __shfl_sync(0xffffffffu, cs_s[j >> 1], src);
            float x = __uint_as_float(rr[e] << 16), y = __uint_as_float(rr[e] & 0xffff0000u);
            const float rx = x * co - y * s, ry = x * s + y * co;  // (cos, sin) = (1, 0) without RoPE: exact
            x = rx * fold;
            y = ry * fold;
            const __nv_bfloat162 hi = __floats2bfloat162_rn(x, y);
            const float2 hf = __bfloat1622float2(hi);
            qhi[j][e] = *reinterpret_cast<const uint32_t *>(&hi);
            qlo[j][e] = pack_bf16(x - hf.x, y - hf.y);
        }
    }
}

// Fragments of 16 tokens of one KV head: K rows g, g+8 (8 dims per 32-dim chunk); V rows 2c, 2c+1, 2c+8, 2c+9 (D/8 dims).
template <int D> struct TileRegs {
    uint4 ka[D / 32], kb[D / 32], vv[4][D / 64];
};

// Row of the cache where the 16 tokens from t0 on start; < 0: the page-table entry is outside the pool, which flags the call.
template <typename Table>
__device__ __forceinline__ int64_t tile_row(const DecodeParams &p, const Table &table, int seq, int t0) {
    if (!p.page_size) return (int64_t)seq * p.seq_stride_rows + t0;
    const int page = table.page(p, seq, t0 / p.page_size);
    // an entry outside the pool is never dereferenced: the tile is skipped and the call is flagged
    if ((unsigned)page >= (unsigned)p.physical_pages) {
        if ((threadIdx.x & 31) == 0 && p.status) {
            p.status->code = FLAT_ERR_PAGE_OUT_OF_RANGE;
            p.status->where = seq;
        }
        return -1;
    }
    return (int64_t)page * p.page_size + t0 % p.page_size;
}

// `left`: live tokens of the tile (16 or more: all of them)
template <int D>
__device__ __forceinline__ void load_tile(const DecodeParams &p, int kv_head, int64_t row0, int left, TileRegs<D> &x) {
    constexpr int kChunks = D / 32, kVecs = D / 64;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, c = lane & 3;
    const int64_t row_bytes = (int64_t)p.kv_heads * D * 2;
    const int64_t head_bytes = (int64_t)kv_head * D * 2;
    const char *ktile = (const char *)p.k + row0 * row_bytes + head_bytes;
    const char *vtile = (const char *)p.v + row0 * row_bytes + head_bytes;
    const bool ok_a = g < left, ok_b = g + 8 < left;
#pragma unroll
    for (int j = 0; j < kChunks; ++j) {
        x.ka[j] = ok_a ? ld_stream(ktile + (int64_t)g * row_bytes + (32 * j + 8 * c) * 2) : make_uint4(0, 0, 0, 0);
        x.kb[j] = ok_b ? ld_stream(ktile + (int64_t)(g + 8) * row_bytes + (32 * j + 8 * c) * 2) : make_uint4(0, 0, 0, 0);
    }
    const int vt[4] = {2 * c, 2 * c + 1, 2 * c + 8, 2 * c + 9};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool ok = vt[i] < left;
#pragma unroll
        for (int u = 0; u < kVecs; ++u)
            x.vv[i][u] = ok ? ld_stream(vtile + (int64_t)vt[i] * row_bytes + ((D / 8) * g + 8 * u) * 2) : make_uint4(0, 0, 0, 0);
    }
}

// Softmax state of a warp: thread (g, c) holds heads 2c, 2c+1 and dims (D/8)*g .. +D/8-1 (acc[i][0], acc[i][2] interleaved);
// the sums are those of the thread's own tokens until reduce_sums().
template <int D> struct WarpState {
    float acc[D / 16][4];
    float m0, m1, l0, l1;
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < D / 16; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
        m0 = m1 = -INFINITY;
        l0 = l1 = 0.f;
    }
    __device__ __forceinline__ void reduce_sums() {
#pragma unroll
        for (int w = 4; w < 32; w <<= 1) {
            l0 += __shfl_xor_sync(0xffffffffu, l0, w);
            l1 += __shfl_xor_sync(0xffffffffu, l1, w);
        }
    }
};

template <int D>
__device__ __forceinline__ void take_tile(const uint32_t (&qhi)[D / 32][4], const uint32_t (&qlo)[D / 32][4], const TileRegs<D> &x, int left,
                                          WarpState<D> &st) {
    constexpr int kChunks = D / 32, kVecs = D / 64, kPv = D / 16;
    const int g = (threadIdx.x & 31) >> 2;
    // ---- S^T = K Q^T (hi + lo)
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < kChunks; ++j) {
        mma_bf16(s, x.ka[j].x, x.kb[j].x, x.ka[j].y, x.kb[j].y, qhi[j][0], qhi[j][1]);
        mma_bf16(s, x.ka[j].z, x.kb[j].z, x.ka[j].w, x.kb[j].w, qhi[j][2], qhi[j][3]);
        mma_bf16(s, x.ka[j].x, x.kb[j].x, x.ka[j].y, x.kb[j].y, qlo[j][0], qlo[j][1]);
        mma_bf16(s, x.ka[j].z, x.kb[j].z, x.ka[j].w, x.kb[j].w, qlo[j][2], qlo[j][3]);
    }
    if (g >= left) s[0] = s[1] = -INFINITY;
    if (g + 8 >= left) s[2] = s[3] = -INFINITY;

    // ---- online softmax per head (columns 2c, 2c+1); tokens live on g: reduce over lanes 4, 8, 16
    const float m0 = st.m0, m1 = st.m1;
    float mx0 = fmaxf(s[0], s[2]), mx1 = fmaxf(s[1], s[3]);
#pragma unroll
    for (int w = 4; w < 32; w <<= 1) {
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, w));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, w));
    }
    st.m0 = fmaxf(st.m0, mx0);
    st.m1 = fmaxf(st.m1, mx1);
    // every score so far -inf: their exponentials are 0 (a NaN stays one)
    const float n0 = st.m0 == -INFINITY ? 0.f : st.m0, n1 = st.m1 == -INFINITY ? 0.f : st.m1;
    const float a0 = ex2f(m0 - n0), a1 = ex2f(m1 - n1);  // m = -inf gives 0
    s[0] = ex2f(s[0] - n0);
    s[2] = ex2f(s[2] - n0);
    s[1] = ex2f(s[1] - n1);
    s[3] = ex2f(s[3] - n1);
    st.l0 = st.l0 * a0 + s[0] + s[2];
    st.l1 = st.l1 * a1 + s[1] + s[3];
    if (__any_sync(0xffffffffu, a0 != 1.0f || a1 != 1.0f)) {
#pragma unroll
        for (int i = 0; i < kPv; ++i) {
            st.acc[i][0] *= a0;
            st.acc[i][2] *= a0;
            st.acc[i][1] *= a1;
            st.acc[i][3] *= a1;
        }
    }
    const uint32_t b0 = movmatrix_trans(pack_bf16(s[0], s[1]));  // {P[2c][g], P[2c+1][g]}
    const uint32_t b1 = movmatrix_trans(pack_bf16(s[2], s[3]));  // {P[2c+8][g], P[2c+9][g]}

    // ---- O^T += V^T P^T: mma i covers dims (D/8)*g + 2i (row g) and + 2i + 1 (row g + 8)
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
        const uint32_t r0[4] = {x.vv[0][u].x, x.vv[0][u].y, x.vv[0][u].z, x.vv[0][u].w};
        const uint32_t r1[4] = {x.vv[1][u].x, x.vv[1][u].y, x.vv[1][u].z, x.vv[1][u].w};
        const uint32_t r2[4] = {x.vv[2][u].x, x.vv[2][u].y, x.vv[2][u].z, x.vv[2][u].w};
        const uint32_t r3[4] = {x.vv[3][u].x, x.vv[3][u].y, x.vv[3][u].z, x.vv[3][u].w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            mma_bf16(st.acc[u * 4 + e], __byte_perm(r0[e], r1[e], 0x5410), __byte_perm(r0[e], r1[e], 0x7632),
                     __byte_perm(r2[e], r3[e], 0x5410), __byte_perm(r2[e], r3[e], 0x7632), b0, b1);
    }
}

// One warp: KV head `kv_head` of sequence `seq`, tokens [begin, end) (begin a multiple of 16).
// to_partial: write the normalised (O, LSE) of this range to partial slot `slot`, else the final result.
template <int D, typename Table>
__device__ __forceinline__ void decode_range(const DecodeParams &p, const Table &table, int seq, int kv_head, int begin, int end, int slot,
                                             bool to_partial) {
    constexpr int kPv = D / 16;       // PV mma per tile
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, c = lane & 3;
    const int split = slot;
    const int G = p.group;
    uint32_t qhi[D / 32][4], qlo[D / 32][4];
    build_q<D>(p, seq, kv_head, qhi, qlo);
    WarpState<D> st;
    st.clear();
    for (int t0 = begin; t0 < end; t0 += 16) {
        const int64_t row0 = tile_row(p, table, seq, t0);
        if (row0 < 0) continue;
        TileRegs<D> x;
        load_tile<D>(p, kv_head, row0, end - t0, x);
        take_tile<D>(qhi, qlo, x, end - t0, st);
    }
    st.reduce_sums();

    // thread (g, c) holds heads 2c, 2c+1 and dims (D/8)*g .. +D/8-1 (acc[i][0], acc[i][2] interleaved)
    constexpr int kDims = D / 8;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int head_in_group = 2 * c + hh;
        if (head_in_group >= G) continue;
        const float m = hh ? st.m1 : st.m0, l = hh ? st.l1 : st.l0;
        // l == 0 only when every tile of the range was skipped (flagged page-table entries): O = 0, LSE = -inf
        const float inv = l > 0.f ? 1.0f / l : 0.f;
        const float lse = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
        const int64_t out_row = (int64_t)seq * p.q_heads + kv_head * G + head_in_group;
        float vals[kDims];
#pragma unroll
        for (int i = 0; i < kPv; ++i) {
            vals[2 * i] = st.acc[i][hh] * inv;
            vals[2 * i + 1] = st.acc[i][2 + hh] * inv;
        }
        if (to_partial) {
            float *po = p.partial_o + ((int64_t)split * p.num_seqs * p.q_heads + out_row) * D + kDims * g;
#pragma unroll
            for (int e = 0; e < kDims; e += 4)
                *reinterpret_cast<float4 *>(po + e) = make_float4(vals[e], vals[e + 1], vals[e + 2], vals[e + 3]);
            if (g == 0) p.partial_lse[(int64_t)split * p.num_seqs * p.q_heads + out_row] = lse;
        } else if (p.out_f32) {
            float *po = (float *)p.o + out_row * D + kDims * g;
#pragma unroll
            for (int e = 0; e < kDims; e += 4)
                *reinterpret_cast<float4 *>(po + e) = make_float4(vals[e], vals[e + 1], vals[e + 2], vals[e + 3]);
            if (g == 0) p.lse[out_row] = lse;
        } else {
            __nv_bfloat16 *op = (__nv_bfloat16 *)p.o + out_row * D + kDims * g;
#pragma unroll
            for (int e = 0; e < kDims; e += 8) {
                uint4 pk;
                pk.x = pack_bf16(vals[e], vals[e + 1]);
                pk.y = pack_bf16(vals[e + 2], vals[e + 3]);
                pk.z = pack_bf16(vals[e + 4], vals[e + 5]);
                pk.w = pack_bf16(vals[e + 6], vals[e + 7]);
                *reinterpret_cast<uint4 *>(op + e) = pk;
            }
            if (g == 0) p.lse[out_row] = lse;
        }
    }
}

// Short contexts: one launch and no partials in memory.  A cluster of up to kMaxDecodeCluster CTAs takes one KV head of one
// sequence; its warps split the tokens, a CTA combines its warps in shared memory, and the CTAs of the cluster read one
// another's results there (distributed shared memory), each finishing its share of the (head, dim) outputs, in warp and rank
// order.  Bound by latency: set-up, one round of K and V loads (the first is requested before Q is rotated, the next before
// a tile is worked on), two barriers.
constexpr int kClusterWarps = 8;
constexpr int kClusterTiles = 4;  // most 16-token tiles of a warp
template <int D, typename Table>
__global__ void __launch_bounds__(32 * kClusterWarps, 1)
    decode_cluster_kernel(const __grid_constant__ DecodeParams p, const __grid_constant__ Table table) {
    __shared__ __align__(16) float part_o[kClusterWarps][8][D];
    __shared__ float2 part_ml[kClusterWarps][8];
    __shared__ __align__(16) float cta_o[8 * D];
    __shared__ float2 cta_ml[8];
    grid_dependency_wait();
    grid_dependency_launch();
    cg::cluster_group cluster = cg::this_cluster();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, c = lane & 3;
    const int ranks = (int)gridDim.x, rank = (int)blockIdx.x;
    const int kv_head = blockIdx.y, seq = blockIdx.z;
    const int G = p.group;
    const int len = p.context_lens ? p.context_lens[seq] : p.uniform_len;
    const int tiles = (len + 15) / 16, warps = ranks * kClusterWarps;
    const int per = (tiles + warps - 1) / warps;  // tiles of a warp
    const int begin = min(tiles, (rank * kClusterWarps + warp) * per) * 16, end = min(len, begin + per * 16);

    WarpState<D> st;
    st.clear();
    if (begin < end) {
        TileRegs<D> x;
        int64_t row = tile_row(p, table, seq, begin);
        if (row >= 0) load_tile<D>(p, kv_head, row, end - begin, x);
        uint32_t qhi[D / 32][4], qlo[D / 32][4];
        build_q<D>(p, seq, kv_head, qhi, qlo);
        for (int t0 = begin; t0 < end; t0 += 16) {
            TileRegs<D> next;
            int64_t next_row = -1;
            if (t0 + 16 < end) {
                next_row = tile_row(p, table, seq, t0 + 16);
                if (next_row >= 0) load_tile<D>(p, kv_head, next_row, end - t0 - 16, next);
            }
            if (row >= 0) take_tile<D>(qhi, qlo, x, end - t0, st);
            x = next;
            row = next_row;
        }
        st.reduce_sums();
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int h = 2 * c + hh;
        if (h >= G) continue;
        const float m = hh ? st.m1 : st.m0, l = hh ? st.l1 : st.l0;
        // A warp without a live token, or whose scores are all -inf, counts for nothing.  A NaN score makes l NaN: such a part
        // counts, here and below, so that O and LSE of the head come out NaN and not as those of the other warps' tokens.
        const bool live = l != 0.f;
        float *to = &part_o[warp][h][(D / 8) * g];
#pragma unroll
        for (int i = 0; i < D / 16; i += 2)
            *reinterpret_cast<float4 *>(to + 2 * i) =
                live ? make_float4(st.acc[i][hh], st.acc[i][2 + hh], st.acc[i + 1][hh], st.acc[i + 1][2 + hh])
                     : make_float4(0.f, 0.f, 0.f, 0.f);
        if (g == 0) part_ml[warp][h] = live ? make_float2(m, l) : make_float2(-INFINITY, 0.f);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < G * D; i += 32 * kClusterWarps) {
        const int h = i / D, d = i % D;
        float mx = -INFINITY, sum = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < kClusterWarps; ++w) mx = fmaxf(mx, part_ml[w][h].x);
#pragma unroll
        for (int w = 0; w < kClusterWarps; ++w) {
            const float2 ml = part_ml[w][h];
            const float f = ml.y == 0.f ? 0.f : ex2f(ml.x - mx);
            sum = fmaf(f, ml.y, sum);
            o = fmaf(f, part_o[w][h][d], o);
        }
        cta_o[i] = o;
        if (d == 0) cta_ml[h] = make_float2(mx, sum);
    }
    cluster.sync();
    // this CTA's share of the outputs, two adjacent dims per thread
    const int pairs = G * D / 2, share = (pairs + ranks - 1) / ranks;
    for (int i = rank * share + threadIdx.x; i < min(pairs, (rank + 1) * share); i += 32 * kClusterWarps) {
        const int h = 2 * i / D, d = 2 * i % D;
        float2 ml[kMaxDecodeCluster], x[kMaxDecodeCluster];
        float mx = -INFINITY, sum = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int r = 0; r < kMaxDecodeCluster; ++r) {
            ml[r] = make_float2(-INFINITY, 0.f);
            x[r] = make_float2(0.f, 0.f);
            if (r < ranks) {
                ml[r] = cluster.map_shared_rank(cta_ml, r)[h];
                x[r] = *reinterpret_cast<const float2 *>(cluster.map_shared_rank(cta_o, r) + 2 * i);
            }
            mx = fmaxf(mx, ml[r].x);
        }
#pragma unroll
        for (int r = 0; r < kMaxDecodeCluster; ++r) {
            const float f = ml[r].y == 0.f ? 0.f : ex2f(ml[r].x - mx);
            sum = fmaf(f, ml[r].y, sum);
            o0 = fmaf(f, x[r].x, o0);
            o1 = fmaf(f, x[r].y, o1);
        }
        // nothing counts only when every tile was skipped (flagged page-table entries): O = 0, LSE = -inf
        const bool empty = sum == 0.f;
        const float inv = empty ? 0.f : 1.0f / sum;
        const int64_t row = (int64_t)seq * p.q_heads + kv_head * G + h;
        if (p.out_f32) *reinterpret_cast<float2 *>((float *)p.o + row * D + d) = make_float2(o0 * inv, o1 * inv);
        else *reinterpret_cast<uint32_t *>((__nv_bfloat16 *)p.o + row * D + d) = pack_bf16(o0 * inv, o1 * inv);
        if (d == 0) p.lse[row] = empty ? -INFINITY : (mx + log2f(sum)) * kLn2;
    }
    cluster.sync();  // the others have read this CTA's shared memory
}

template <int D, typename Table>
__global__ void __launch_bounds__(256, 2) decode_mma_kernel(const __grid_constant__ DecodeParams p, const __grid_constant__ Table table) {
    grid_dependency_wait();
    const int warp = threadIdx.x >> 5;
    const int kv_head = blockIdx.y * (blockDim.x >> 5) + warp;
    if (kv_head >= p.kv_heads) return;
    if (!p.balanced) {
        const int seq = blockIdx.z;
        const int split = blockIdx.x;
        const int ctx_len = p.context_lens ? p.context_lens[seq] : p.uniform_len;
        int begin = 0, end = ctx_len;
        if (p.kv_splits > 1) {
            begin = split * p.chunk_tokens;
            end = min(ctx_len, begin + p.chunk_tokens);
            if (begin >= end) return;
        }
        decode_range<D>(p, table, seq, kv_head, begin, end, split, p.kv_splits > 1);
        return;
    }
    // balanced: this CTA streams [cta*span, (cta+1)*span) of the concatenated (16-padded) sequences
    const int cta = blockIdx.x;
    const int total = p.seq_offsets[p.num_seqs];
    int pos = cta * p.span_tokens;
    const int span_end = min(total, pos + p.span_tokens);
    if (pos >= span_end) return;
    int seq = 0;
    while (seq + 1 < p.num_seqs && p.seq_offsets[seq + 1] <= pos) ++seq;
    while (pos < span_end) {
        const int off = p.seq_offsets[seq], next = p.seq_offsets[seq + 1];
        const int seg_end = min(span_end, next);
        const int ctx_len = p.context_lens ? p.context_lens[seq] : p.uniform_len;
        const int first_cta = off / p.span_tokens, last_cta = (next - 1) / p.span_tokens;
        decode_range<D>(p, table, seq, kv_head, pos - off, min(ctx_len, seg_end - off), cta - first_cta, last_cta > first_cta);
        pos = seg_end;
        ++seq;
    }
}

}  // namespace

bool decode_mma_supported(int dtype, const DecodeParams &p) {
    if (dtype != FLAT_BF16) return false;
    if (p.head_dim != 64 && p.head_dim != 128) return false;
    if (p.group > 8) return false;
    if (p.page_size != 0 && p.page_size % 16 != 0) return false;  // a 16-token tile must stay inside one page
    if (p.kv_splits > 1 && p.chunk_tokens % 16 != 0) return false;
    return true;
}

// CTAs per KV head for a batch whose longest context has `max_len` tokens, or 0: the spans of decode_mma_kernel.  One tile per
// warp where the CTAs suffice, up to kClusterTiles; all clusters have to be resident at once, which with one CTA per SM more
// than eight of the largest are not (16 KV heads, 1000 tokens: 12.3 us with 16 clusters of eight, 10.3 with spans and a merge).
// Spans and merge / cluster, launches not yet overlapped (common.h), D = 128, 32 / 8 heads: 700 tokens 10.3 / 8.2 us, 2000
// 12.3 / 10.3, 4096 14.4 / 13.3 (overlapped 6.7, 8.0 and 10.4); 64 / 8 heads, 300 10.3 / 9.0, 3500 14.4 / 14.3; 16 / 16 heads,
// 400 10.3 / 8.2; four sequences of up to 1500 tokens 17.5 / 14.8, 16 of up to 500 20.4 / 15.0; D = 64, 16 / 4 heads, 300 9.0 /
// 7.0, 4096 10.2 / 10.3.
int decode_cluster_size(const flat_ctx *ctx, const DecodeParams &p, int max_len) {
    if (p.kv_heads > 65535 || p.num_seqs > 65535 || max_len < 1) return 0;
    const int tiles = (max_len + 15) / 16;
    const int64_t units = (int64_t)p.num_seqs * p.kv_heads;
    int c = 1;
    while (c < kMaxDecodeCluster && c * kClusterWarps < tiles) c *= 2;
    while (c > 1 && units * c > (c == kMaxDecodeCluster ? 8 * kMaxDecodeCluster : ctx->sm_count)) c /= 2;
    if (units * c > ctx->sm_count) return 0;
    return tiles <= kClusterTiles * c * kClusterWarps ? c : 0;
}

template <int D, typename Table>
static cudaError_t launch_cluster(flat_ctx *ctx, const DecodeParams &p, const Table &table) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)p.cluster, (unsigned)p.kv_heads, (unsigned)p.num_seqs);
    cfg.blockDim = dim3(32 * kClusterWarps);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {(unsigned)p.cluster, 1, 1};
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch_dependent()
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = may_overlap_previous(ctx) ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, decode_cluster_kernel<D, Table>, p, table);
}

int launch_decode_mma(flat_ctx *ctx, const DecodeParams &p) {
    if (p.cluster) {
        KernelTimer timer(ctx);
        if (p.host_pages) {
            InlineTable table;
            std::copy(p.host_pages, p.host_pages + p.max_pages, table.pages);
            FLAT_CUDA_OK(ctx, p.head_dim == 128 ? launch_cluster<128>(ctx, p, table) : launch_cluster<64>(ctx, p, table));
        } else {
            FLAT_CUDA_OK(ctx, p.head_dim == 128 ? launch_cluster<128>(ctx, p, DeviceTable{}) : launch_cluster<64>(ctx, p, DeviceTable{}));
        }
        return FLAT_OK;
    }
    const int warps = p.kv_heads < 8 ? p.kv_heads : 8;
    dim3 grid(p.kv_splits, (p.kv_heads + warps - 1) / warps, p.num_seqs);
    if (p.balanced) grid = dim3(p.num_ctas, (p.kv_heads + warps - 1) / warps, 1);
    const bool overlap = may_overlap_previous(ctx);
    KernelTimer timer(ctx);
    if (p.host_pages) {
        InlineTable table;
        std::copy(p.host_pages, p.host_pages + p.max_pages, table.pages);
        FLAT_CUDA_OK(ctx, launch_dependent(overlap, p.head_dim == 128 ? decode_mma_kernel<128, InlineTable> : decode_mma_kernel<64, InlineTable>,
                                           grid, warps * 32, 0, ctx->stream, p, table));
    } else {
        FLAT_CUDA_OK(ctx, launch_dependent(overlap, p.head_dim == 128 ? decode_mma_kernel<128, DeviceTable> : decode_mma_kernel<64, DeviceTable>,
                                           grid, warps * 32, 0, ctx->stream, p, DeviceTable{}));
    }
    return FLAT_OK;
}

}  // namespace flat
