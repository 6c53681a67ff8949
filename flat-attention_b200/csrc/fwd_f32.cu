// f32 forward for head_dim 64 and 128: register-tiled products on the FMA pipe.
//
// Bound by the f32 FMA pipe (128 lanes per clock and SM; the tensor cores have no f32 mode of this precision), so both
// products are laid out to feed it: a CTA owns 64 query rows of one (batch, q_head) and streams K/V tiles of 64 keys
// through shared memory; at D = 128 256 threads hold 4 rows x 4 keys of the scores and 4 rows x D/16 columns of O in
// registers, at D = 64 128 threads twice that, so a 16-byte shared-memory read serves 8 to 13 multiply-adds (the
// row-per-four-threads kernel in fwd_simt.cu reads one K and one V vector for four).  Products run as packed f32x2 FMAs: a
// score is two running sums (even and odd dimensions) over each half of the head dimension, an O pair is two adjacent columns.
// Few query blocks leave most SMs idle and the causal diagonal makes them uneven, so the KV tiles of a query block are
// dealt to a cluster of up to 8 CTAs, which combine their (max, sum, O) through distributed shared memory in rank
// order: one launch, no scratch, bitwise repeatable.  8 / 2 heads, 512 rows, D = 128, causal, RoPE: 219 us with the kernel of
// fwd_simt.cu, 42 us here; 2 x 2048 rows, 16 / 4 heads 3470 us and 1180 us (29 TFLOP/s).
// RoPE: K and Q are rotated on the way into shared memory with the (cos, sin) table of the call's positions (find_tables());
// without one the same sincosf runs here.
#include <cooperative_groups.h>

#include <cstring>
#include <type_traits>

#include "common.h"

namespace flat {
namespace {

namespace cg = cooperative_groups;

constexpr int kRows = 64;    // query rows per CTA
constexpr int kKeys = 64;    // keys per tile
// tx: lanes that share a row.  Twice the threads with half the tile each hide more of the shared-memory latency at D = 128 (8 / 2
// heads: 356 rows 41.3 -> 37.0 us, 512 rows 45.1 -> 43.6, 2 x 2048 rows, 16 / 4 heads 1207 both); at D = 64 a read then serves too
// few multiply-adds (1784 rows 164 -> 166 us, 2 x 2048 rows without a mask 1049 -> 1068).  The 128 registers of the 256 threads
// do not hold all of it: 80 bytes of a thread spill, 64 with ALiBi.
template <int D> constexpr int kLanes = D == 128 ? 16 : 8;
template <int D> constexpr int kThreads = kRows / 4 * kLanes<D>;
constexpr int kRowsPerThread = 4;   // ty + 16 r
template <int D> constexpr int kKeysPerThread = kKeys / kLanes<D>;  // tx + kLanes i
constexpr int kMaxCluster = 8;

struct F32Params {
    FwdParams f;
    const float2 *q_table, *k_table;  // (cos, sin) of query row / key r, pair j at [r * D/2 + j]
};

template <int D> struct Tile {
    static constexpr int kStride = D + 4;       // floats per Q / K row: 8 rows cover all banks
    static constexpr int kPStride = kKeys + 4;  // P takes K's place
    static constexpr int kQ = 0, kK = kRows * kStride, kV = kK + kKeys * kStride, kStat = kV + kKeys * D;
    static constexpr int kFloats = kStat + 2 * kRows;
    static_assert(kPStride <= kStride, "P fits K's rows");
};

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void mul2(uint64_t &d, uint64_t a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }

__device__ __forceinline__ void cp_async16(float *dst, const float *src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(live ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// 64 rows of `src` (row stride rs) into dst (row stride `stride`) with cp.async; rows from `live` on become zero.
template <int D>
__device__ __forceinline__ void load_rows(float *dst, int stride, const float *src, int64_t rs, int64_t first, int live) {
    constexpr int kVec = D / 4;
#pragma unroll
    for (int u = 0; u < 64 * kVec / kThreads<D>; ++u) {
        const int i = u * kThreads<D> + threadIdx.x, r = i / kVec, v = i % kVec;
        cp_async16(dst + r * stride + 4 * v, src + (first + (r < live ? r : 0)) * rs + 4 * v, r < live);
    }
}
// Whether the part of those rows that this thread copied (and has waited for) holds an infinity or NaN: 0 times it is NaN.
template <int D>
__device__ __forceinline__ bool copied_non_finite(const float *src) {
    constexpr int kVec = D / 4;
    uint64_t zero[4] = {};
#pragma unroll 2
    for (int u = 0; u < 64 * kVec / kThreads<D>; ++u) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(src + 4 * (u * kThreads<D> + threadIdx.x));
        fma2(zero[2 * u & 3], x.x, 0);
        fma2(zero[2 * u + 1 & 3], x.y, 0);
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) sum += unpack2(zero[i]).x + unpack2(zero[i]).y;
    return sum != 0.f;  // true for NaN
}
// The same with the interleaved pairs of row r rotated by the table's row first + r, or by the angle of position
// pos0 + first + r.  A thread's loads are in flight eight at a time: the tile waits for the last of them.
template <int D>
__device__ __forceinline__ void load_rotated_rows(float *dst, int stride, const float *src, int64_t rs, int64_t first, int live,
                                                  const float2 *table, int64_t pos0, const float *inv_freq) {
    constexpr int kVec = D / 4, kBatch = 64 * kVec / kThreads<D> < 8 ? 64 * kVec / kThreads<D> : 8;
#pragma unroll
    for (int u0 = 0; u0 < 64 * kVec / kThreads<D>; u0 += kBatch) {
        float4 x[kBatch], cs[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = (u0 + u) * kThreads<D> + threadIdx.x, r = i / kVec, v = i % kVec;
            x[u] = *reinterpret_cast<const float4 *>(src + (first + (r < live ? r : 0)) * rs + 4 * v);
        }
        if (table) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int i = (u0 + u) * kThreads<D> + threadIdx.x, r = i / kVec, v = i % kVec;
                cs[u] = *reinterpret_cast<const float4 *>(table + (first + (r < live ? r : 0)) * (D / 2) + 2 * v);
            }
        } else {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int i = (u0 + u) * kThreads<D> + threadIdx.x, r = i / kVec, v = i % kVec;
                const float pos = (float)(pos0 + first + r);
                sincosf(__fmul_rn(pos, inv_freq[2 * v]), &cs[u].y, &cs[u].x);
                sincosf(__fmul_rn(pos, inv_freq[2 * v + 1]), &cs[u].w, &cs[u].z);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = (u0 + u) * kThreads<D> + threadIdx.x, r = i / kVec, v = i % kVec;
            const float4 y = x[u], c = cs[u];
            *reinterpret_cast<float4 *>(dst + r * stride + 4 * v) =
                r < live ? make_float4(y.x * c.x - y.y * c.y, y.x * c.y + y.y * c.x, y.z * c.z - y.w * c.w, y.z * c.w + y.w * c.z)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

// O += P V of a tile of which row r of the thread sees the first `seen` + 16 r keys.  Not inlined: a call of it is rare, and
// its code beside the plain loop costs that one registers.
template <int D>
__device__ __noinline__ void accumulate_seen(uint64_t *o, const float *ps, const float *vs, int seen) {
    const int tx = threadIdx.x % kLanes<D>, ty = threadIdx.x / kLanes<D>;
    for (int r = 0; r < kRowsPerThread; ++r)
        for (int k = 0; k < min(kKeys, seen + 16 * r); ++k) {
            constexpr int kCols = D / (4 * kLanes<D>);
            const float x = ps[(ty + 16 * r) * Tile<D>::kPStride + k];
            for (int c = 0; c < kCols; ++c) {
                const ulonglong2 vv = *reinterpret_cast<const ulonglong2 *>(vs + k * D + 4 * tx + 4 * kLanes<D> * c);
                fma2(o[(r * kCols + c) * 2], pack2(x, x), vv.x);
                fma2(o[(r * kCols + c) * 2 + 1], pack2(x, x), vv.y);
            }
        }
}

template <int D, bool ALIBI>
__global__ void __launch_bounds__(kThreads<D>, 2) fwd_f32_kernel(const __grid_constant__ F32Params fp) {
    using T = Tile<D>;
    constexpr int kCols = D / (4 * kLanes<D>);  // float4 columns of O per thread and row
    const FwdParams &p = fp.f;
    grid_dependency_wait();
    grid_dependency_launch();
    extern __shared__ __align__(16) float smem[];
    float *qs = smem + T::kQ, *ks = smem + T::kK, *vs = smem + T::kV, *stat = smem + T::kStat;
    float *ps = ks;

    const int tx = threadIdx.x % kLanes<D>, ty = threadIdx.x / kLanes<D>;
    cg::cluster_group cluster = cg::this_cluster();
    const int parts = (int)cluster.num_blocks(), part = (int)cluster.block_rank();
    const int q_blocks = (int)gridDim.x / parts;
    const int r0 = (q_blocks - 1 - (int)blockIdx.x / parts) * kRows;  // long query blocks first
    const int h = blockIdx.y, b = blockIdx.z, kvh = h / p.group;

    const int rows = min(kRows, p.q_len - r0);
    int64_t visible = p.kv_len;  // keys the block's last row sees
    if (p.causal) visible = min(visible, p.causal_off + r0 + rows);
    const int n_tiles = (int)((visible + kKeys - 1) / kKeys);
    const int t_begin = (int)((int64_t)part * n_tiles / parts), t_end = (int)((int64_t)(part + 1) * n_tiles / parts);

    const float *kbase = (const float *)p.k + (int64_t)b * p.kv_bs + (int64_t)kvh * p.kv_hs;
    const float *vbase = (const float *)p.v + (int64_t)b * p.kv_bs + (int64_t)kvh * p.kv_hs;

    const float slope = ALIBI ? p.alibi_slopes[h] : 0.f;
    uint64_t o[kRowsPerThread][2 * kCols];
    float m[kRowsPerThread], l[kRowsPerThread];  // l: this thread's keys only
#pragma unroll
    for (int r = 0; r < kRowsPerThread; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int c = 0; c < 2 * kCols; ++c) o[r][c] = 0;
    }

    if (t_begin < t_end) {
        const float *qbase = (const float *)p.q + (int64_t)b * p.q_bs + (int64_t)h * p.q_hs;
        if (p.rope_q) load_rotated_rows<D>(qs, T::kStride, qbase, p.q_rs, r0, rows, fp.q_table, p.q_rope_off, p.inv_freq);
        else load_rows<D>(qs, T::kStride, qbase, p.q_rs, r0, rows);
    }
    for (int t = t_begin; t < t_end; ++t) {
        const int64_t k0 = (int64_t)t * kKeys;
        const int live = (int)min((int64_t)kKeys, visible - k0);
        // V is asked for first where K takes a detour through registers, and arrives during the score product
        if (!p.rope_k) load_rows<D>(ks, T::kStride, kbase, p.kv_rs, k0, live);
        cp_async_commit();
        load_rows<D>(vs, D, vbase, p.kv_rs, k0, live);
        cp_async_commit();
        if (p.rope_k) load_rotated_rows<D>(ks, T::kStride, kbase, p.kv_rs, k0, live, fp.k_table, p.k_rope_off, p.inv_freq);
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // Q and K
        __syncthreads();

        // S = Q K^T: two half products of D/2 dimensions, each as sums over even and over odd dimensions
        float s[kRowsPerThread][kKeysPerThread<D>];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint64_t acc[kRowsPerThread][kKeysPerThread<D>];
#pragma unroll
            for (int r = 0; r < kRowsPerThread; ++r)
#pragma unroll
                for (int i = 0; i < kKeysPerThread<D>; ++i) acc[r][i] = 0;
            const float *qp = qs + ty * T::kStride + half * (D / 2), *kp = ks + tx * T::kStride + half * (D / 2);
#pragma unroll 2
            for (int d = 0; d < D / 2; d += 4) {
                ulonglong2 qv[kRowsPerThread];
#pragma unroll
                for (int r = 0; r < kRowsPerThread; ++r) qv[r] = *reinterpret_cast<const ulonglong2 *>(qp + 16 * r * T::kStride + d);
#pragma unroll
                for (int i = 0; i < kKeysPerThread<D>; ++i) {
                    const ulonglong2 kv = *reinterpret_cast<const ulonglong2 *>(kp + kLanes<D> * i * T::kStride + d);
#pragma unroll
                    for (int r = 0; r < kRowsPerThread; ++r) {
                        fma2(acc[r][i], qv[r].x, kv.x);
                        fma2(acc[r][i], qv[r].y, kv.y);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < kRowsPerThread; ++r)
#pragma unroll
                for (int i = 0; i < kKeysPerThread<D>; ++i) {
                    const float2 e = unpack2(acc[r][i]);
                    s[r][i] = half ? s[r][i] + (e.x + e.y) : e.x + e.y;
                }
        }
        __syncthreads();  // K has been read: P takes its place

#pragma unroll
        for (int r = 0; r < kRowsPerThread; ++r) {
            const int row = ty + 16 * r;
            int64_t limit = p.kv_len;  // visible keys of this row
            if (p.causal) limit = min(limit, p.causal_off + r0 + row + 1);
            const int lim = (int)min((int64_t)kKeys, limit - k0);
            float mx = -INFINITY;
            // ALiBi: the position difference is formed in integers and rounded to f32 once, like the f64 difference of
            // src/attention_bias.rs:93-94
            const int64_t bias0 = ALIBI ? p.alibi_kv_off - p.alibi_q_off - (r0 + row) + k0 + tx : 0;
#pragma unroll
            for (int i = 0; i < kKeysPerThread<D>; ++i) {
                float sc = s[r][i] * p.scale;
                if constexpr (ALIBI) sc = __fadd_rn(sc, __fmul_rn(slope, (float)(bias0 + kLanes<D> * i)));
                s[r][i] = tx + kLanes<D> * i < lim ? sc : -INFINITY;
                mx = fmaxf(mx, s[r][i]);
            }
#pragma unroll
            for (int w = 1; w < kLanes<D>; w <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const bool any = mx != -INFINITY;  // a row none of whose keys counts in this tile keeps its state
            const float m_new = fmaxf(m[r], mx);
            const float alpha = !any ? 1.f : m[r] == -INFINITY ? 0.f : expf(m[r] - m_new);
            m[r] = m_new;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < kKeysPerThread<D>; ++i) {
                const float e = !any || s[r][i] == -INFINITY ? 0.f : expf(s[r][i] - m_new);
                sum += e;
                ps[row * T::kPStride + tx + kLanes<D> * i] = e;
            }
            l[r] = l[r] * alpha + sum;
            const uint64_t a2 = pack2(alpha, alpha);
#pragma unroll
            for (int c = 0; c < 2 * kCols; ++c) mul2(o[r][c], a2);
        }
        cp_async_wait_all();
        // On the causal diagonal a row does not see all keys of the tile: their probability is 0, which keeps a finite V out
        // of the row and a non-finite one not.  Each thread looks through the V it copied itself, and only a tile that does
        // hold a non-finite value takes the loop that leaves keys out row by row.  Kernel times without / with the search, 8 / 2
        // heads, D = 128: 512 rows 43.6 / 43.9 us, 356 rows 37.9 / 38.7, 2048 rows 393 / 391; D = 64, 300 rows 15.9 / 16.1
        // (that loop in every diagonal tile: 64 rows 16.4 -> 20.5 us; inlined for the rare case, 2048 rows 403).
        const bool diagonal = p.causal && k0 + kKeys > p.causal_off + r0 + 1;
        bool by_row = false;
        if (diagonal) by_row = __syncthreads_or(copied_non_finite<D>(vs));
        else __syncthreads();
        // V is there; a row of P is written and read by the same lanes of one warp
        if (!by_row) {
            // O += P V
#pragma unroll 2
            for (int k = 0; k < kKeys; k += 4) {
                float4 pv[kRowsPerThread];
#pragma unroll
                for (int r = 0; r < kRowsPerThread; ++r)
                    pv[r] = *reinterpret_cast<const float4 *>(ps + (ty + 16 * r) * T::kPStride + k);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    ulonglong2 vv[kCols];
#pragma unroll
                    for (int c = 0; c < kCols; ++c)
                        vv[c] = *reinterpret_cast<const ulonglong2 *>(vs + (k + e) * D + 4 * tx + 4 * kLanes<D> * c);
#pragma unroll
                    for (int r = 0; r < kRowsPerThread; ++r) {
                        const float x = e == 0 ? pv[r].x : e == 1 ? pv[r].y : e == 2 ? pv[r].z : pv[r].w;
                        const uint64_t x2 = pack2(x, x);
#pragma unroll
                        for (int c = 0; c < kCols; ++c) {
                            fma2(o[r][2 * c], x2, vv[c].x);
                            fma2(o[r][2 * c + 1], x2, vv[c].y);
                        }
                    }
                }
            }
        } else {
            uint64_t copy[kRowsPerThread * 2 * kCols];
#pragma unroll
            for (int i = 0; i < kRowsPerThread * 2 * kCols; ++i) copy[i] = o[i / (2 * kCols)][i % (2 * kCols)];
            accumulate_seen<D>(copy, ps, vs, (int)(p.causal_off + r0 + ty + 1 - k0));
#pragma unroll
            for (int i = 0; i < kRowsPerThread * 2 * kCols; ++i) o[i / (2 * kCols)][i % (2 * kCols)] = copy[i];
        }
        __syncthreads();  // the next tile overwrites P and V
    }

#pragma unroll
    for (int r = 0; r < kRowsPerThread; ++r)
#pragma unroll
        for (int w = 1; w < kLanes<D>; w <<= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], w);

    float *obase = (float *)p.o + (int64_t)b * p.o_bs + (int64_t)h * p.o_hs;
    float *lse = p.lse + ((int64_t)b * p.q_heads + h) * p.lse_hs;
    if (parts == 1) {
#pragma unroll
        for (int r = 0; r < kRowsPerThread; ++r) {
            const int row = ty + 16 * r;
            if (row >= rows) continue;
            const float inv = 1.0f / l[r];
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                const float2 a = unpack2(o[r][2 * c]), e = unpack2(o[r][2 * c + 1]);
                *reinterpret_cast<float4 *>(obase + (int64_t)(r0 + row) * p.o_rs + 4 * tx + 4 * kLanes<D> * c) =
                    make_float4(a.x * inv, a.y * inv, e.x * inv, e.y * inv);
            }
            if (tx == 0) lse[r0 + row] = m[r] + logf(l[r]);
        }
        return;
    }

    // ---- combine the cluster's parts: each CTA leaves (max, sum) and its O rows in its own shared memory (over Q and
    // K/P, which are read no more), and finishes its share of the 16-byte vectors, adding the parts in rank order
    float *os = smem;
    if (tx == 0)
#pragma unroll
        for (int r = 0; r < kRowsPerThread; ++r) {
            stat[2 * (ty + 16 * r)] = m[r];
            stat[2 * (ty + 16 * r) + 1] = l[r];
        }
#pragma unroll
    for (int r = 0; r < kRowsPerThread; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c)
            *reinterpret_cast<ulonglong2 *>(os + (ty + 16 * r) * D + 4 * tx + 4 * kLanes<D> * c) = make_ulonglong2(o[r][2 * c], o[r][2 * c + 1]);
    cluster.sync();
    constexpr int kVecs = kRows * (D / 4);
    for (int i = part * kVecs / parts + threadIdx.x; i < (part + 1) * kVecs / parts; i += kThreads<D>) {
        const int row = i / (D / 4), v = i % (D / 4);
        if (row >= rows) continue;
        float mx = -INFINITY;
        for (int x = 0; x < parts; ++x) mx = fmaxf(mx, cluster.map_shared_rank(stat, x)[2 * row]);
        float sum = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int x = 0; x < parts; ++x) {
            const float2 ml = *reinterpret_cast<const float2 *>(cluster.map_shared_rank(stat, x) + 2 * row);
            const float w = ml.x == -INFINITY ? 0.f : expf(ml.x - mx);
            const float4 part_o = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(os, x) + row * D + 4 * v);
            sum = fmaf(w, ml.y, sum);
            acc = make_float4(fmaf(w, part_o.x, acc.x), fmaf(w, part_o.y, acc.y), fmaf(w, part_o.z, acc.z), fmaf(w, part_o.w, acc.w));
        }
        const float inv = 1.0f / sum;
        *reinterpret_cast<float4 *>(obase + (int64_t)(r0 + row) * p.o_rs + 4 * v) =
            make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
        if (v == 0) lse[r0 + row] = mx + logf(sum);
    }
    cluster.sync();  // a CTA's shared memory outlives its readers
}

template <int D>
int launch(flat_ctx *ctx, const F32Params &fp, int parts) {
    const FwdParams &p = fp.f;
    const int smem = Tile<D>::kFloats * (int)sizeof(float);
    auto *kernel = p.alibi_slopes ? fwd_f32_kernel<D, true> : fwd_f32_kernel<D, false>;
    FLAT_CUDA_OK(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((p.q_len + kRows - 1) / kRows * parts), (unsigned)p.q_heads, (unsigned)p.batch);
    cfg.blockDim = dim3(kThreads<D>);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch_dependent()
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)parts;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = may_overlap_previous(ctx) ? 2 : 1;
    FLAT_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, kernel, fp));
    ctx->launches += 1;
    return FLAT_OK;
}

// CTAs per query block.  A CTA costs its tiles and about kOverheadTiles more (its Q rows, its share of the combination); the
// call lasts as long as its longest CTA, and as long as everything takes over the CTAs that run at once (two per SM).
// The cluster size with the smaller of the two maxima is taken.  An overhead of 1 / 2 / 3 tiles, 8 / 2 heads, causal: D = 128,
// 512 rows 48.0 / 42.0 / 42.0 us, 768 77.9 / 77.8 / 78.1, 1024 119.6 / 119.7 / 119.2, 2048 356 / 377 / 379; D = 64, 512 rows
// 28.8 / 24.5 / 24.5, 1024 68.4 / 68.6 / 68.4, 1784 164 / 164 / 172.
constexpr int kOverheadTiles = 2;
int cluster_parts(const flat_ctx *ctx, const FwdParams &p) {
    const int64_t blocks = (p.q_len + kRows - 1) / kRows;
    int64_t tiles = 0, longest = 0;
    for (int64_t i = 0; i < blocks; ++i) {
        int64_t keys = p.kv_len;
        if (p.causal) keys = std::min<int64_t>(keys, p.causal_off + std::min<int64_t>((i + 1) * kRows, p.q_len));
        const int64_t n = (keys + kKeys - 1) / kKeys;
        tiles += n;
        longest = std::max(longest, n);
    }
    tiles *= (int64_t)p.q_heads * p.batch;
    const int64_t slots = 2 * (int64_t)ctx->sm_count, all = blocks * p.q_heads * p.batch;
    int parts = 1;
    int64_t best = INT64_MAX;
    for (int c = 1; c <= kMaxCluster && c <= longest; ++c) {
        const int64_t cost = std::max(slots * (kOverheadTiles + (longest + c - 1) / c), tiles + kOverheadTiles * all * c);
        if (cost < best) best = cost, parts = c;
    }
    return parts;
}

bool holds(const flat_ctx::RopeTable &t, const FwdParams &p, int64_t first, int64_t rows) {
    return t.dev && !t.replays_write && t.half_dim == p.head_dim / 2 && t.pos_off <= first && first + rows <= t.pos_off + t.rows &&
           std::memcmp(t.inv_freq, p.inv_freq, p.head_dim / 2 * sizeof(float)) == 0;
}

// The (cos, sin) tables of a call.  Those of the tensor-core kernels are read where they hold the positions, and never
// written; else the context's table of this mode is made to hold one range with the positions of Q and of K, unless it does.
// Without a table the kernel evaluates the same angles itself, for every tile again (512 rows 47 us instead of 42): under
// stream capture, where a replay would read what later calls have put there, beyond kF32TableBytes, and where the context
// got no memory.
void find_tables(flat_ctx *ctx, F32Params *fp) {
    const FwdParams &p = fp->f;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusActive;
    if (cudaStreamIsCapturing(ctx->stream, &capture) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (capture != cudaStreamCaptureStatusNone) return;
    const int half_dim = p.head_dim / 2;
    auto at = [&](const flat_ctx::RopeTable &t, int64_t pos) {
        return static_cast<const float2 *>(t.dev) + (pos - t.pos_off) * half_dim;
    };
    for (const auto &t : ctx->rope_tables) {
        if (p.rope_q && holds(t, p, p.q_rope_off, p.q_len)) fp->q_table = at(t, p.q_rope_off);
        if (p.rope_k && holds(t, p, p.k_rope_off, p.kv_len)) fp->k_table = at(t, p.k_rope_off);
    }
    const bool want_q = p.rope_q && !fp->q_table, want_k = p.rope_k && !fp->k_table;
    if (!want_q && !want_k) return;
    int64_t lo = INT64_MAX, hi = 0;
    if (want_q) lo = p.q_rope_off, hi = lo + p.q_len;
    if (want_k) lo = std::min(lo, p.k_rope_off), hi = std::max(hi, p.k_rope_off + p.kv_len);
    flat_ctx::RopeTable &t = ctx->f32_table;
    if (!holds(t, p, lo, hi - lo)) {
        if (!t.dev || (uint64_t)(hi - lo) * half_dim * sizeof(float2) > t.bytes) return;
        t.rows = 0;
        if (fill_rope_table(ctx, t.dev, p.inv_freq, half_dim, (int)(hi - lo), lo)) return;
        std::memcpy(t.inv_freq, p.inv_freq, half_dim * sizeof(float));
        t.half_dim = half_dim;
        t.pos_off = lo;
        t.rows = (int)(hi - lo);
    }
    if (want_q) fp->q_table = at(t, p.q_rope_off);
    if (want_k) fp->k_table = at(t, p.k_rope_off);
}

}  // namespace

bool forward_f32_supported(const FwdParams &p) {
    if (p.head_dim != 64 && p.head_dim != 128) return false;
    if (p.varlen || p.page_table) return false;
    // a block has 64 rows, most of them idle in a short call; from 16 rows on it is still the faster one (8 / 2 heads: 16 rows
    // against 16 keys, D = 64 12.3 -> 10.3 us, against 2000 keys 514 -> 33 us)
    if (p.q_len < 16) return false;
    const void *ptrs[] = {p.q, p.k, p.v, p.o};
    for (const void *x : ptrs)
        if (reinterpret_cast<uintptr_t>(x) & 15) return false;
    const int64_t strides[] = {p.q_bs, p.q_hs, p.q_rs, p.kv_bs, p.kv_hs, p.kv_rs, p.o_bs, p.o_hs, p.o_rs};
    for (int64_t s : strides)
        if (s % 4 != 0) return false;
    return true;
}

void forward_f32_geometry(const flat_ctx *ctx, const FwdParams &p, uint32_t *query_rows, uint32_t *kv_rows, uint32_t grid[3]) {
    *query_rows = kRows;
    *kv_rows = kKeys;
    grid[0] = (uint32_t)((p.q_len + kRows - 1) / kRows * cluster_parts(ctx, p));
    grid[1] = (uint32_t)p.q_heads;
    grid[2] = (uint32_t)p.batch;
}

int launch_forward_f32(flat_ctx *ctx, const FwdParams &p) {
    if (p.q_heads > 65535 || p.batch > 65535)
        return fail(ctx, FLAT_ERR_DISPATCH_LIMIT, "grid dimension %d exceeds 65535", p.q_heads > 65535 ? p.q_heads : p.batch);
    F32Params fp{};
    fp.f = p;
    if (p.rope_q || p.rope_k) find_tables(ctx, &fp);
    const int parts = cluster_parts(ctx, p);
    return p.head_dim == 128 ? launch<128>(ctx, fp, parts) : launch<64>(ctx, fp, parts);
}

}  // namespace flat
