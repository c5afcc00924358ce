// Edge softmax over the incoming edges of every destination, forward and gradient, in two flavours.
//
// fused GAT attention:
//   forward : a[e,h]  = softmax over the incoming edges of dst(e) of leaky_relu(el_q[src(e),h]*sl + er_q[dst(e),h]*sr)
//   backward: dz[e,h] = a * (da - sum_row a*da) * (z > 0 ? 1 : slope)   (PyTorch's LeakyReLU gradient convention at 0)
// plain scores (zin given):
//   forward : a[e,h]  = softmax over the incoming edges of dst(e) of zin[e,h] * zmul
//   backward: dz[e,h] = a * (da - sum_row a*da) * zmul
//
// two-step forward without an fp32 copy of the attention weights (stats / quantized):
//   stats     : per (row, head) the softmax statistics m = max z and inv = 1 / sum exp(z - m); the largest weight of a
//               row is exp(0) * inv = inv, so max over rows of inv is max|a| and fixes the int8 scale of a up front
//   quantized : a_q[e,h] = round(exp(z - m) * inv / scale) -- the int8 weights the aggregation consumes, written once
//   backward  : the same gradient as above with a recomputed from (z, m, inv) instead of being read
//
// A destination row is owned by a thread team: a whole CTA for the rows at the head of the degree-sorted order (a
// power-law graph has rows with 10^5 incoming edges; one warp would serialise them), a warp for the rest.  All heads
// of an edge are handled together (one 128-bit access per edge when H == 4).  The softmax statistics are
// accumulated "online" (running maximum with rescaling), so the forward needs two sweeps over a row.
//
// Every sum over a row runs in ONE order that depends on the row's length alone: up to 1024 slots (rows behind
// n_block_rows), lane l of 32 takes slots l, l + 32, ... one after the other and the lanes meet in a butterfly (16, 8, 4, 2,
// 1); longer rows have 256 lanes, a butterfly per 32 of them, then the eight results in turn.  Narrower teams (short rows,
// below) keep the lanes they stand in for apart and follow the same tree.  The weights are quantized to int8 behind this
// kernel, and one ulp in the largest of them can move every code: a layer must not change with the graph around a row or
// with the launch shape.
#include "common.cuh"

namespace tango {

constexpr int kMaxHeads = 8;

struct GatArgs {
    const int32_t *indptr, *indices, *edge_ids, *row_order;
    int64_t n_rows, n_block_rows;
    const int8_t *elq, *erq;
    int H;
    const float *sl, *sr;
    float slope;
    float *att;          // forward: output; backward: input
    const float *datt;   // backward
    float *dz;           // backward
    const float *zin;    // plain-score flavour: fp32 scores [E, H] in edge-id order (elq / erq / sl / sr unused)
    float zmul;          // factor applied to zin before the softmax
    float *out_absmax;   // optional: receives max|output| / 127 (forward: of a, backward: of dz); must hold 0
    // two-step forward / recomputing backward
    float *row_m, *row_inv;        // [n_rows, H] softmax statistics (written by STATS, read by QUANT and by BWD)
    int8_t *att_q;                 // QUANT: int8 output [E, H] in edge-id order
    const float *att_scale;        // QUANT: scale of a (device, 1 element)
    int round_mode;
    uint64_t seed, call;
    const unsigned long long *step;
};

enum { FWD_FLOAT = 0, FWD_STATS = 1, FWD_QUANT = 2 };

__device__ __forceinline__ float leaky(float z, float slope) { return z >= 0.f ? z : __fmul_rn(z, slope); }

// Heads handled together (HT = 0: any number up to kMaxHeads, element by element) and edges in flight per thread.
template <int HT> struct Shape {
    static constexpr int N = HT ? HT : kMaxHeads;
    static constexpr int U = HT == 1 ? 8 : HT == 2 || HT == 4 ? 4 : 2;
    static constexpr int kKept = HT == 8 ? 512 : 1024;      // gathered records a warp keeps between its two sweeps
};
template <int HT> struct Record { typedef uint8_t T; };
template <> struct Record<2> { typedef uint16_t T; };
template <> struct Record<4> { typedef uint32_t T; };
template <> struct Record<8> { typedef uint2 T; };

// The H floats of an edge, H <= N; the base of the array is aligned to the access.
template <int HT>
__device__ __forceinline__ void load_heads(const float *p, int H, float (&v)[Shape<HT>::N]) {
    constexpr int N = Shape<HT>::N;
    if (HT == 8 || HT == 4) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) {
            const float4 t = __ldg(reinterpret_cast<const float4 *>(p) + i);
            v[4 * i] = t.x; v[(4 * i + 1) % N] = t.y; v[(4 * i + 2) % N] = t.z; v[(4 * i + 3) % N] = t.w;
        }
    } else if (HT == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
        v[0] = t.x; v[1 % N] = t.y;
    } else {
#pragma unroll
        for (int h = 0; h < N; ++h) v[h] = h < H ? __ldg(p + h) : 0.f;
    }
}
template <int HT>
__device__ __forceinline__ void store_heads(float *p, int H, const float (&v)[Shape<HT>::N]) {
    constexpr int N = Shape<HT>::N;
    if (HT == 8 || HT == 4) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i)
            reinterpret_cast<float4 *>(p)[i] = make_float4(v[4 * i], v[(4 * i + 1) % N], v[(4 * i + 2) % N], v[(4 * i + 3) % N]);
    } else if (HT == 2) {
        *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1 % N]);
    } else {
#pragma unroll
        for (int h = 0; h < N; ++h)
            if (h < H) p[h] = v[h];
    }
}
// The int8 features of a node, all heads in one record; HT = 0 head by head.
template <int HT>
__device__ __forceinline__ void decode(const typename Record<HT>::T &r, float (&v)[Shape<HT>::N]) {
    constexpr int N = Shape<HT>::N;
    uint32_t w[2] = {0, 0};
    if constexpr (HT == 8) { w[0] = r.x; w[1] = r.y; }
    else w[0] = r;
#pragma unroll
    for (int h = 0; h < N; ++h) v[h] = (float)(int8_t)(w[h >> 2] >> (8 * (h & 3)));
}

// The edges of one trip of a team over a row: thread `tid` takes slots j0 + u * NT.  Their logits for all heads; slots beyond
// the row get -infinity, which adds nothing to a softmax.  `kept`: records of the row's first `cap` slots in shared memory,
// written (SAVE) or read instead of gathered (every thread meets its own slots again).
enum { GATHER = 0, SAVE = 1, REUSE = 2 };
template <int NT, int HT, int U, bool PLAIN, int KEEP = GATHER>
__device__ __forceinline__ void trip_logits(const GatArgs &a, int j0, int beg, int end, const float (&er)[Shape<HT>::N], float sl,
                                            float (&z)[U][Shape<HT>::N], typename Record<HT>::T *kept = nullptr, int cap = 0) {
    constexpr int N = Shape<HT>::N;
    typedef typename Record<HT>::T R;
    const int H = HT ? HT : a.H;
    int at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int j = j0 + u * NT;
        at[u] = j >= end ? -1
              : PLAIN ? (a.edge_ids ? __ldg(a.edge_ids + j) : j)
              : KEEP == REUSE && j - beg < cap ? 0 : __ldg(a.indices + j);
    }
    R rec[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int h = 0; h < N; ++h) z[u][h] = -INFINITY;
        rec[u] = R();
        if (at[u] < 0) continue;
        if constexpr (PLAIN) {
            load_heads<HT>(a.zin + (int64_t)at[u] * H, H, z[u]);
        } else if constexpr (HT == 0) {
            for (int h = 0; h < N; ++h) z[u][h] = h < H ? (float)__ldg(a.elq + (int64_t)at[u] * H + h) : 0.f;
        } else {
            const int slot = j0 + u * NT - beg;
            if (KEEP == REUSE && slot < cap) rec[u] = kept[slot];
            else rec[u] = __ldg(reinterpret_cast<const R *>(a.elq) + at[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (at[u] < 0) continue;
        if constexpr (PLAIN) {
#pragma unroll
            for (int h = 0; h < N; ++h) z[u][h] = __fmul_rn(z[u][h], a.zmul);
        } else {
            if constexpr (HT != 0) {
                const int slot = j0 + u * NT - beg;
                if (KEEP == SAVE && slot < cap) kept[slot] = rec[u];
                decode<HT>(rec[u], z[u]);
            }
#pragma unroll
            for (int h = 0; h < N; ++h) z[u][h] = leaky(__fadd_rn(__fmul_rn(z[u][h], sl), er[h]), a.slope);
        }
    }
}

// Fixed-order reductions over a team of NT threads (up to 32: aligned lanes of a warp; else the whole CTA through shared memory).
template <int NT>
__device__ __forceinline__ float team_sum(float v, float *smem) {
#pragma unroll
    for (int o = NT < 32 ? NT / 2 : 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (NT <= 32) return v;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    float t = 0.f;
    for (int w = 0; w < NT / 32; ++w) t += smem[w];
    return t;
}

// Takes in the logits z[0..U) one after the other: s = s * exp(m - z) + 1 at a new maximum z, else s + exp(z - m); -infinity
// adds nothing, NaN stays in the sum.  The maxima come first, so that only a product and a sum per logit are a chain.
template <int U>
__device__ __forceinline__ void online_softmax(const float (&z)[U], float &m, float &s) {
    float keep[U], e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const bool up = z[u] > m;
        const float d = __expf(-fabsf(z[u] - fmaxf(m, -3.402823466e+38f)));     // (a finite base: -infinity twice is no NaN)
        keep[u] = up ? d : 1.f;
        e[u] = up ? 1.f : d;
        m = up ? z[u] : m;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) s = __fadd_rn(__fmul_rn(s, keep[u]), e[u]);
}

// (m, s) of two disjoint sets of logits; symmetric in them
__device__ __forceinline__ void merge_softmax(float &m, float &s, float m2, float s2) {
    const float mm = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * __expf(m - mm)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mm));
    m = mm;
}

// merges online-softmax states (m, s): fixed butterfly inside a warp, then warp 0..n in order
template <int NT>
__device__ __forceinline__ void team_softmax_merge(float &m, float &s, float *smem) {
#pragma unroll
    for (int o = NT < 32 ? NT / 2 : 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
        merge_softmax(m, s, m2, s2);
    }
    if (NT <= 32) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) { smem[warp] = m; smem[32 + warp] = s; }
    __syncthreads();
    float mm = -INFINITY, ss = 0.f;
    for (int w = 0; w < NT / 32; ++w) merge_softmax(mm, ss, smem[w], smem[32 + w]);
    m = mm; s = ss;
}

// Slots [beg, end) of row `row` by a team of NT threads.  `kept`: cap records of shared memory (FWD_FLOAT).
template <int NT, int HT, int U, bool PLAIN, int STAGE>
__device__ __forceinline__ void softmax_row(const GatArgs &a, int64_t row, int beg, int end, int tid, float *smem,
                                            typename Record<HT>::T *kept, int cap, float &amax) {
    constexpr int N = Shape<HT>::N, K = U < 4 ? U : 4;
    static_assert(NT == 8 || NT >= 32, "eight lanes stand in for 32");
    constexpr bool kKeep = STAGE == FWD_FLOAT && !PLAIN && HT != 0 && NT >= 32;
    const float sl = PLAIN ? 0.f : __ldg(a.sl), sr = PLAIN ? 0.f : __ldg(a.sr);
    const int H = HT ? HT : a.H;
    const int trips = (end - beg + NT * U - 1) / (NT * U);
    float er[N], m[N], s[N], inv[N], z[U][N];
#pragma unroll
    for (int h = 0; h < N; ++h) {
        er[h] = (h < H && !PLAIN) ? __fmul_rn((float)__ldg(a.erq + row * H + h), sr) : 0.f;
        m[h] = -INFINITY; s[h] = 0.f;
    }
    if (STAGE == FWD_QUANT) {
        // second step: statistics from the first step, int8 weights out
#pragma unroll
        for (int h = 0; h < N; ++h) {
            m[h] = h < H ? __ldg(a.row_m + row * H + h) : 0.f;
            inv[h] = h < H ? __ldg(a.row_inv + row * H + h) : 0.f;
        }
        const float inv_s = inv_scale(__ldg(a.att_scale));
        const uint64_t call = effective_call(a.call, a.step);
        const Philox ph{(uint32_t)a.seed, (uint32_t)(a.seed >> 32)};
        for (int t = 0; t < trips; ++t) {
            const int j0 = beg + tid + t * NT * U;
            trip_logits<NT, HT, U, PLAIN>(a, j0, beg, end, er, sl, z);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + u * NT;
                if (j >= end) break;
                const int64_t eid = a.edge_ids ? __ldg(a.edge_ids + j) : j;
                uint32_t packed[2] = {0, 0};
                uint64_t cached_blk = ~0ull;
                uint4 rnd = make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int h = 0; h < N; ++h) {
                    if (h < H) {
                        const float v = __fmul_rn(__expf(z[u][h] - m[h]) * inv[h], inv_s);
                        float r = 0.f;
                        if (a.round_mode == TANGO_ROUND_STOCHASTIC)
                            r = sr_uniform(ph, (uint64_t)eid * (uint64_t)H + (uint64_t)h, call, cached_blk, rnd);
                        const int qi = round_to_i8(v, a.round_mode, r);
                        if (HT >= 2) packed[h >> 2] |= ((uint32_t)qi & 0xffu) << (8 * (h & 3));
                        else a.att_q[eid * H + h] = (int8_t)qi;
                    }
                }
                if (HT == 8) *reinterpret_cast<uint2 *>(a.att_q + eid * 8) = make_uint2(packed[0], packed[1]);
                if (HT == 4) *reinterpret_cast<uint32_t *>(a.att_q + eid * 4) = packed[0];
                if (HT == 2) *reinterpret_cast<uint16_t *>(a.att_q + eid * 2) = (uint16_t)packed[0];
            }
        }
        return;
    }
    for (int t = 0; t < trips; ++t) {
        trip_logits<NT, HT, U, PLAIN, kKeep ? SAVE : GATHER>(a, beg + tid + t * NT * U, beg, end, er, sl, z, kept, cap);
#pragma unroll
        for (int h = 0; h < N; ++h) {
            if (h >= H) continue;
            if (NT >= 32) {
                float zh[U];
#pragma unroll
                for (int u = 0; u < U; ++u) zh[u] = z[u][h];
                online_softmax<U>(zh, m[h], s[h]);
            } else {
                // the only trip: logit u belongs to lane tid + 8 * (u % 4) of 32
                float mk[K], sk[K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    float zk[U / K];
#pragma unroll
                    for (int i = 0; i < U / K; ++i) zk[i] = z[i * K + k][h];
                    mk[k] = -INFINITY; sk[k] = 0.f;
                    online_softmax<U / K>(zk, mk[k], sk[k]);
                }
#pragma unroll
                for (int o = K / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int k = 0; k < o; ++k) merge_softmax(mk[k], sk[k], mk[(k + o) % K], sk[(k + o) % K]);
                m[h] = mk[0]; s[h] = sk[0];
            }
        }
    }
#pragma unroll
    for (int h = 0; h < N; ++h)
        if (h < H) team_softmax_merge<NT>(m[h], s[h], smem);
#pragma unroll
    for (int h = 0; h < N; ++h) inv[h] = h < H ? 1.f / s[h] : 0.f;
    if (STAGE == FWD_STATS) {
        // first step: keep (m, inv); the row's largest weight is exp(0) * inv = inv
        if (tid == 0 && end > beg) {
#pragma unroll
            for (int h = 0; h < N; ++h) {
                if (h < H) {
                    a.row_m[row * H + h] = m[h];
                    a.row_inv[row * H + h] = inv[h];
                    amax = fmaxf(amax, inv[h]);
                }
            }
        }
        return;
    }
    for (int t = trips - 1; t >= 0; --t) {          // the last trip's logits are still in registers
        const int j0 = beg + tid + t * NT * U;
        if (t != trips - 1) trip_logits<NT, HT, U, PLAIN, kKeep ? REUSE : GATHER>(a, j0, beg, end, er, sl, z, kept, cap);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + u * NT;
            if (j >= end) break;
            const int64_t eid = a.edge_ids ? __ldg(a.edge_ids + j) : j;
            float o[N];
#pragma unroll
            for (int h = 0; h < N; ++h) {
                o[h] = h < H ? __expf(z[u][h] - m[h]) * inv[h] : 0.f;
                amax = fmaxf(amax, o[h]);
            }
            store_heads<HT>(a.att + eid * H, H, o);
        }
    }
}

// RECOMPUTE: the attention weights are not read but recomputed as exp(z - m) * inv from the forward's statistics.
template <int NT, int HT, int U, bool PLAIN, bool RECOMPUTE>
__device__ __forceinline__ void softmax_bwd_row(const GatArgs &a, int64_t row, int beg, int end, int tid, float *smem,
                                                float &amax) {
    constexpr int N = Shape<HT>::N, K = U < 4 ? U : 4;
    const float sl = PLAIN ? 0.f : __ldg(a.sl), sr = PLAIN ? 0.f : __ldg(a.sr);
    const int H = HT ? HT : a.H;
    const int trips = (end - beg + NT * U - 1) / (NT * U);
    float er[N], dot[N], m[N], inv[N], z[U][N], p[U][N], g[U][N];
#pragma unroll
    for (int h = 0; h < N; ++h) {
        er[h] = (h < H && !PLAIN) ? __fmul_rn((float)__ldg(a.erq + row * H + h), sr) : 0.f;
        dot[h] = 0.f;
        m[h] = (RECOMPUTE && h < H) ? __ldg(a.row_m + row * H + h) : 0.f;
        inv[h] = (RECOMPUTE && h < H) ? __ldg(a.row_inv + row * H + h) : 0.f;
    }
    int eid[U];
    const auto load = [&](int t, bool logits) {
        const int j0 = beg + tid + t * NT * U;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + u * NT;
            eid[u] = j < end ? (a.edge_ids ? __ldg(a.edge_ids + j) : j) : -1;
        }
        if (!PLAIN && (RECOMPUTE || logits)) trip_logits<NT, HT, U, PLAIN>(a, j0, beg, end, er, sl, z);
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int h = 0; h < N; ++h) p[u][h] = g[u][h] = 0.f;
            if (eid[u] >= 0) {
                if (!RECOMPUTE) load_heads<HT>(a.att + (int64_t)eid[u] * H, H, p[u]);
                load_heads<HT>(a.datt + (int64_t)eid[u] * H, H, g[u]);
            }
        }
        if (RECOMPUTE) {
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int h = 0; h < N; ++h) p[u][h] = eid[u] >= 0 ? __expf(z[u][h] - m[h]) * inv[h] : 0.f;
        }
    };
    for (int t = 0; t < trips; ++t) {
        load(t, t == trips - 1);
#pragma unroll
        for (int h = 0; h < N; ++h) {
            if (h >= H) continue;
            if (NT >= 32) {
#pragma unroll
                for (int u = 0; u < U; ++u) dot[h] += p[u][h] * g[u][h];
            } else {                               // the only trip, as in the forward
                float d[K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    d[k] = p[k][h] * g[k][h];
#pragma unroll
                    for (int u = k + K; u < U; u += K) d[k] += p[u][h] * g[u][h];
                }
#pragma unroll
                for (int o = K / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int k = 0; k < o; ++k) d[k] += d[(k + o) % K];
                dot[h] = d[0];
            }
        }
    }
#pragma unroll
    for (int h = 0; h < N; ++h)
        if (h < H) dot[h] = team_sum<NT>(dot[h], smem);
    for (int t = trips - 1; t >= 0; --t) {          // the last trip is still in registers
        if (t != trips - 1) load(t, true);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (eid[u] < 0) break;
            float o[N];
#pragma unroll
            for (int h = 0; h < N; ++h) {
                o[h] = p[u][h] * (g[u][h] - dot[h]);
                if (PLAIN) o[h] *= a.zmul;
                else if (!(z[u][h] > 0.f)) o[h] *= a.slope;      // leaky(z) has the sign of z
                if (h < H) amax = fmaxf(amax, fabsf(o[h]));
            }
            store_heads<HT>(a.dz + (int64_t)eid[u] * H, H, o);
        }
    }
}

template <int NT, int HT, int U, bool PLAIN, bool BWD, int STAGE>
__device__ __forceinline__ void one_row(const GatArgs &a, int64_t row, int beg, int end, int tid, float *smem,
                                        typename Record<HT>::T *kept, int cap, float &amax) {
    if (BWD) softmax_bwd_row<NT, HT, U, PLAIN, STAGE != 0>(a, row, beg, end, tid, smem, amax);
    else softmax_row<NT, HT, U, PLAIN, STAGE>(a, row, beg, end, tid, smem, kept, cap, amax);
}

// CTAs [0, n_block_rows): one row each.  In the CTAs behind them a warp takes four rows in a row of the order: side by side
// with eight lanes each when the longest of them fits one trip of eight lanes, else one after the other with the whole warp.
// BWD: gradient kernel; STAGE: forward flavour (FWD_*) or, for BWD, 1 = recompute the weights from the statistics
//
// What bounds it: on long rows the [E, H] streams (forward 4 B in and 4 * H out per edge, backward 8 * H in and 4 * H out,
// less what the second sweep finds in L2) and, in the forward, a warp's load of 32 random int8 records, which takes 32 passes
// through L1: the records are kept in shared memory between the sweeps.  On short rows it is rows in flight: half the rows
// of a sparse power-law graph have one edge, and had a warp each.  One edge in flight per thread -> as it is, us:
//   114.6 M edges, 4 heads: forward 1224 -> 1195, backward 1577 -> 1386;  1 head: 593 -> 427, 668 -> 565
//   1.3 M edges on 169 K nodes, 4 heads, plain scores: 153 -> 50, 55 -> 39;  0.1 M edges, 8 heads: 53 -> 50, 40 -> 40 (a CTA
//   for rows of 128 edges and more took 28 and 13 there, but their terms were then added in another order)
template <int HT, bool PLAIN, bool BWD, int STAGE>
__global__ void __launch_bounds__(256, HT == 1 || HT == 2 ? (BWD ? 4 : 6) : (HT == 4 ? 4 : 3) - (BWD ? 1 : 0)) gat_softmax_kernel(const GatArgs a) {
    constexpr int U = Shape<HT>::U;
    constexpr bool kKeep = !BWD && STAGE == FWD_FLOAT && !PLAIN && HT != 0;
    constexpr int kCap = kKeep ? Shape<HT>::kKept : 0;
    typedef typename Record<HT>::T R;
    __shared__ float smem[64];
    __shared__ R s_kept[kKeep ? 8 * kCap : 1];
    float amax = 0.f;
    if ((int64_t)blockIdx.x < a.n_block_rows) {
        const int64_t row = a.row_order ? (int64_t)__ldg(a.row_order + blockIdx.x) : (int64_t)blockIdx.x;
        const int beg = __ldg(a.indptr + row), end = __ldg(a.indptr + row + 1);
        one_row<256, HT, U, PLAIN, BWD, STAGE>(a, row, beg, end, threadIdx.x, smem, s_kept, 8 * kCap, amax);
    } else {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int64_t i = a.n_block_rows + (((int64_t)blockIdx.x - a.n_block_rows) * 8 + warp) * 4 + (lane & 3);
        int row = -1, beg = 0, end = 0;
        if (i < a.n_rows) {
            row = a.row_order ? __ldg(a.row_order + i) : (int)i;
            beg = __ldg(a.indptr + row); end = __ldg(a.indptr + row + 1);
        }
        int longest = max(end - beg, __shfl_xor_sync(0xffffffffu, end - beg, 1));
        longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, 2));
        if (longest <= 8 * U) {
            const int team = lane >> 3;
            row = max(0, __shfl_sync(0xffffffffu, row, team));       // (a missing row has no slots)
            beg = __shfl_sync(0xffffffffu, beg, team);
            end = __shfl_sync(0xffffffffu, end, team);
            if (longest <= 8) one_row<8, HT, 1, PLAIN, BWD, STAGE>(a, row, beg, end, lane & 7, smem, nullptr, 0, amax);
            else one_row<8, HT, U, PLAIN, BWD, STAGE>(a, row, beg, end, lane & 7, smem, nullptr, 0, amax);
        } else {
            for (int r = 0; r < 4; ++r) {
                const int rr = __shfl_sync(0xffffffffu, row, r);
                if (rr < 0) break;
                one_row<32, HT, U, PLAIN, BWD, STAGE>(a, rr, __shfl_sync(0xffffffffu, beg, r), __shfl_sync(0xffffffffu, end, r),
                                                      lane, smem, s_kept + (kKeep ? warp * kCap : 0), kCap, amax);
            }
        }
    }
    if (a.out_absmax) {
        amax = warp_max(amax);
        if ((threadIdx.x & 31) == 0 && amax > 0.f) {
            const float s = __fdiv_rn(amax, 127.0f);
            if (s > __ldcg(a.out_absmax)) atomic_max_nonneg(a.out_absmax, s);
        }
    }
}

template <int HT, bool BWD, int STAGE>
static void launch_heads(const GatArgs &a, unsigned blocks, cudaStream_t stream) {
    if (STAGE == 0 && a.zin) gat_softmax_kernel<HT, true, BWD, 0><<<blocks, 256, 0, stream>>>(a);
    else gat_softmax_kernel<HT, false, BWD, STAGE><<<blocks, 256, 0, stream>>>(a);
}

template <bool BWD, int STAGE = 0>
static int launch_gat(GatArgs &a, cudaStream_t stream) {
    if (a.n_rows < 0 || a.H < 1 || a.H > kMaxHeads) return TANGO_EINVAL;
    if (a.n_rows == 0) return TANGO_OK;
    if (!a.row_order) a.n_block_rows = 0;
    if (a.n_block_rows < 0 || a.n_block_rows > a.n_rows) return TANGO_EINVAL;
    const int64_t blocks = a.n_block_rows + ceil_div(a.n_rows - a.n_block_rows, 8 * 4);
    if (blocks > 0x7fffffff || a.n_rows > 0x7fffffff) return TANGO_ESIZE;
    // all heads of an edge in one access where every array allows it
    const int f = 4 * (a.H < 4 ? a.H : 4);
    const bool whole = (a.H == 1 || a.H == 2 || a.H == 4 || a.H == 8) && aligned(a.att, f) && aligned(a.zin, f) &&
                       aligned(a.datt, f) && aligned(a.dz, f) && aligned(a.elq, a.H) && aligned(a.att_q, a.H);
    const unsigned nb = (unsigned)blocks;
    if (whole && a.H == 1) launch_heads<1, BWD, STAGE>(a, nb, stream);
    else if (whole && a.H == 2) launch_heads<2, BWD, STAGE>(a, nb, stream);
    else if (whole && a.H == 4) launch_heads<4, BWD, STAGE>(a, nb, stream);
    else if (whole && a.H == 8) launch_heads<8, BWD, STAGE>(a, nb, stream);
    else launch_heads<0, BWD, STAGE>(a, nb, stream);
    TANGO_LAUNCH_CHECK();
    return TANGO_OK;
}

}  // namespace tango

using namespace tango;

extern "C" int tango_gat_edge_softmax(const int32_t *indptr, const int32_t *indices, const int32_t *edge_ids,
                                      const int32_t *row_order, int64_t n_block_rows, int64_t n_rows,
                                      const int8_t *elq, const int8_t *erq, int h, const float *sl, const float *sr,
                                      float slope, float *a, float *a_absmax, tango_stream_t stream) {
    if (n_rows > 0 && (!indptr || !indices || !elq || !erq || !sl || !sr || !a)) return TANGO_EINVAL;
    GatArgs g{indptr, indices, edge_ids, row_order, n_rows, n_block_rows, elq, erq, h, sl, sr, slope, a, nullptr, nullptr,
              nullptr, 1.f, a_absmax};
    return launch_gat<false>(g, (cudaStream_t)stream);
}

extern "C" int tango_gat_edge_softmax_bwd(const int32_t *indptr, const int32_t *indices, const int32_t *edge_ids,
                                          const int32_t *row_order, int64_t n_block_rows, int64_t n_rows,
                                          const int8_t *elq, const int8_t *erq, int h, const float *sl,
                                          const float *sr, float slope, const float *a, const float *da, float *dz,
                                          float *dz_absmax, tango_stream_t stream) {
    if (n_rows > 0 && (!indptr || !indices || !elq || !erq || !sl || !sr || !a || !da || !dz)) return TANGO_EINVAL;
    GatArgs g{indptr, indices, edge_ids, row_order, n_rows, n_block_rows, elq, erq, h, sl, sr, slope,
              const_cast<float *>(a), da, dz, nullptr, 1.f, dz_absmax};
    return launch_gat<true>(g, (cudaStream_t)stream);
}

extern "C" int tango_gat_edge_softmax_stats(const int32_t *indptr, const int32_t *indices, const int32_t *row_order,
                                            int64_t n_block_rows, int64_t n_rows, const int8_t *elq, const int8_t *erq,
                                            int h, const float *sl, const float *sr, float slope, float *row_m,
                                            float *row_inv, float *a_absmax, tango_stream_t stream) {
    if (n_rows > 0 && (!indptr || !indices || !elq || !erq || !sl || !sr || !row_m || !row_inv)) return TANGO_EINVAL;
    GatArgs g{};
    g.indptr = indptr; g.indices = indices; g.row_order = row_order; g.n_rows = n_rows; g.n_block_rows = n_block_rows;
    g.elq = elq; g.erq = erq; g.H = h; g.sl = sl; g.sr = sr; g.slope = slope; g.zmul = 1.f;
    g.row_m = row_m; g.row_inv = row_inv; g.out_absmax = a_absmax;
    return launch_gat<false, FWD_STATS>(g, (cudaStream_t)stream);
}

extern "C" int tango_gat_edge_softmax_quantized(const int32_t *indptr, const int32_t *indices, const int32_t *edge_ids,
                                                const int32_t *row_order, int64_t n_block_rows, int64_t n_rows,
                                                const int8_t *elq, const int8_t *erq, int h, const float *sl,
                                                const float *sr, float slope, const float *row_m, const float *row_inv,
                                                const float *a_scale, int8_t *aq, int mode, uint64_t seed,
                                                uint64_t call, const uint64_t *step, tango_stream_t stream) {
    if (mode < 0 || mode > 2) return TANGO_EINVAL;
    if (n_rows > 0 && (!indptr || !indices || !elq || !erq || !sl || !sr || !row_m || !row_inv || !a_scale || !aq))
        return TANGO_EINVAL;
    GatArgs g{};
    g.indptr = indptr; g.indices = indices; g.edge_ids = edge_ids; g.row_order = row_order; g.n_rows = n_rows;
    g.n_block_rows = n_block_rows; g.elq = elq; g.erq = erq; g.H = h; g.sl = sl; g.sr = sr; g.slope = slope; g.zmul = 1.f;
    g.row_m = const_cast<float *>(row_m); g.row_inv = const_cast<float *>(row_inv); g.att_q = aq; g.att_scale = a_scale;
    g.round_mode = mode; g.seed = seed; g.call = call; g.step = reinterpret_cast<const unsigned long long *>(step);
    return launch_gat<false, FWD_QUANT>(g, (cudaStream_t)stream);
}

extern "C" int tango_gat_edge_softmax_bwd_stats(const int32_t *indptr, const int32_t *indices, const int32_t *edge_ids,
                                                const int32_t *row_order, int64_t n_block_rows, int64_t n_rows,
                                                const int8_t *elq, const int8_t *erq, int h, const float *sl,
                                                const float *sr, float slope, const float *row_m, const float *row_inv,
                                                const float *da, float *dz, float *dz_absmax, tango_stream_t stream) {
    if (n_rows > 0 && (!indptr || !indices || !elq || !erq || !sl || !sr || !row_m || !row_inv || !da || !dz))
        return TANGO_EINVAL;
    GatArgs g{};
    g.indptr = indptr; g.indices = indices; g.edge_ids = edge_ids; g.row_order = row_order; g.n_rows = n_rows;
    g.n_block_rows = n_block_rows; g.elq = elq; g.erq = erq; g.H = h; g.sl = sl; g.sr = sr; g.slope = slope; g.zmul = 1.f;
    g.row_m = const_cast<float *>(row_m); g.row_inv = const_cast<float *>(row_inv); g.datt = da; g.dz = dz;
    g.out_absmax = dz_absmax;
    return launch_gat<true, 1>(g, (cudaStream_t)stream);
}

extern "C" int tango_edge_softmax(const int32_t *indptr, const int32_t *edge_ids, const int32_t *row_order,
                                  int64_t n_block_rows, int64_t n_rows, const float *z, int h, float zmul, float *a,
                                  float *a_absmax, tango_stream_t stream) {
    if (n_rows > 0 && (!indptr || !z || !a)) return TANGO_EINVAL;
    GatArgs g{indptr, nullptr, edge_ids, row_order, n_rows, n_block_rows, nullptr, nullptr, h, nullptr, nullptr, 1.f,
              a, nullptr, nullptr, z, zmul, a_absmax};
    return launch_gat<false>(g, (cudaStream_t)stream);
}

extern "C" int tango_edge_softmax_bwd(const int32_t *indptr, const int32_t *edge_ids, const int32_t *row_order,
                                      int64_t n_block_rows, int64_t n_rows, int h, float zmul, const float *a,
                                      const float *da, float *dz, float *dz_absmax, tango_stream_t stream) {
    if (n_rows > 0 && (!indptr || !a || !da || !dz)) return TANGO_EINVAL;
    GatArgs g{indptr, nullptr, edge_ids, row_order, n_rows, n_block_rows, nullptr, nullptr, h, nullptr, nullptr, 1.f,
              const_cast<float *>(a), da, dz, a, zmul, dz_absmax};
    return launch_gat<true>(g, (cudaStream_t)stream);
}
