// Absmax scale and quantisation of one or several fp32 matrices in ONE launch.
//
// Quantising a tensor needs its largest magnitude first, so it takes two sweeps over the data with a device-wide
// dependency in between.  Here both sweeps belong to one cooperative kernel: every CTA owns a contiguous band of a
// matrix, finds its maximum (and, on request, the column sums of the band), all CTAs meet at a grid barrier, and every CTA
// then quantises its own band BACKWARDS, so that what it read last -- up to about 100 MB over the whole grid -- comes
// from L2 instead of HBM.  Against a clear, an absmax kernel and a quantiser this saves two launches and a gap per
// tensor where the data is small (a layer's activation and weight share one launch), and most of the second read where
// it is large.
//
// Bound: HBM, 4 B (absmax sweep) + 4 B (quantise sweep, less what L2 keeps) + 1 B written per element.  A thread takes
// four consecutive elements of a row per step -- 128-bit loads where the row pitch allows, else 64- or 32-bit loads of
// neighbouring addresses that L1 merges -- and stores one packed word, so a warp reads 512 and writes 128 contiguous
// bytes whatever the row width; four steps are in flight per thread.
#include <cooperative_groups.h>

#include "common.cuh"

namespace tango {
namespace {

constexpr int kThreads = 256;
constexpr int kSteps = 4;            // units in flight per thread
constexpr int kStatRows = 8;         // rows in flight per thread of the sweep with column sums: latency-bound at four
                                     // (169,343 x 128: 49 us a launch with four, 43 with eight; 232,965 x 256: 125 and 109)
constexpr int kMaxJobs = 4;
constexpr float kRoundMagic = 12582912.f;   // 1.5 * 2^23: adding it leaves the integer nearest to t in the low mantissa bits

// Exact quotient of numbers below 2^31 by a fixed divisor.
struct FastDiv {
    uint32_t mul, shift, d;
    __host__ void set(uint32_t divisor) {
        d = divisor;
        uint32_t s = 0;
        while ((1ull << s) < d) ++s;
        shift = 31 + s;
        mul = (uint32_t)(((1ull << shift) + d - 1) / d);
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return (uint32_t)(((uint64_t)n * mul) >> shift); }
};

struct Job {
    const float *x, *gate, *row_scale;
    float *scale;               // read when `fixed`, else written
    const float *times[2];      // optional: product[i][0] = scale[0] * (times[i][0], or the scale of job times_job)
    float *product[2];
    int times_job;
    float *colsum;              // optional
    uint32_t *clear[2];         // optional: words set to zero for the kernels behind this one
    int64_t clear_words[2];
    int8_t *q;
    int64_t ldx, ldgate, ldq;
    uint32_t rows, cols;
    uint32_t upr;               // four-element units per output row
    FastDiv by_upr;
    uint32_t band;              // units of a CTA (rows of a CTA when column sums are taken)
    int first_block, n_blocks;
    float *part_max, *part_sum; // one maximum per CTA, [n_blocks, cols] column sums
    int vec;                    // floats per load: 4, 2 or 1
    int whole;                  // cols % 4 == 0: no unit is cut by the end of a row
    int word_store;             // rows of q start on 4-byte boundaries
    int flat_stats;             // x is one contiguous, 16-byte aligned stretch and needs no per-row factor: sweep it flat
    int fixed;                  // the scale is given
    uint64_t seed, call;
};

// The sweeps of a launch.
enum { BOTH_SWEEPS = 0, FIRST_SWEEP = 1, SECOND_SWEEP = 2 };

struct Params {
    Job job[kMaxJobs];
    int n_jobs;
    const unsigned long long *step;
};

// columns of a four-element unit at column c that exist (0..4)
__device__ __forceinline__ int left_in_row(uint32_t cols, uint32_t c) { return c < cols ? (int)min(4u, cols - c) : 0; }

// Four floats at p, of which `left` (0..4; WHOLE: 0 or 4) exist; the others read as zero, and zeros quantise to the zero
// bytes that the padding of a row has to hold.
template <int VEC, bool WHOLE>
__device__ __forceinline__ float4 load4(const float *p, int left) {
    if (left >= 4) {
        if (VEC == 4) return __ldg(reinterpret_cast<const float4 *>(p));
        if (VEC == 2) {
            const float2 a = __ldg(reinterpret_cast<const float2 *>(p)), b = __ldg(reinterpret_cast<const float2 *>(p) + 1);
            return make_float4(a.x, a.y, b.x, b.y);
        }
        return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
    }
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (WHOLE) return v;
    if (left > 0) v.x = __ldg(p);
    if (left > 1) v.y = __ldg(p + 1);
    if (left > 2) v.z = __ldg(p + 2);
    return v;
}

__device__ __forceinline__ float4 gated(const float4 &v, const float4 &g) {
    return make_float4(g.x <= 0.f ? 0.f : v.x, g.y <= 0.f ? 0.f : v.y, g.z <= 0.f ? 0.f : v.z, g.w <= 0.f ? 0.f : v.w);
}
__device__ __forceinline__ float4 scaled(const float4 &v, float s) {
    return make_float4(__fmul_rn(v.x, s), __fmul_rn(v.y, s), __fmul_rn(v.z, s), __fmul_rn(v.w, s));
}
__device__ __forceinline__ float absmax4(const float4 &v) {
    return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}

// ---- sweep 1, without column sums
template <int VEC, bool WHOLE, bool GATE>
__device__ __forceinline__ float rows_absmax(const Job &j, uint32_t beg, uint32_t end) {
    const float *x = j.x, *gate = j.gate, *row_scale = j.row_scale;
    float m = 0.f;
    for (uint32_t u0 = beg + threadIdx.x; u0 < end; u0 += kSteps * kThreads) {
        float4 v[kSteps];
        float s[kSteps];
#pragma unroll
        for (int k = 0; k < kSteps; ++k) {
            const uint32_t u = u0 + k * kThreads;
            v[k] = make_float4(0.f, 0.f, 0.f, 0.f); s[k] = 1.f;
            if (u < end) {
                const uint32_t r = j.by_upr.div(u), c = (u - r * j.upr) << 2;
                const int left = left_in_row(j.cols, c);
                v[k] = load4<VEC, WHOLE>(x + r * j.ldx + c, left);
                if (GATE) v[k] = gated(v[k], load4<VEC, WHOLE>(gate + r * j.ldgate + c, left));
                if (row_scale) s[k] = fabsf(__ldg(row_scale + r));
            }
        }
#pragma unroll
        for (int k = 0; k < kSteps; ++k) m = fmaxf(m, __fmul_rn(absmax4(v[k]), s[k]));
    }
    return m;
}

template <bool GATE>
__device__ __forceinline__ float band_absmax(const Job &j, int block) {
    if (j.flat_stats) {
        const int64_t numel = (int64_t)j.rows * j.cols, n4 = numel >> 2, per = (n4 + j.n_blocks - 1) / j.n_blocks;
        const int64_t beg = min(n4, per * block);
        const uint32_t n = (uint32_t)(min(n4, beg + per) - beg);
        const float4 *x4 = reinterpret_cast<const float4 *>(j.x) + beg;
        float m = 0.f;
        for (uint32_t i0 = threadIdx.x; i0 < n; i0 += kSteps * kThreads) {
            float4 v[kSteps];
#pragma unroll
            for (int k = 0; k < kSteps; ++k)
                v[k] = i0 + k * kThreads < n ? __ldg(x4 + i0 + k * kThreads) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < kSteps; ++k) m = fmaxf(m, absmax4(v[k]));
        }
        if (block == 0 && threadIdx.x < (numel & 3)) m = fmaxf(m, fabsf(__ldg(j.x + (n4 << 2) + threadIdx.x)));
        return m;
    }
    const uint32_t units = j.rows * j.upr, beg = min(units, j.band * block), end = min(units, j.band * (block + 1));
    if (GATE && j.gate) {
        if (j.vec == 4 && j.whole) return rows_absmax<4, true, true>(j, beg, end);
        if (j.vec >= 2) return rows_absmax<2, false, true>(j, beg, end);
        return rows_absmax<1, false, true>(j, beg, end);
    }
    if (j.vec == 4 && j.whole) return rows_absmax<4, true, false>(j, beg, end);
    if (j.vec >= 2) return rows_absmax<2, false, false>(j, beg, end);
    return rows_absmax<1, false, false>(j, beg, end);
}

// ---- sweep 1 with column sums of the (gated) values, before the per-row factor: thread tx owns VW columns, rows of the
// band are dealt to the thread groups and their sums added in a fixed order
template <int VW>
__device__ __forceinline__ float band_stats(const Job &j, int block, float *s_part) {
    const uint32_t r0 = j.band * block, r1 = min(j.rows, r0 + j.band);
    const float *x = j.x, *gate = j.gate, *row_scale = j.row_scale;
    const int64_t ldx = j.ldx, ldgate = j.ldgate;
    const uint32_t groups = (j.cols + VW - 1) / VW;
    int cw = 1;
    while (cw < (int)groups && cw < kThreads) cw <<= 1;
    const int tx = threadIdx.x & (cw - 1), ty = threadIdx.x / cw, nty = kThreads / cw;
    float m = 0.f;
    for (uint32_t g0 = 0; g0 < groups; g0 += cw) {
        const uint32_t c = (g0 + tx) * VW;
        float sum[VW];
#pragma unroll
        for (int i = 0; i < VW; ++i) sum[i] = 0.f;
        if (c < j.cols) {
            for (uint32_t r = r0 + ty; r < r1; r += nty * kStatRows) {
                float v[kStatRows][VW], s[kStatRows];
#pragma unroll
                for (int k = 0; k < kStatRows; ++k) {
                    const uint32_t rr = r + k * nty;
                    const bool in = rr < r1;
                    s[k] = 1.f;
                    if (VW == 4) {
                        float4 t = in ? __ldg(reinterpret_cast<const float4 *>(x + rr * ldx + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
                        if (in && gate) t = gated(t, __ldg(reinterpret_cast<const float4 *>(gate + rr * ldgate + c)));
                        v[k][0] = t.x; v[k][VW > 1 ? 1 : 0] = t.y; v[k][VW > 2 ? 2 : 0] = t.z; v[k][VW > 3 ? 3 : 0] = t.w;
                    } else {
                        v[k][0] = in ? __ldg(x + rr * ldx + c) : 0.f;
                        if (in && gate && __ldg(gate + rr * ldgate + c) <= 0.f) v[k][0] = 0.f;
                    }
                    if (in && row_scale) s[k] = fabsf(__ldg(row_scale + rr));
                }
#pragma unroll
                for (int k = 0; k < kStatRows; ++k)
#pragma unroll
                    for (int i = 0; i < VW; ++i) {
                        sum[i] = __fadd_rn(sum[i], v[k][i]);
                        m = fmaxf(m, __fmul_rn(fabsf(v[k][i]), s[k]));
                    }
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < VW; ++i) s_part[threadIdx.x * VW + i] = sum[i];
        __syncthreads();
        if (ty == 0 && c < j.cols) {
#pragma unroll
            for (int i = 0; i < VW; ++i) {
                float t = 0.f;
                for (int y = 0; y < nty; ++y) t = __fadd_rn(t, s_part[(y * cw + tx) * VW + i]);
                j.part_sum[(int64_t)block * j.cols + c + i] = t;
            }
        }
    }
    return m;
}

__device__ __forceinline__ float block_max(float m, float *s_warp) {
    m = warp_max(m);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = m;
    __syncthreads();
    float t = s_warp[0];
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w) t = fmaxf(t, s_warp[w]);
    return t;
}

// max / 127 over the CTAs of a job, once all of them have met
__device__ __forceinline__ float job_scale(const Job &j, float *s_warp) {
    float t = 0.f;
    for (int b = threadIdx.x; b < j.n_blocks; b += kThreads) t = fmaxf(t, __ldcg(j.part_max + b));
    return __fdiv_rn(block_max(t, s_warp), 127.0f);
}

// ---- sweep 2
// The clamp comes before the rounding, which changes nothing (127 is an integer) and makes NaN round to -127.
template <int MODE>
__device__ __forceinline__ uint32_t pack4(const float4 &v4, float inv, uint32_t f, const uint4 &r0, const uint4 &r1) {
    const float v[4] = {v4.x, v4.y, v4.z, v4.w};
    uint32_t b[4];
    if (MODE == TANGO_ROUND_STOCHASTIC) {
        // element i of flat index n draws lane n % 4 of Philox block n / 4: r0 is the block of the first element, whose
        // lane is f, r1 the block after it
        const uint32_t w[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t bits = f == 0 ? w[i] : f == 1 ? w[i + 1] : f == 2 ? w[i + 2] : w[i + 3];
            const float u = __fmul_rn((float)(bits >> 8), 5.9604644775390625e-08f);      // 2^-24
            b[i] = (uint32_t)round_to_i8(__fmul_rn(v[i], inv), TANGO_ROUND_STOCHASTIC, u);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float t = fminf(fmaxf(__fmul_rn(v[i], inv), -127.f), 127.f);
            b[i] = MODE == TANGO_ROUND_NEAREST ? __float_as_uint(__fadd_rn(t, kRoundMagic)) : (uint32_t)__float2int_rz(t);
        }
    }
    return __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}

// Quantises units [beg, end) of a job, from the end to the beginning.  FLAT: x and q are packed alike (one row).
template <int MODE, int VEC, bool WHOLE, bool FLAT, bool GATE>
__device__ __forceinline__ void quantize_units(const Job &j, uint32_t beg, uint32_t end, float inv, uint64_t call) {
    constexpr int S = MODE == TANGO_ROUND_STOCHASTIC ? 2 : kSteps;     // (bound by the random numbers, and by registers)
    const float *x = j.x, *gate = j.gate, *row_scale = j.row_scale;
    const Philox ph{(uint32_t)j.seed, (uint32_t)(j.seed >> 32)};
    const auto block_of = [&](uint64_t flat) {
        const uint64_t blk = flat >> 2;
        return ph((uint32_t)blk, (uint32_t)(blk >> 32), (uint32_t)call, (uint32_t)(call >> 32));
    };
    constexpr bool kOwnBlock = WHOLE || FLAT;      // units are aligned to the Philox blocks
    const uint32_t trips = end > beg ? (end - beg + S * kThreads - 1) / (S * kThreads) : 0;
    for (uint32_t t = trips; t-- > 0;) {
        const uint32_t u0 = beg + t * (S * kThreads) + threadIdx.x;
        float4 v[S];
        float s[S];
        uint32_t row[S], col[S];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const uint32_t u = u0 + k * kThreads;
            v[k] = make_float4(0.f, 0.f, 0.f, 0.f); s[k] = 1.f;
            row[k] = FLAT ? 0 : j.by_upr.div(u);
            col[k] = (u - row[k] * j.upr * (FLAT ? 0u : 1u)) << 2;
            if (u < end) {
                const int left = left_in_row(j.cols, col[k]);
                const int64_t off = FLAT ? (int64_t)col[k] : row[k] * j.ldx + col[k];
                v[k] = load4<VEC, WHOLE>(x + off, left);
                if (GATE) v[k] = gated(v[k], load4<VEC, WHOLE>(gate + (FLAT ? off : row[k] * j.ldgate + col[k]), left));
                if (!FLAT && row_scale) s[k] = __ldg(row_scale + row[k]);
            }
        }
        uint4 edge = make_uint4(0, 0, 0, 0);
        if (MODE == TANGO_ROUND_STOCHASTIC && !kOwnBlock) {
            // a unit that is not aligned to the Philox blocks needs the block of the unit after it, which the next lane
            // computes for itself; for lane 31 the first S lanes compute it, one step each
            const uint32_t un = u0 - (threadIdx.x & 31) + 32 + (threadIdx.x & 31) % S * kThreads;
            const uint32_t rn = j.by_upr.div(un);
            edge = block_of((uint64_t)rn * j.cols + ((un - rn * j.upr) << 2));
        }
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const bool in = u0 + k * kThreads < end;
            const uint64_t flat = (uint64_t)row[k] * j.cols + col[k];
            uint4 r0 = make_uint4(0, 0, 0, 0), r1 = r0;
            if (MODE == TANGO_ROUND_STOCHASTIC) {
                r0 = block_of(flat);
                if (!kOwnBlock) {
                    r1 = make_uint4(__shfl_down_sync(0xffffffffu, r0.x, 1), __shfl_down_sync(0xffffffffu, r0.y, 1),
                                    __shfl_down_sync(0xffffffffu, r0.z, 1), __shfl_down_sync(0xffffffffu, r0.w, 1));
                    const uint4 e = make_uint4(__shfl_sync(0xffffffffu, edge.x, k), __shfl_sync(0xffffffffu, edge.y, k),
                                               __shfl_sync(0xffffffffu, edge.z, k), __shfl_sync(0xffffffffu, edge.w, k));
                    if ((threadIdx.x & 31) == 31) r1 = e;
                }
            }
            if (!in) continue;
            if (!FLAT && row_scale) v[k] = scaled(v[k], s[k]);
            const uint32_t w = pack4<MODE>(v[k], inv, kOwnBlock ? 0 : (uint32_t)flat & 3u, r0, r1);
            int8_t *o = j.q + (FLAT ? (int64_t)col[k] : row[k] * j.ldq + col[k]);
            if (WHOLE || (j.word_store && (int64_t)col[k] + 4 <= j.ldq)) {
                *reinterpret_cast<uint32_t *>(o) = w;
            } else {
                for (int i = 0; i < 4 && (int64_t)col[k] + i < j.ldq; ++i) o[i] = (int8_t)(w >> (8 * i));
            }
        }
    }
}

// The variants worth having: packed words, aligned rows of whole units, and rows that are only 8- or 4-byte aligned or cut.
template <int MODE, bool GATE>
__device__ __forceinline__ void quantize_band(const Job &j, uint32_t beg, uint32_t end, float inv, uint64_t call) {
    const bool words = j.whole && j.word_store && j.ldq % 4 == 0;
    if (j.vec == 4 && j.rows == 1 && !j.row_scale) quantize_units<MODE, 4, false, true, GATE>(j, beg, end, inv, call);
    else if (j.vec == 4 && words) quantize_units<MODE, 4, true, false, GATE>(j, beg, end, inv, call);
    else if (j.vec >= 2) quantize_units<MODE, 2, false, false, GATE>(j, beg, end, inv, call);
    else quantize_units<MODE, 1, false, false, GATE>(j, beg, end, inv, call);
}

// EXT: jobs with a gate or column sums take part; STATS: false when every scale is given (no barrier, ordinary launch).
// SWEEPS is a template parameter because a test of it at run time cost the EXT forms registers (1 % of a launch).
template <bool STATS, int MODE, bool EXT, int SWEEPS>
__global__ void __launch_bounds__(kThreads, MODE == TANGO_ROUND_STOCHASTIC && EXT ? 3 : MODE == TANGO_ROUND_STOCHASTIC || EXT ? 4 : 5) quantize_fused_kernel(const __grid_constant__ Params p) {
    __shared__ float s_part[EXT && STATS ? kThreads * 4 : 1];
    __shared__ float s_warp[kThreads / 32];
    int ji = 0;
    while (ji + 1 < p.n_jobs && (int)blockIdx.x >= p.job[ji + 1].first_block) ++ji;
    const Job &j = p.job[ji];
    const int block = blockIdx.x - j.first_block;
    if (SWEEPS != SECOND_SWEEP) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
            for (int64_t i = (int64_t)block * kThreads + threadIdx.x; i < j.clear_words[k]; i += (int64_t)j.n_blocks * kThreads)
                j.clear[k][i] = 0;
    }
    float scale;
    if (STATS) {
        if (SWEEPS != SECOND_SWEEP) {
            float m = 0.f;
            if (EXT && j.colsum) m = j.vec == 4 && j.cols % 4 == 0 ? band_stats<4>(j, block, s_part) : band_stats<1>(j, block, s_part);
            else if (!j.fixed) m = band_absmax<EXT>(j, block);
            m = block_max(m, s_warp);
            if (threadIdx.x == 0) j.part_max[block] = m;
            if (SWEEPS == FIRST_SWEEP) return;
            if (gridDim.x > 1) cooperative_groups::this_grid().sync();
            else __syncthreads();
        }
        if (j.fixed) {
            scale = __ldg(j.scale);
        } else {
            scale = job_scale(j, s_warp);
            if (block == 0 && threadIdx.x == 0) *j.scale = scale;
        }
        if (EXT && j.colsum) {
            // one warp per column, the columns spread over the CTAs: the CTAs' sums in 32 interleaved chains, then a fixed
            // butterfly (the other warps are already quantising)
            const int lane = threadIdx.x & 31;
            for (uint32_t c = block + (threadIdx.x >> 5) * j.n_blocks; c < j.cols; c += j.n_blocks * (kThreads / 32)) {
                float t = 0.f;
                for (int b = lane; b < j.n_blocks; b += 32) t = __fadd_rn(t, __ldcg(j.part_sum + (int64_t)b * j.cols + c));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
                if (lane == 0) j.colsum[c] = t;
            }
        }
    } else {
        scale = __ldg(j.scale);
    }
    if (block == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (!j.product[i]) continue;
            float other;
            if (j.times[i]) other = __ldg(j.times[i]);
            else if (p.job[j.times_job].fixed) other = __ldg(p.job[j.times_job].scale);
            else other = job_scale(p.job[j.times_job], s_warp);
            if (threadIdx.x == 0) *j.product[i] = __fmul_rn(scale, other);
        }
    }
    const uint64_t call = effective_call(j.call, p.step);
    const float inv = inv_scale(scale);
    uint32_t beg, end;
    if (EXT && j.colsum) {                       // the band is whole rows
        beg = min(j.rows, j.band * block) * j.upr;
        end = min(j.rows, j.band * (block + 1)) * j.upr;
    } else {
        beg = min(j.rows * j.upr, j.band * block);
        end = min(j.rows * j.upr, j.band * (block + 1));
    }
    if (EXT && j.gate) quantize_band<MODE, EXT>(j, beg, end, inv, call);
    else quantize_band<MODE, false>(j, beg, end, inv, call);
}

typedef void (*KernelFn)(const Params);

struct Launch {
    Params p;
    KernelFn fn;
    int blocks;
    bool cooperative, ext;
    int64_t scratch_floats;
};

template <bool STATS, bool EXT, int SWEEPS>
KernelFn pick_mode(int mode) {
    return mode == TANGO_ROUND_STOCHASTIC ? quantize_fused_kernel<STATS, TANGO_ROUND_STOCHASTIC, EXT, SWEEPS>
         : mode == TANGO_ROUND_NEAREST    ? quantize_fused_kernel<STATS, TANGO_ROUND_NEAREST, EXT, SWEEPS>
                                          : quantize_fused_kernel<STATS, TANGO_ROUND_TRUNC, EXT, SWEEPS>;
}
template <int SWEEPS>
KernelFn pick(bool stats, int mode, bool ext) {
    if constexpr (SWEEPS != BOTH_SWEEPS) return ext ? pick_mode<true, true, SWEEPS>(mode) : pick_mode<true, false, SWEEPS>(mode);
    return stats ? (ext ? pick_mode<true, true, BOTH_SWEEPS>(mode) : pick_mode<true, false, BOTH_SWEEPS>(mode))
                 : (ext ? pick_mode<false, true, BOTH_SWEEPS>(mode) : pick_mode<false, false, BOTH_SWEEPS>(mode));
}

// Resident CTAs per SM of a variant; the same on every B200, so one query per variant and process.
int occupancy(KernelFn fn, int variant) {
    static int known[12] = {0};       // benign race: every thread computes the same value
    if (!known[variant]) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kThreads, 0) != cudaSuccess || n < 1) n = 1;
        known[variant] = n;
    }
    return known[variant];
}

// SMs of the current device, asked for once per device; a B200's where there is none to ask (size queries on a host).
int device_sms() {
    constexpr int kDevices = 64;
    static int known[kDevices] = {0};      // benign race: every thread stores the same value
    int dev = -1, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return kNumSMs;
    if (!known[dev] && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) known[dev] = n;
    return known[dev] ? known[dev] : kNumSMs;
}

// Column sums: every CTA writes one row of them to scratch.  Beyond 2^24 floats (64 MB; rows of 28,000 columns and more where
// the matrix fills the device) the caller sums the columns apart.
constexpr int64_t kMaxPartSums = 1 << 24;

int plan(const tango_quant_job *jobs, int n, const uint64_t *step, Launch &l) {
    if (!jobs || n < 1 || n > kMaxJobs) return TANGO_EINVAL;
    l.p = Params{};
    l.p.step = reinterpret_cast<const unsigned long long *>(step);
    bool stats = false, ext = false;
    int64_t units[kMaxJobs], total = 0;
    int m = 0;
    for (int k = 0; k < n; ++k) {
        const tango_quant_job &s = jobs[k];
        if (s.rows < 0 || s.cols < 0 || s.ldx < s.cols || s.ldq < s.cols || s.mode < 0 || s.mode > 2 || !s.scale ||
            (s.gate && s.ldgate < s.cols) || (s.colsum && s.fixed_scale))
            return TANGO_EINVAL;
        for (int i = 0; i < 2; ++i) {
            if (s.clear_words[i] < 0 || (s.clear_words[i] > 0 && !s.clear[i])) return TANGO_EINVAL;
            if (s.product[i] && !s.times[i] && (s.times_job < 0 || s.times_job >= n || s.fixed_scale)) return TANGO_EINVAL;
        }
        if (s.rows > 0 && s.cols > 0 && (!s.x || !s.q)) return TANGO_EINVAL;
        if (s.rows > 0 && s.ldq > 0 && !s.q) return TANGO_EINVAL;
        Job j{};
        j.x = s.x; j.gate = s.gate; j.row_scale = s.row_scale; j.scale = s.scale;
        j.times_job = s.times_job;
        for (int i = 0; i < 2; ++i) { j.times[i] = s.times[i]; j.product[i] = s.product[i]; }
        for (int i = 0; i < 2; ++i) { j.clear[i] = static_cast<uint32_t *>(s.clear[i]); j.clear_words[i] = s.clear_words[i]; }
        j.colsum = s.colsum; j.q = s.q; j.seed = s.seed; j.call = s.call; j.fixed = s.fixed_scale;
        int64_t rows = s.rows, cols = s.cols, ldx = s.ldx, ldq = s.ldq, ldg = s.ldgate;
        const bool packed = ldx == cols && (!s.gate || ldg == cols);
        j.flat_stats = ldx == cols && !s.gate && !s.row_scale && !s.colsum && aligned(s.x, 16);
        if (packed && ldq == cols && !s.row_scale && !s.colsum && rows * cols < (1ll << 32)) {
            cols = rows * cols; rows = 1; ldx = ldq = ldg = cols;      // one flat row: the same flat element index
        }
        const int64_t upr = ceil_div(ldq, 4);
        if (rows >= (1ll << 31) || cols >= (1ll << 32) || rows * upr >= (1ll << 31) - 65536 * 1024) return TANGO_ESIZE;
        j.rows = (uint32_t)rows; j.cols = (uint32_t)cols; j.ldx = ldx; j.ldq = ldq; j.ldgate = ldg;
        j.upr = (uint32_t)(upr > 0 ? upr : 1);
        j.by_upr.set(j.upr);
        auto fits = [&](int v) {
            return aligned(s.x, 4 * v) && (rows == 1 || ldx % v == 0) && (!s.gate || (aligned(s.gate, 4 * v) && (rows == 1 || ldg % v == 0)));
        };
        j.vec = fits(4) ? 4 : fits(2) ? 2 : 1;
        j.whole = cols % 4 == 0;
        j.word_store = aligned(s.q, 4) && (rows == 1 || ldq % 4 == 0);
        stats |= !s.fixed_scale;
        if (s.mode != jobs[0].mode) return TANGO_EINVAL;
        ext |= s.gate != nullptr || s.colsum != nullptr;
        units[m] = rows * upr;
        total += units[m];
        l.p.job[m++] = j;
    }
    l.p.n_jobs = m;
    l.fn = pick<BOTH_SWEEPS>(stats, jobs[0].mode, ext);
    l.ext = ext;
    // enough CTAs to fill the device with four units per thread, never more than are resident at once (the barrier)
    const int64_t resident = (int64_t)device_sms() * occupancy(l.fn, (stats ? 6 : 0) + (ext ? 3 : 0) + jobs[0].mode);
    int64_t want = ceil_div(total, kThreads * (total < 148 * 4 * kThreads ? 2 : kSteps));
    if (stats && want > resident) want = resident;
    if (want > (1 << 20)) want = 1 << 20;
    int first = 0;
    l.scratch_floats = 0;
    for (int k = 0; k < m; ++k) {
        Job &j = l.p.job[k];
        int64_t nb = total > 0 ? (int64_t)((double)want * units[k] / total + 0.5) : 1;
        const int64_t left = resident - (m - 1 - k) - first;      // one CTA at least for every job that follows
        if (stats && nb > left) nb = left;
        if (nb < 1) nb = 1;
        if (j.colsum) {
            if (nb > j.rows && j.rows > 0) nb = j.rows;
            j.band = (uint32_t)ceil_div(j.rows, nb);
            if (j.band > 0) nb = ceil_div(j.rows, j.band);
        } else {
            j.band = (uint32_t)round_up(ceil_div(units[k], nb), kThreads);
            if (j.band > 0 && units[k] > 0) nb = ceil_div(units[k], j.band);
        }
        if (nb < 1) nb = 1;
        j.first_block = first;
        j.n_blocks = (int)nb;
        first += (int)nb;
        if (j.colsum && nb * (int64_t)j.cols > kMaxPartSums) return TANGO_ESIZE;
        l.scratch_floats += nb + (j.colsum ? nb * (int64_t)j.cols : 0);
    }
    l.blocks = first;
    if (!stats) l.scratch_floats = 0;
    l.cooperative = stats && first > 1;
    return TANGO_OK;
}

}  // namespace
}  // namespace tango

using namespace tango;

extern "C" int64_t tango_quantize_fused_scratch_bytes(const tango_quant_job *jobs, int n_jobs) {
    Launch l;
    const int rc = plan(jobs, n_jobs, nullptr, l);
    return rc == TANGO_OK ? l.scratch_floats * (int64_t)sizeof(float) : rc;
}

static int run(const tango_quant_job *jobs, int n_jobs, const uint64_t *step, void *scratch, int64_t scratch_bytes,
               bool one_launch, cudaStream_t stream) {
    Launch l;
    const int rc = plan(jobs, n_jobs, step, l);
    if (rc) return rc;
    if (l.scratch_floats > 0 && (!scratch || l.scratch_floats * (int64_t)sizeof(float) > scratch_bytes)) return TANGO_EINVAL;
    float *f = static_cast<float *>(scratch);
    for (int k = 0; k < l.p.n_jobs && l.scratch_floats > 0; ++k) {
        Job &j = l.p.job[k];
        j.part_max = f;
        f += j.n_blocks;
        j.part_sum = f;
        if (j.colsum) f += (int64_t)j.n_blocks * j.cols;
    }
    void *args[] = {&l.p};
    const dim3 grid(l.blocks), block(kThreads);
    if (!l.cooperative) {
        TANGO_CUDA_TRY(cudaLaunchKernel((const void *)l.fn, grid, block, args, 0, stream));
        return TANGO_OK;
    }
    if (one_launch) {
        const cudaError_t e = cudaLaunchCooperativeKernel((const void *)l.fn, grid, block, args, 0, stream);
        if (e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorNotSupported) {
            TANGO_CUDA_TRY(e);
            return TANGO_OK;
        }
        (void)cudaGetLastError();        // fewer SMs for this process than the device has: no barrier then
    }
    TANGO_CUDA_TRY(cudaLaunchKernel((const void *)pick<FIRST_SWEEP>(true, jobs[0].mode, l.ext), grid, block, args, 0, stream));
    TANGO_CUDA_TRY(cudaLaunchKernel((const void *)pick<SECOND_SWEEP>(true, jobs[0].mode, l.ext), grid, block, args, 0, stream));
    return TANGO_OK;
}

extern "C" int tango_quantize_fused(const tango_quant_job *jobs, int n_jobs, const uint64_t *step, void *scratch,
                                    int64_t scratch_bytes, tango_stream_t stream) {
    return run(jobs, n_jobs, step, scratch, scratch_bytes, true, (cudaStream_t)stream);
}

extern "C" int tango_quantize_two_launches(const tango_quant_job *jobs, int n_jobs, const uint64_t *step, void *scratch,
                                           int64_t scratch_bytes, tango_stream_t stream) {
    return run(jobs, n_jobs, step, scratch, scratch_bytes, false, (cudaStream_t)stream);
}
