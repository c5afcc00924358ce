// Gradients of the attention projections of a GAT layer, el[n,h] = <x[n,h,:], al[h,:]> and er with ar, fp32 throughout:
//   dx[n,h,:] = (dx + dr[n,h] * ar[h,:]) + dl[n,h] * al[h,:],  dal[h,:] = sum_n dl[n,h] * x[n,h,:],  dar likewise
//
// Bound: HBM, one sweep that reads x and dx and writes dx.  Operator by operator it is four products of the size of x, two
// reductions over them and two sums.
#include "common.cuh"

namespace tango {
namespace {

constexpr int kThreads = 256;
constexpr int kRows = 4;       // rows in flight per thread

struct ProjArgs {
    const float *x, *al, *ar;
    int64_t rows;
    int H, D, F;
    const float *dl, *dr;
    float *dx;
    float *part;               // [bands, 2, F]
    int64_t band;              // rows per CTA
};

template <int VEC>
__device__ __forceinline__ void load(const float *p, float (&v)[VEC]) {
    if (VEC == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
        v[0] = t.x; v[1 % VEC] = t.y; v[2 % VEC] = t.z; v[3 % VEC] = t.w;
    } else {
        v[0] = __ldg(p);
    }
}

// Thread tx of a CTA owns VEC columns, the rows of the CTA's band are dealt to its thread rows; their sums are added in a
// fixed order.  blockIdx.y: which kThreads * VEC columns.
template <int VEC>
__global__ void __launch_bounds__(kThreads) project_bwd_kernel(const ProjArgs a, int cw) {
    __shared__ float s_part[2][kThreads * VEC];
    const int tx = threadIdx.x % cw, ty = threadIdx.x / cw, nty = kThreads / cw;
    const int c = (blockIdx.y * cw + tx) * VEC;
    const int64_t r0 = (int64_t)blockIdx.x * a.band, r1 = min(a.rows, r0 + a.band);
    float sl[VEC], sr[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) sl[e] = sr[e] = 0.f;
    if (c < a.F) {
        const int head = c / a.D;
        float wl[VEC], wr[VEC];
        load<VEC>(a.al + c, wl);
        load<VEC>(a.ar + c, wr);
        for (int64_t r = r0 + ty; r < r1; r += (int64_t)nty * kRows) {
            float v[kRows][VEC], d[kRows][VEC], gl[kRows], gr[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const int64_t rr = r + (int64_t)k * nty;
                gl[k] = gr[k] = 0.f;
#pragma unroll
                for (int e = 0; e < VEC; ++e) v[k][e] = d[k][e] = 0.f;
                if (rr < r1) {
                    gl[k] = __ldg(a.dl + rr * a.H + head);
                    gr[k] = __ldg(a.dr + rr * a.H + head);
                    if (a.part) load<VEC>(a.x + rr * a.F + c, v[k]);
                    if (a.dx) {
#pragma unroll
                        for (int e = 0; e < VEC; ++e)
                            if (VEC == 1) d[k][e] = a.dx[rr * a.F + c + e];
                        if (VEC == 4) {
                            const float4 t = *reinterpret_cast<const float4 *>(a.dx + rr * a.F + c);
                            d[k][0] = t.x; d[k][1 % VEC] = t.y; d[k][2 % VEC] = t.z; d[k][3 % VEC] = t.w;
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const int64_t rr = r + (int64_t)k * nty;
                if (rr >= r1) break;
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    sl[e] += gl[k] * v[k][e];
                    sr[e] += gr[k] * v[k][e];
                    d[k][e] += gr[k] * wr[e];      // the order in which the operator chain's gradients of x meet
                    d[k][e] += gl[k] * wl[e];
                }
                if (a.dx) {
                    float *o = a.dx + rr * a.F + c;
                    if (VEC == 4) *reinterpret_cast<float4 *>(o) = make_float4(d[k][0], d[k][1 % VEC], d[k][2 % VEC], d[k][3 % VEC]);
                    else o[0] = d[k][0];
                }
            }
        }
    }
    if (!a.part) return;
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
        s_part[0][threadIdx.x * VEC + e] = sl[e];
        s_part[1][threadIdx.x * VEC + e] = sr[e];
    }
    __syncthreads();
    if (ty == 0 && c < a.F) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            float tl = 0.f, tr = 0.f;
            for (int y = 0; y < nty; ++y) {
                tl += s_part[0][(y * cw + tx) * VEC + e];
                tr += s_part[1][(y * cw + tx) * VEC + e];
            }
            float *p = a.part + (int64_t)blockIdx.x * 2 * a.F + c + e;
            p[0] = tl;
            p[a.F] = tr;
        }
    }
}

// One warp per column of the [bands, 2, F] partial sums: 32 interleaved chains, then a fixed butterfly.
__global__ void __launch_bounds__(kThreads) project_sum_kernel(const float *__restrict__ part, int64_t bands, int F,
                                                               float *__restrict__ dal, float *__restrict__ dar) {
    const int64_t c = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (c >= 2 * (int64_t)F) return;
    float t = 0.f;
    for (int64_t b = lane; b < bands; b += 32) t += __ldg(part + b * 2 * F + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) (c < F ? dal : dar)[c < F ? c : c - F] = t;
}

struct Split {
    int vec, cw;
    int64_t band, bands;
};

Split split(int64_t n, int h, int d, bool wide) {
    Split s;
    const int64_t f = (int64_t)h * d;
    s.vec = wide && d % 4 == 0 ? 4 : 1;
    s.cw = 1;
    while (s.cw < (f + s.vec - 1) / s.vec && s.cw < kThreads) s.cw <<= 1;
    // four CTAs per SM if that leaves a thread a few trips over its rows, fewer where there are not enough rows
    const int64_t trip = (int64_t)(kThreads / s.cw) * kRows;
    const int64_t bands = n > 0 ? ceil_div(n, trip) : 0;
    s.band = ceil_div(n, bands < kNumSMs * 4 ? (bands > 0 ? bands : 1) : kNumSMs * 4);
    s.bands = s.band > 0 ? ceil_div(n, s.band) : 0;
    return s;
}

bool valid(int64_t n, int h, int d) { return n >= 0 && h >= 1 && d >= 1 && (int64_t)h * d <= (1 << 20); }

}  // namespace
}  // namespace tango

using namespace tango;

extern "C" int64_t tango_gat_project_bwd_scratch_bytes(int64_t n, int h, int d) {
    if (!valid(n, h, d)) return TANGO_EINVAL;
    const Split wide = split(n, h, d, true), narrow = split(n, h, d, false);
    return (wide.bands > narrow.bands ? wide.bands : narrow.bands) * 2 * h * d * (int64_t)sizeof(float);
}

extern "C" int tango_gat_project_bwd(const float *x, int64_t n, int h, int d, const float *al, const float *ar,
                                     const float *dl, const float *dr, float *dx, float *dal, float *dar, void *scratch,
                                     int64_t scratch_bytes, tango_stream_t stream) {
    if (!valid(n, h, d) || (dal == nullptr) != (dar == nullptr)) return TANGO_EINVAL;
    const int f = h * d;
    if (n > 0 && (!al || !ar || !dl || !dr || (dal && !x))) return TANGO_EINVAL;
    if (dal && n > 0 && (!scratch || scratch_bytes < tango_gat_project_bwd_scratch_bytes(n, h, d))) return TANGO_EINVAL;
    ProjArgs a{};
    a.x = x; a.al = al; a.ar = ar; a.rows = n; a.H = h; a.D = d; a.F = f; a.dl = dl; a.dr = dr; a.dx = dx;
    a.part = dal ? static_cast<float *>(scratch) : nullptr;
    const Split s = split(n, h, d, aligned(x, 16) && aligned(al, 16) && aligned(ar, 16) && aligned(dx, 16));
    a.band = s.band;
    if (n > 0 && (dx || dal)) {
        const dim3 grid((unsigned)s.bands, (unsigned)ceil_div(ceil_div(f, s.vec), s.cw));
        if (s.vec == 4) project_bwd_kernel<4><<<grid, kThreads, 0, (cudaStream_t)stream>>>(a, s.cw);
        else project_bwd_kernel<1><<<grid, kThreads, 0, (cudaStream_t)stream>>>(a, s.cw);
        TANGO_LAUNCH_CHECK();
    }
    if (dal) {
        project_sum_kernel<<<(unsigned)ceil_div(2 * (int64_t)f, kThreads / 32), kThreads, 0, (cudaStream_t)stream>>>(
            static_cast<const float *>(scratch), s.bands, f, dal, dar);
        TANGO_LAUNCH_CHECK();
    }
    return TANGO_OK;
}
