// CSR SpMM over int8 node (or edge) features with exact int32 accumulation.
//
// One warp owns one output row (or one "unit" = slice of a long row).  Within the warp, G lanes cover one
// neighbour's feature row with VEC-byte loads (G * VEC >= padded feature width) and 32/G neighbours are gathered per
// step.  Neighbour ids are fetched 32 at a time with one coalesced load (the next batch is prefetched) and handed out
// by shuffle; four gathers are in flight per lane (eight for narrow rows).  The same word of four neighbours is
// byte-transposed with PRMT and added with a 4-way dp4a against (1,1,1,1) (copy-u) or the four neighbours' int8
// weights (u_mul_e), so every accumulator is an exact int32.  Rows longer than the plan's threshold are cut into
// units that add into an int32 scratch row with integer atomics (order independent => deterministic), and the last one to
// arrive finishes the row; rows of at most 48 neighbours are handled by lane groups (short_rows); all three kinds share
// one launch; in-edge sums over contiguous edge rows have their own streaming kernel (incidence_kernel).
#include "common.cuh"

namespace tango {

struct SpmmArgs {
    const int32_t *indptr;
    const int32_t *indices;   // feature-row id per slot; NULL => the slot number itself
    const int32_t *edge_ids;  // edge id per slot for the weight lookup; NULL => the slot number itself
    int64_t n_rows;
    int nseg;
    const int8_t *feat;
    int64_t ld;
    int f;      // logical feature bytes per row
    int f_pad;  // bytes the lanes may read (multiple of VEC, <= ld)
    const int8_t *ew;  // [E, H] int8 edge weights (weighted modes)
    int H, D;
    const float *scales;  // [nseg]
    const float *row_scale;
    const float *bias;
    int relu;
    float *out;
    int64_t ldo;
    float *out_absmax;
    const int32_t *units;
    int64_t n_units;
    const int32_t *heavy_rows;
    int64_t n_heavy;
    int32_t *ws;
    int64_t ws_ld;
    int split_threshold;
    const int32_t *row_order;
    const int4 *row_info;  // optional, in row_order's order: (row, first slot, end slot, -), one load instead of two trips
    int32_t *arrivals;     // optional, one counter per heavy row: the last unit of a row finishes it (ws and counters hold 0)
    int unit;              // slots per unit
    int64_t n_long;   // rows row_order[0, n_long) get a warp each, the rest a lane group
    int64_t n_few, n_one;  // with row_info: rows from n_few on have at most kFew neighbours, from n_one on at most one
    int64_t long_blocks, short_blocks, few_blocks;   // CTAs of units and long rows, then of the short rows, then of those with
                                                     // a few neighbours; the rest of the grid takes the rows with one
    int G;  // lanes per neighbour (power of two)
    int word_weights;      // the H weights of an edge are one aligned word of 1, 2 or 4 bytes
};

// WEIGHT_WORD: the lane that holds a neighbour's id also loads its weights, as one word (H = 1, 2, 4), and hands it out by
// shuffle; WEIGHT_LANE: every lane of a group loads its head's byte; WEIGHT_ELEM: one byte per element.
enum { MODE_COPY = 0, MODE_WEIGHT_LANE = 1, MODE_WEIGHT_ELEM = 2, MODE_WEIGHT_WORD = 3 };

template <int VEC> struct VecLoad;
template <> struct VecLoad<16> {
    uint32_t w[4];
    __device__ __forceinline__ void load(const int8_t *p) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    }
    __device__ __forceinline__ void zero() { w[0] = w[1] = w[2] = w[3] = 0; }
};
template <> struct VecLoad<4> {
    uint32_t w[1];
    __device__ __forceinline__ void load(const int8_t *p) { w[0] = __ldg(reinterpret_cast<const uint32_t *>(p)); }
    __device__ __forceinline__ void zero() { w[0] = 0; }
};
template <> struct VecLoad<1> {
    uint32_t w[1];
    __device__ __forceinline__ void load(const int8_t *p) { w[0] = (uint32_t)(uint8_t)__ldg(p); }
    __device__ __forceinline__ void zero() { w[0] = 0; }
};

// Adds one byte of one neighbour (VEC == 1) or, for the per-element weight mode, VEC bytes with their own weights.
template <int VEC, int MODE>
__device__ __forceinline__ void accumulate_one(int (&acc)[VEC], const VecLoad<VEC> &v, uint32_t wsel,
                                               const int8_t *wrow, int off, const SpmmArgs &a) {
    if (VEC == 1) {
        const int b = (int)(int8_t)(v.w[0] & 0xff);
        if (MODE == MODE_COPY) acc[0] += b;
        else acc[0] += b * (int)(int8_t)wsel;
        return;
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const uint32_t word = v.w[i >> 2];
        const int col = off + i;
        const int wv = (wrow && col < a.f) ? (int)__ldg(wrow + col / a.D) : 0;
        acc[i] += (int)(int8_t)((word >> (8 * (i & 3))) & 0xff) * wv;
    }
}

// Adds four neighbours at once.  The same word of the four rows is byte-transposed with 8 PRMTs so that each result
// word holds one feature of the four neighbours; one 4-way dp4a against (1,1,1,1) -- or against the four neighbours'
// int8 weights -- then adds all four into the int32 accumulator: 12 instructions per 16 gathered bytes.
template <int VEC>
__device__ __forceinline__ void accumulate_four(int (&acc)[VEC], const VecLoad<VEC> *v, uint32_t wvec) {
#pragma unroll
    for (int wp = 0; wp < VEC / 4; ++wp) {
        const uint32_t a = v[0].w[wp], b = v[1].w[wp], c = v[2].w[wp], d = v[3].w[wp];
        const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(c, d, 0x5140);
        const uint32_t t2 = __byte_perm(a, b, 0x7362), t3 = __byte_perm(c, d, 0x7362);
        acc[4 * wp + 0] = __dp4a((int)__byte_perm(t0, t1, 0x5410), (int)wvec, acc[4 * wp + 0]);
        acc[4 * wp + 1] = __dp4a((int)__byte_perm(t0, t1, 0x7632), (int)wvec, acc[4 * wp + 1]);
        acc[4 * wp + 2] = __dp4a((int)__byte_perm(t2, t3, 0x5410), (int)wvec, acc[4 * wp + 2]);
        acc[4 * wp + 3] = __dp4a((int)__byte_perm(t2, t3, 0x7632), (int)wvec, acc[4 * wp + 3]);
    }
}

// The weights of one edge as a packed word (head h in byte h); H is 1, 2 or 4.
__device__ __forceinline__ uint32_t weight_word(const SpmmArgs &a, int eid) {
    const int8_t *p = a.ew + (uint64_t)(uint32_t)eid * (uint32_t)a.H;
    return a.H == 4 ? __ldg(reinterpret_cast<const uint32_t *>(p))
         : a.H == 2 ? (uint32_t)__ldg(reinterpret_cast<const uint16_t *>(p)) : (uint32_t)(uint8_t)__ldg(p);
}
// Byte `head` of four edges' words as the multiplier of accumulate_four; sel = head | (head + 4) << 4.
__device__ __forceinline__ uint32_t four_weights(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t sel) {
    return __byte_perm(__byte_perm(w0, w1, sel), __byte_perm(w2, w3, sel), 0x5410);
}

// Sums the neighbours of slots [beg, end) into acc for the feature bytes [off, off + VEC) handled by this lane.
// On return every lane of group 0 (lane < G) holds the full sum for its bytes.  Lanes whose bytes lie beyond the
// feature width run the same instruction stream on the row's first bytes (their sums are never stored), so the hot
// loop over full batches of 32 neighbours carries no predicates at all.
template <int VEC, int MODE, bool DEEP = false>
__device__ __forceinline__ void gather_segment(int (&acc)[VEC], int beg, int end, int off, bool active,
                                               const SpmmArgs &a) {
    const int lane = threadIdx.x & 31;
    const int G = a.G, NB = 32 / G, grp = lane / G;
    constexpr int U = 4;
    constexpr bool kFour = (VEC >= 4) && (MODE != MODE_WEIGHT_ELEM);
#pragma unroll
    for (int i = 0; i < VEC; ++i) acc[i] = 0;
    const int ld_off = active ? off : 0;
    const int head = (MODE == MODE_WEIGHT_LANE || MODE == MODE_WEIGHT_WORD) ? ld_off / a.D : 0;
    const uint32_t wsel_of = (uint32_t)head | (uint32_t)(head + 4) << 4;
    const int8_t *base = a.feat + ld_off;
    const int8_t *wbase = (MODE == MODE_WEIGHT_LANE) ? a.ew + head : a.ew;
    const uint32_t ld = (uint32_t)a.ld;   // 32 x 32 -> 64-bit products: one wide multiply per gathered row
    const int H = a.H;
    int j0 = beg;
    if (DEEP && kFour && G == 4) {
        // ---- narrow rows (four lanes per neighbour): a batch of 32 ids is only four gathers per lane, so two batches
        // are taken together to keep eight gathers in flight per lane.
        int nxt_a = 0, nxt_b = 0, nxt_ea = 0, nxt_eb = 0;
        if (j0 + 64 <= end) {
            nxt_a = a.indices ? __ldg(a.indices + j0 + lane) : j0 + lane;
            nxt_b = a.indices ? __ldg(a.indices + j0 + 32 + lane) : j0 + 32 + lane;
            if (MODE != MODE_COPY) {
                nxt_ea = a.edge_ids ? __ldg(a.edge_ids + j0 + lane) : j0 + lane;
                nxt_eb = a.edge_ids ? __ldg(a.edge_ids + j0 + 32 + lane) : j0 + 32 + lane;
            }
        }
        for (; j0 + 64 <= end; j0 += 64) {
            const int idx_a = nxt_a, idx_b = nxt_b, eid_a = nxt_ea, eid_b = nxt_eb;
            if (j0 + 128 <= end) {
                nxt_a = a.indices ? __ldg(a.indices + j0 + 64 + lane) : j0 + 64 + lane;
                nxt_b = a.indices ? __ldg(a.indices + j0 + 96 + lane) : j0 + 96 + lane;
                if (MODE != MODE_COPY) {
                    nxt_ea = a.edge_ids ? __ldg(a.edge_ids + j0 + 64 + lane) : j0 + 64 + lane;
                    nxt_eb = a.edge_ids ? __ldg(a.edge_ids + j0 + 96 + lane) : j0 + 96 + lane;
                }
            }
            VecLoad<VEC> v[8];
            uint32_t wv0 = 0x01010101u, wv1 = 0x01010101u;
            uint32_t w_a = 0, w_b = 0;
            if (MODE == MODE_WEIGHT_WORD) { w_a = weight_word(a, eid_a); w_b = weight_word(a, eid_b); }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int src_lane = grp + (u & 3) * 8;
                const int idx = __shfl_sync(0xffffffffu, u < 4 ? idx_a : idx_b, src_lane);
                v[u].load(base + (uint64_t)(uint32_t)idx * ld);
                if (MODE == MODE_WEIGHT_LANE) {
                    const int eid = __shfl_sync(0xffffffffu, u < 4 ? eid_a : eid_b, src_lane);
                    const uint32_t wb = (uint32_t)(uint8_t)__ldg(wbase + (uint64_t)(uint32_t)eid * (uint32_t)H);
                    if (u < 4) wv0 = (u == 0) ? wb : (wv0 | (wb << (8 * u)));
                    else wv1 = (u == 4) ? wb : (wv1 | (wb << (8 * (u - 4))));
                }
            }
            if (MODE == MODE_WEIGHT_WORD) {
                wv0 = four_weights(__shfl_sync(0xffffffffu, w_a, grp), __shfl_sync(0xffffffffu, w_a, grp + 8),
                                   __shfl_sync(0xffffffffu, w_a, grp + 16), __shfl_sync(0xffffffffu, w_a, grp + 24), wsel_of);
                wv1 = four_weights(__shfl_sync(0xffffffffu, w_b, grp), __shfl_sync(0xffffffffu, w_b, grp + 8),
                                   __shfl_sync(0xffffffffu, w_b, grp + 16), __shfl_sync(0xffffffffu, w_b, grp + 24), wsel_of);
            }
            accumulate_four<VEC>(acc, v, wv0);
            accumulate_four<VEC>(acc, v + 4, wv1);
        }
    }
    if (kFour && G >= U) {
        // ---- full batches: every shuffled index is valid, four loads in flight per lane, no predicates.
        // The indices of the next batch are fetched while the current one is processed.
        int nxt_idx = 0, nxt_eid = 0;
        if (j0 + 32 <= end) {
            nxt_idx = a.indices ? __ldg(a.indices + j0 + lane) : j0 + lane;
            if (MODE != MODE_COPY) nxt_eid = a.edge_ids ? __ldg(a.edge_ids + j0 + lane) : j0 + lane;
        }
        for (; j0 + 32 <= end; j0 += 32) {
            const int my_idx = nxt_idx, my_eid = nxt_eid;
            if (j0 + 64 <= end) {
                nxt_idx = a.indices ? __ldg(a.indices + j0 + 32 + lane) : j0 + 32 + lane;
                if (MODE != MODE_COPY) nxt_eid = a.edge_ids ? __ldg(a.edge_ids + j0 + 32 + lane) : j0 + 32 + lane;
            }
            uint32_t my_w = 0;
            if (MODE == MODE_WEIGHT_WORD) my_w = weight_word(a, my_eid);
            for (int s = 0, lane0 = grp; s < G; s += U, lane0 += U * NB) {
                VecLoad<VEC> v[U];
                uint32_t wvec = 0x01010101u;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int src_lane = lane0 + u * NB;
                    const int idx = __shfl_sync(0xffffffffu, my_idx, src_lane);
                    v[u].load(base + (uint64_t)(uint32_t)idx * ld);
                    if (MODE == MODE_WEIGHT_LANE) {
                        const int eid = __shfl_sync(0xffffffffu, my_eid, src_lane);
                        const uint32_t wb = (uint32_t)(uint8_t)__ldg(wbase + (uint64_t)(uint32_t)eid * (uint32_t)H);
                        wvec = (u == 0) ? wb : (wvec | (wb << (8 * u)));
                    }
                }
                if (MODE == MODE_WEIGHT_WORD)
                    wvec = four_weights(__shfl_sync(0xffffffffu, my_w, lane0), __shfl_sync(0xffffffffu, my_w, lane0 + NB),
                                        __shfl_sync(0xffffffffu, my_w, lane0 + 2 * NB),
                                        __shfl_sync(0xffffffffu, my_w, lane0 + 3 * NB), wsel_of);
                accumulate_four<VEC>(acc, v, wvec);
            }
        }
    }
    // ---- ragged tail (and every batch of the narrow or per-element-weight configurations): predicated
    for (; j0 < end; j0 += 32) {
        const int j = j0 + lane;
        int my_idx = -1, my_eid = 0;
        if (j < end) {
            my_idx = a.indices ? __ldg(a.indices + j) : j;
            if (MODE != MODE_COPY) my_eid = a.edge_ids ? __ldg(a.edge_ids + j) : j;
        }
        uint32_t my_w = 0;
        if (MODE == MODE_WEIGHT_WORD && my_idx >= 0) my_w = weight_word(a, my_eid);
        const int steps = min(G, (end - j0 + NB - 1) / NB);
        for (int s = 0; s < steps; s += U) {
            VecLoad<VEC> v[U];
            uint32_t wsel[U];
            const int8_t *wrow[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int src_lane = ((s + u) * NB + grp) & 31;
                int idx = __shfl_sync(0xffffffffu, my_idx, src_lane);
                int eid = 0;
                if (MODE == MODE_WEIGHT_LANE || MODE == MODE_WEIGHT_ELEM) eid = __shfl_sync(0xffffffffu, my_eid, src_lane);
                if (s + u >= steps) idx = -1;
                wsel[u] = 0; wrow[u] = nullptr;
                if (MODE == MODE_WEIGHT_WORD) wsel[u] = __shfl_sync(0xffffffffu, my_w, src_lane);
                if (idx >= 0) {
                    v[u].load(base + (uint64_t)(uint32_t)idx * ld);
                    if (MODE == MODE_WEIGHT_LANE) wsel[u] = (uint32_t)(uint8_t)__ldg(wbase + (uint64_t)(uint32_t)eid * (uint32_t)H);
                    if (MODE == MODE_WEIGHT_ELEM) wrow[u] = a.ew + (uint64_t)(uint32_t)eid * (uint32_t)H;
                } else {
                    v[u].zero();
                }
            }
            if (kFour) {
                uint32_t wvec = 0x01010101u;
                if (MODE == MODE_WEIGHT_LANE) wvec = wsel[0] | (wsel[1] << 8) | (wsel[2] << 16) | (wsel[3] << 24);
                if (MODE == MODE_WEIGHT_WORD) wvec = four_weights(wsel[0], wsel[1], wsel[2], wsel[3], wsel_of);
                accumulate_four<VEC>(acc, v, wvec);
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) accumulate_one<VEC, MODE>(acc, v[u], wsel[u], wrow[u], ld_off, a);
            }
        }
    }
    for (int o = G; o < 32; o <<= 1) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    }
}

__device__ __forceinline__ float finish_value(float v, int64_t row, int col, const SpmmArgs &a) {
    if (a.row_scale) v = __fmul_rn(v, __ldg(a.row_scale + row));
    if (a.bias) v = __fadd_rn(v, __ldg(a.bias + col));
    if (a.relu) v = fmaxf(v, 0.f);
    return v;
}

constexpr int kSpmmThreads = 128;   // four warps (four rows or slices) per CTA
constexpr int kFew = 4, kFewRows = 2, kOneRows = 2;   // rows of at most 4 neighbours: two at a time

__device__ __forceinline__ void record_absmax(const SpmmArgs &a, float amax) {
    if (!a.out_absmax) return;
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0 && amax > 0.f) {
        const float s = __fdiv_rn(amax, 127.0f);
        if (s > __ldcg(a.out_absmax)) atomic_max_nonneg(a.out_absmax, s);
    }
}

// Finishes one row that went through the int32 scratch: four features per lane.
__device__ __forceinline__ void finish_columns(const SpmmArgs &a, int64_t slot, int64_t row, int col0, float &amax) {
    float facc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < a.nseg; ++k) {
        const int4 v = __ldcg(reinterpret_cast<const int4 *>(a.ws + (slot * a.nseg + k) * a.ws_ld + col0));   // ws_ld % 16 == 0
        const float sc = __ldg(a.scales + k);
        facc[0] = __fadd_rn(facc[0], __fmul_rn((float)v.x, sc));
        facc[1] = __fadd_rn(facc[1], __fmul_rn((float)v.y, sc));
        facc[2] = __fadd_rn(facc[2], __fmul_rn((float)v.z, sc));
        facc[3] = __fadd_rn(facc[3], __fmul_rn((float)v.w, sc));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        facc[i] = finish_value(facc[i], row, min(col0 + i, a.f - 1), a);
        if (col0 + i < a.f) amax = fmaxf(amax, fabsf(facc[i]));
    }
    float *o = a.out + row * a.ldo + col0;
    if (col0 + 4 <= a.f && (a.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0) {
        *reinterpret_cast<float4 *>(o) = make_float4(facc[0], facc[1], facc[2], facc[3]);
    } else {
        for (int i = 0; i < 4 && col0 + i < a.f; ++i) o[i] = facc[i];
    }
}

// Stores the lane's VEC values of a row.
template <int VEC>
__device__ __forceinline__ void store_values(const SpmmArgs &a, const float (&facc)[VEC], int64_t row, int off) {
    float *o = a.out + row * a.ldo + off;
    if (VEC == 16 && off + 16 <= a.f && (a.ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 31) == 0) {
        uint32_t r[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) r[i] = __float_as_uint(facc[i]);
        store_v8(o, r);
        store_v8(o + 8, r + (VEC == 16 ? 8 : 0));
    } else if (VEC >= 4 && off + VEC <= a.f && (a.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < VEC / 4; ++i)
            reinterpret_cast<float4 *>(o)[i] = make_float4(facc[4 * i], facc[(4 * i + 1) % VEC], facc[(4 * i + 2) % VEC], facc[(4 * i + 3) % VEC]);
    } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i)
            if (off + i < a.f) o[i] = facc[i];
    }
}

// With arrival counters, the warp that has added the last slice of a row finishes it.
__device__ __forceinline__ void finish_if_last(const SpmmArgs &a, const int4 &u, float &amax) {
    if (!a.arrivals) return;
    const int lane = threadIdx.x & 31;
    __threadfence();
    __syncwarp();
    const int units = (__ldg(a.indptr + u.x + 1) - __ldg(a.indptr + u.x) + a.unit - 1) / a.unit;
    int before = 0;
    if (lane == 0) before = atomicAdd(a.arrivals + u.w, 1);
    if (__shfl_sync(0xffffffffu, before, 0) != units - 1) return;
    __threadfence();
    for (int c = lane * 4; c < a.f; c += 128) finish_columns(a, u.w, u.x, c, amax);
}

// A slice of a long row: integer partial sums into scratch.
template <int VEC, int MODE, bool DEEP>
__device__ __forceinline__ void long_row_unit(const SpmmArgs &a, int64_t w, float &amax) {
    const int lane = threadIdx.x & 31, sub = lane % a.G;
    const int4 u = __ldg(reinterpret_cast<const int4 *>(a.units) + w);  // (vrow, beg, end, slot)
    for (int fb = 0; fb < a.f_pad; fb += 32 * VEC) {
        const int off = fb + sub * VEC;
        const bool active = off < a.f_pad;
        int acc[VEC];
        gather_segment<VEC, MODE, DEEP>(acc, u.y, u.z, off, active, a);
        if (active && lane < a.G) {
#pragma unroll
            for (int i = 0; i < VEC; ++i)
                if (off + i < a.f && acc[i] != 0) atomicAdd(a.ws + (int64_t)u.w * a.ws_ld + off + i, acc[i]);
        }
    }
    finish_if_last(a, u, amax);
}

template <int VEC, int MODE, bool DEEP>
__device__ __forceinline__ void long_row(const SpmmArgs &a, int64_t i, float &amax) {
    const int lane = threadIdx.x & 31, sub = lane % a.G;
    const int64_t row = a.row_order ? (int64_t)__ldg(a.row_order + i) : i;
    const int32_t *ip = a.indptr + row * a.nseg;
    const int row_beg = __ldg(ip), row_end = __ldg(ip + a.nseg);
    if (a.n_heavy > 0 && row_end - row_beg > a.split_threshold) return;  // covered by units
    for (int fb = 0; fb < a.f_pad; fb += 32 * VEC) {
        const int off = fb + sub * VEC;
        const bool active = off < a.f_pad;
        float facc[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) facc[i] = 0.f;
        for (int k = 0; k < a.nseg; ++k) {
            int acc[VEC];
            gather_segment<VEC, MODE, DEEP>(acc, __ldg(ip + k), __ldg(ip + k + 1), off, active, a);
            const float sc = __ldg(a.scales + k);
#pragma unroll
            for (int i = 0; i < VEC; ++i) facc[i] = __fadd_rn(facc[i], __fmul_rn((float)acc[i], sc));
        }
        if (active && lane < a.G) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                facc[i] = finish_value(facc[i], row, min(off + i, a.f - 1), a);
                if (off + i < a.f) amax = fmaxf(amax, fabsf(facc[i]));
            }
            store_values<VEC>(a, facc, row, off);
        }
    }
}

// Adds `cnt` (1..4) neighbours whose pieces are v[0..cnt): one or two of them byte by byte (4 instructions a word each),
// three or four with the transpose (12 a word whatever the count).
template <int VEC, int MODE>
__device__ __forceinline__ void accumulate_some(int (&acc)[VEC], VecLoad<VEC> (&v)[4], uint32_t wvec, int cnt) {
    if (cnt > 2) {
        accumulate_four<VEC>(acc, v, wvec);
        return;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        if (u < cnt) {
            // byte i of the word times the neighbour's weight: the weight in byte i of an otherwise zero multiplier
            const uint32_t w = (wvec >> (8 * u)) & 0xffu;
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[i] = __dp4a((int)v[u].w[i >> 2], (int)(w << (8 * (i & 3))), acc[i]);
        }
    }
}

// One segment: 0 + acc * scale as in the segmented form (adding zero only matters for a product of -0, which a positive
// scale does not give).
template <int VEC>
__device__ __forceinline__ void dequantize_row(const SpmmArgs &a, const int (&acc)[VEC], float (&facc)[VEC]) {
    const float sc = __ldg(a.scales);
#pragma unroll
    for (int i = 0; i < VEC; ++i) facc[i] = __fmul_rn((float)acc[i], sc);
    if (!(sc > 0.f)) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) facc[i] = __fadd_rn(0.f, facc[i]);
    }
}

// The optional steps and the store of a short row's bytes [off, off + VEC).
template <int VEC>
__device__ __forceinline__ void store_row(const SpmmArgs &a, float (&facc)[VEC], int64_t row, int off, float &amax) {
    // short rows are as much epilogue as gather: the optional per-element steps are decided once, not per element
    if (a.row_scale) {
        const float rs = __ldg(a.row_scale + row);
#pragma unroll
        for (int i = 0; i < VEC; ++i) facc[i] = __fmul_rn(facc[i], rs);
    }
    if (a.bias) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) facc[i] = __fadd_rn(facc[i], __ldg(a.bias + min(off + i, a.f - 1)));
    }
    if (a.relu) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) facc[i] = fmaxf(facc[i], 0.f);
    }
    if (a.out_absmax) {
#pragma unroll
        for (int i = 0; i < VEC; ++i)
            if (off + i < a.f) amax = fmaxf(amax, fabsf(facc[i]));
    }
    store_values<VEC>(a, facc, row, off);
}

// Short rows: a group of G lanes owns one row (32 / G rows per warp) and needs no cross-lane reduction -- the
// warp-per-row form would spend most of its time in the ragged tail on rows with a handful of neighbours.  Such a
// row is a short dependent chain (row bounds -> neighbour ids -> gathers -> store), so what matters is how few round
// trips it takes and how many rows are in flight: row_info brings a row and its bounds in one load, and with four or more
// lanes per row the group fetches G neighbour ids (and edge ids) with ONE coalesced load and hands them out by shuffles
// restricted to the group; narrower groups read the ids one by one.
// MULTI: rows cut into per-shard segments with a scale each (row-partitioned multi-GPU aggregation).
template <int VEC, int MODE, bool MULTI>
__device__ __forceinline__ void short_rows(const SpmmArgs &a, int64_t block, float &amax) {
    const int lane = threadIdx.x & 31;
    const int G = a.G, sub = lane % G;
    const int64_t gid = (block * blockDim.x + threadIdx.x) / G;
    const int64_t n_short = (a.row_info && !MULTI ? a.n_few : a.n_rows) - a.n_long;
    const int off = sub * VEC;
    const bool in_range = gid < n_short;
    const bool active = in_range && off < a.f_pad;
    const unsigned gmask = (G >= 32) ? 0xffffffffu : (((1u << G) - 1u) << (lane - sub));
    const int base_lane = lane - sub;
    int64_t row = 0;
    int row_beg = 0, row_end = 0;
    const int32_t *ip = a.indptr;
    if (in_range) {
        if (a.row_info && !MULTI) {
            const int4 r = __ldg(a.row_info + a.n_long + gid);
            row = r.x; row_beg = r.y; row_end = r.z;
        } else {
            row = a.row_order ? (int64_t)__ldg(a.row_order + a.n_long + gid) : a.n_long + gid;
            ip = a.indptr + row * a.nseg;
            if (!MULTI) { row_beg = __ldg(ip); row_end = __ldg(ip + 1); }
        }
    }
    const int8_t *base = a.feat + (active ? off : 0);
    const int head = (MODE == MODE_WEIGHT_LANE || MODE == MODE_WEIGHT_WORD) ? (active ? off : 0) / a.D : 0;
    const uint32_t wsel = (uint32_t)head | (uint32_t)(head + 4) << 4;
    float facc[VEC];
    if (MULTI) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) facc[i] = 0.f;
    }
    const int nseg = in_range ? (MULTI ? a.nseg : 1) : 0;
    int acc[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) acc[i] = 0;
    for (int k = 0; k < nseg; ++k) {
        const int beg = MULTI ? __ldg(ip + k) : row_beg, end = MULTI ? __ldg(ip + k + 1) : row_end;
        if (MULTI) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[i] = 0;
        }
        if (G >= 4) {
            for (int j0 = beg; j0 < end; j0 += G) {
                const int j = j0 + sub;
                int my_idx = 0, my_eid = 0;
                uint32_t my_w = 0;
                if (j < end) {
                    my_idx = a.indices ? __ldg(a.indices + j) : j;
                    if (MODE == MODE_WEIGHT_LANE || MODE == MODE_WEIGHT_WORD) my_eid = a.edge_ids ? __ldg(a.edge_ids + j) : j;
                    if (MODE == MODE_WEIGHT_WORD) my_w = weight_word(a, my_eid);
                }
                const int cnt = min(G, end - j0);
                for (int s0 = 0; s0 < cnt; s0 += 4) {
                    VecLoad<VEC> v[4];
                    uint32_t wvec = (MODE == MODE_WEIGHT_LANE) ? 0u : 0x01010101u;
                    uint32_t ww[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int src = base_lane + ((s0 + u) & (G - 1));
                        const int idx = __shfl_sync(gmask, my_idx, src);
                        int eid = 0;
                        if (MODE == MODE_WEIGHT_LANE) eid = __shfl_sync(gmask, my_eid, src);
                        if (MODE == MODE_WEIGHT_WORD) ww[u] = __shfl_sync(gmask, my_w, src);
                        if (s0 + u < cnt) {
                            v[u].load(base + (uint64_t)(uint32_t)idx * (uint32_t)a.ld);
                            if (MODE == MODE_WEIGHT_LANE)
                                wvec |= (uint32_t)(uint8_t)__ldg(a.ew + (uint64_t)(uint32_t)eid * (uint32_t)a.H + head) << (8 * u);
                        } else {
                            v[u].zero();
                        }
                    }
                    if (MODE == MODE_WEIGHT_WORD) wvec = four_weights(ww[0], ww[1], ww[2], ww[3], wsel);
                    accumulate_some<VEC, MODE>(acc, v, wvec, cnt - s0);
                }
            }
        } else {
            for (int j = beg; j < end; j += 4) {
                VecLoad<VEC> v[4];
                uint32_t wvec = (MODE == MODE_COPY) ? 0x01010101u : 0u;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (j + u < end) {
                        const int idx = a.indices ? __ldg(a.indices + j + u) : j + u;
                        v[u].load(base + (uint64_t)(uint32_t)idx * (uint32_t)a.ld);
                        if (MODE == MODE_WEIGHT_LANE || MODE == MODE_WEIGHT_WORD) {
                            const int eid = a.edge_ids ? __ldg(a.edge_ids + j + u) : j + u;
                            wvec |= (uint32_t)(uint8_t)__ldg(a.ew + (uint64_t)(uint32_t)eid * (uint32_t)a.H + head) << (8 * u);
                        }
                    } else {
                        v[u].zero();
                    }
                }
                accumulate_some<VEC, MODE>(acc, v, wvec, end - j);
            }
        }
        if (MULTI) {
            const float sc = __ldg(a.scales + k);
#pragma unroll
            for (int i = 0; i < VEC; ++i) facc[i] = __fadd_rn(facc[i], __fmul_rn((float)acc[i], sc));
        }
    }
    if (!active) return;
    if (!MULTI) dequantize_row<VEC>(a, acc, facc);
    store_row<VEC>(a, facc, row, off, amax);
}

// Rows with at most K neighbours -- four fifths of the rows of a sparse power-law graph, half of them with their self loop
// alone.  Such a row is three dependent loads (bounds, ids, features) and a store, so the time is latency over rows in
// flight: a lane group takes R rows side by side.
template <int VEC, int MODE, int R, int K>
__device__ __forceinline__ void few_rows(const SpmmArgs &a, int64_t block, int64_t first, int64_t last, float &amax) {
    const int lane = threadIdx.x & 31;
    const int G = a.G, sub = lane % G;                      // G >= 4
    const int64_t r0 = first + (block * blockDim.x + threadIdx.x) / G * R;
    const int off = sub * VEC;
    const bool active = off < a.f_pad;
    const unsigned gmask = (G >= 32) ? 0xffffffffu : (((1u << G) - 1u) << (lane - sub));
    const int base_lane = lane - sub;
    if (r0 >= last) return;                                 // uniform in a group
    const int4 mine = sub < R && r0 + sub < last ? __ldg(a.row_info + r0 + sub) : make_int4(-1, 0, 0, 0);
    int row[R], cnt[R], id[R];
    uint32_t w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        row[r] = __shfl_sync(gmask, mine.x, base_lane + r);
        const int beg = __shfl_sync(gmask, mine.y, base_lane + r);
        cnt[r] = __shfl_sync(gmask, mine.z, base_lane + r) - beg;
        id[r] = 0; w[r] = 0;
        const int j = beg + sub;
        if (sub < cnt[r]) {
            id[r] = a.indices ? __ldg(a.indices + j) : j;
            if (MODE == MODE_WEIGHT_WORD) w[r] = weight_word(a, a.edge_ids ? __ldg(a.edge_ids + j) : j);
        }
    }
    const int8_t *base = a.feat + (active ? off : 0);
    const int head = MODE == MODE_WEIGHT_WORD ? (active ? off : 0) / a.D : 0;
    VecLoad<VEC> v[R][K];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int idx = __shfl_sync(gmask, id[r], base_lane + k);
            if (k < cnt[r]) v[r][k].load(base + (uint64_t)(uint32_t)idx * (uint32_t)a.ld);
            else v[r][k].zero();
        }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        uint32_t wvec = 0x01010101u;
        if (MODE == MODE_WEIGHT_WORD) {
            wvec = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) wvec |= ((__shfl_sync(gmask, w[r], base_lane + k) >> (8 * head)) & 0xffu) << (8 * k);
        }
        int acc[VEC];
        if (K == 1) {
            const int wt = MODE == MODE_WEIGHT_WORD ? (int)(int8_t)wvec : 1;
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[i] = (int)(int8_t)(v[r][0].w[i >> 2] >> (8 * (i & 3))) * wt;
        } else {
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[i] = 0;
            VecLoad<VEC> four[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) four[k] = v[r][k < K ? k : 0];
            accumulate_some<VEC, MODE>(acc, four, wvec, cnt[r]);
        }
        if (row[r] >= 0 && active) {
            float facc[VEC];
            dequantize_row<VEC>(a, acc, facc);
            store_row<VEC>(a, facc, row[r], off, amax);
        }
    }
}

// One launch for all rows: the CTAs in front take the slices of the long rows and the medium rows (a warp each, the longest
// first), the CTAs behind them the short rows, which fill the SMs while the last long ones finish (interleaving the two
// kinds measured 5 % slower).  169 K rows of 8 edges, F = 128: 61 us as a clear, two gather kernels and a finalize kernel,
// 44 us as one launch; 22 us are the 87 MB of output at the card's write rate, half of the rest is the chain
// bounds -> ids -> features of the long rows.  Eight CTAs per SM: at six and seven (no spills) the gathers of a 114.6 M-edge
// graph measured 5 and 15 % slower, at ten the spills cost more than the warps gain.
template <int VEC, int MODE, bool DEEP, bool MULTI>
__global__ void __launch_bounds__(kSpmmThreads, DEEP || MULTI ? 6 : 8) spmm_kernel(const SpmmArgs a) {
    float amax = 0.f;
    if ((int64_t)blockIdx.x < a.long_blocks) {
        const int64_t w = (int64_t)blockIdx.x * (kSpmmThreads / 32) + (threadIdx.x >> 5);
        if (w < a.n_units) long_row_unit<VEC, MODE, DEEP>(a, w, amax);
        else if (w - a.n_units < a.n_long) long_row<VEC, MODE, DEEP>(a, w - a.n_units, amax);
    } else if (VEC >= 4 && MODE != MODE_WEIGHT_ELEM) {
        int64_t block = (int64_t)blockIdx.x - a.long_blocks;
        if (block < a.short_blocks) {
            short_rows<VEC, MODE, MULTI>(a, block, amax);
        } else if (!MULTI && MODE != MODE_WEIGHT_LANE) {
            block -= a.short_blocks;
            if (block < a.few_blocks) few_rows<VEC, MODE, kFewRows, kFew>(a, block, a.n_few, a.n_one, amax);
            else few_rows<VEC, MODE, kOneRows, 1>(a, block - a.few_blocks, a.n_one, a.n_rows, amax);
        }
    }
    record_absmax(a, amax);
}

// ---- incidence sums over contiguous edge rows: when slot j of a row IS edge j (edge ids follow the row order) and
// the edge features are packed [E, F] with F dividing 16, the edges of a row are one contiguous byte range.  It is
// streamed with aligned 128-bit loads, four in flight per lane; byte b of an aligned chunk belongs to column b % F.
template <int F>
__device__ __forceinline__ void add_chunk(int (&acc)[F], const uint4 &w) {
    if (F == 1) {
        acc[0] = __dp4a((int)w.x, 0x01010101, acc[0]); acc[0] = __dp4a((int)w.y, 0x01010101, acc[0]);
        acc[0] = __dp4a((int)w.z, 0x01010101, acc[0]); acc[0] = __dp4a((int)w.w, 0x01010101, acc[0]);
    } else if (F == 4) {
        const uint32_t t0 = __byte_perm(w.x, w.y, 0x5140), t1 = __byte_perm(w.z, w.w, 0x5140);
        const uint32_t t2 = __byte_perm(w.x, w.y, 0x7362), t3 = __byte_perm(w.z, w.w, 0x7362);
        acc[0 % F] = __dp4a((int)__byte_perm(t0, t1, 0x5410), 0x01010101, acc[0 % F]);
        acc[1 % F] = __dp4a((int)__byte_perm(t0, t1, 0x7632), 0x01010101, acc[1 % F]);
        acc[2 % F] = __dp4a((int)__byte_perm(t2, t3, 0x5410), 0x01010101, acc[2 % F]);
        acc[3 % F] = __dp4a((int)__byte_perm(t2, t3, 0x7632), 0x01010101, acc[3 % F]);
    } else {
        const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i % F] += (int)(int8_t)(ws[i >> 2] >> (8 * (i & 3)));
    }
}

template <int F>
__device__ __forceinline__ void contig_segment(int (&acc)[F], int beg, int end, const SpmmArgs &a) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < F; ++c) acc[c] = 0;
    const int64_t b0 = (int64_t)beg * F, b1 = (int64_t)end * F;
    const int64_t a0 = min(b1, (b0 + 15) & ~(int64_t)15), a1 = max(a0, b1 & ~(int64_t)15);
    // ragged head [b0, a0) and tail [a1, b1): fewer than 16 bytes each; both start on a multiple of F
    const int nh = (int)(a0 - b0), nt = (int)(b1 - a1);
    if (lane < nh || lane < nt) {
        const int vh = lane < nh ? (int)__ldg(a.feat + b0 + lane) : 0;
        const int vt = lane < nt ? (int)__ldg(a.feat + a1 + lane) : 0;
#pragma unroll
        for (int c = 0; c < F; ++c)
            if (lane % F == c) acc[c] += vh + vt;
    }
    const uint4 *chunks = reinterpret_cast<const uint4 *>(a.feat);
    const int64_t c1 = a1 >> 4;
    for (int64_t c = (a0 >> 4) + lane; c < c1; c += 128) {
        uint4 w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = (c + 32 * u < c1) ? __ldcs(chunks + c + 32 * u) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < 4; ++u) add_chunk<F>(acc, w[u]);
    }
#pragma unroll
    for (int c = 0; c < F; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
}

// The same when the edge ids are a list: a lane takes a whole record of F bytes, eight (four) of them in flight.
// Random records out of an array of E * F bytes are bound by L2 sectors in flight, not by bytes.
template <int F>
__device__ __forceinline__ void listed_segment(int (&acc)[F], int beg, int end, const SpmmArgs &a) {
    constexpr int U = F <= 4 ? 8 : 4;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < F; ++c) acc[c] = 0;
    for (int j0 = beg + lane; j0 < end; j0 += 32 * U) {
        int id[U];
#pragma unroll
        for (int u = 0; u < U; ++u) id[u] = j0 + 32 * u < end ? __ldg(a.indices + j0 + 32 * u) : -1;
        uint4 w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            w[u] = make_uint4(0, 0, 0, 0);
            if (id[u] < 0) continue;
            const int8_t *p = a.feat + (int64_t)id[u] * F;
            if (F == 16) w[u] = __ldg(reinterpret_cast<const uint4 *>(p));
            else if (F == 8) { const uint2 t = __ldg(reinterpret_cast<const uint2 *>(p)); w[u].x = t.x; w[u].y = t.y; }
            else if (F == 4) w[u].x = __ldg(reinterpret_cast<const uint32_t *>(p));
            else if (F == 2) w[u].x = __ldg(reinterpret_cast<const uint16_t *>(p));
            else w[u].x = (uint32_t)(uint8_t)__ldg(p);
        }
        if (F == 4) {
#pragma unroll
            for (int u = 0; u < U; u += 4) add_chunk<F>(acc, make_uint4(w[u].x, w[u + 1].x, w[u + 2].x, w[u + 3].x));
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t ws[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
                for (int c = 0; c < F; ++c) acc[c] += (int)(int8_t)(ws[c >> 2] >> (8 * (c & 3)));
            }
        }
    }
#pragma unroll
    for (int c = 0; c < F; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
}

// Units and medium rows as above, short rows (F of 4, 8 or 16) by lane groups in the CTAs behind them.
template <int F, bool LISTED>
__global__ void __launch_bounds__(kSpmmThreads, LISTED && F <= 4 ? 12 : 8) incidence_kernel(const SpmmArgs a) {
    if ((int64_t)blockIdx.x >= a.long_blocks) {
        float amax = 0.f;
        if (F >= 4) short_rows<F == 16 ? 16 : 4, MODE_COPY, false>(a, (int64_t)blockIdx.x - a.long_blocks, amax);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * (kSpmmThreads / 32) + (threadIdx.x >> 5);
    int acc[F];
    if (w < a.n_units) {
        const int4 u = __ldg(reinterpret_cast<const int4 *>(a.units) + w);
        if (LISTED) listed_segment<F>(acc, u.y, u.z, a);
        else contig_segment<F>(acc, u.y, u.z, a);
#pragma unroll
        for (int c = 0; c < F; ++c)
            if (lane == c && acc[c] != 0) atomicAdd(a.ws + (int64_t)u.w * a.ws_ld + c, acc[c]);
        float amax = 0.f;
        finish_if_last(a, u, amax);
    } else if (w - a.n_units < a.n_long) {
        int64_t row = w - a.n_units;
        if (a.row_order) row = __ldg(a.row_order + row);
        const int beg = __ldg(a.indptr + row), end = __ldg(a.indptr + row + 1);
        if (a.n_heavy > 0 && end - beg > a.split_threshold) return;   // covered by units
        if (LISTED) listed_segment<F>(acc, beg, end, a);
        else contig_segment<F>(acc, beg, end, a);
        const float sc = __ldg(a.scales);
#pragma unroll
        for (int c = 0; c < F; ++c)
            if (lane == c) a.out[row * a.ldo + c] = __fadd_rn(0.f, __fmul_rn((float)acc[c], sc));
    }
}

// Finishes the rows that went through the int32 scratch when no arrival counters were given (and the rows of the dense hub
// region): one thread per (heavy row, four features).
__global__ void __launch_bounds__(256) spmm_finalize_kernel(const SpmmArgs a) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int f4 = (a.f + 3) >> 2;
    float amax = 0.f;
    if (t < a.n_heavy * f4) {
        const int64_t slot = t / f4;
        finish_columns(a, slot, __ldg(a.heavy_rows + slot), (int)(t - slot * f4) << 2, amax);
    }
    record_absmax(a, amax);
}

// Packs the feature rows ids[0..n) of `src` ([*, ld] int8, ld a multiple of 16) into dst [n, ld]: the B operand of
// the dense hub block.
__global__ void __launch_bounds__(256) gather_rows_kernel(const int8_t *__restrict__ src, int64_t ld,
                                                          const int32_t *__restrict__ ids, int64_t n,
                                                          int8_t *__restrict__ dst) {
    const int64_t pieces = ld >> 4, total = n * pieces;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / pieces, c = i - r * pieces;
        reinterpret_cast<uint4 *>(dst + r * ld)[c] =
            __ldg(reinterpret_cast<const uint4 *>(src + (int64_t)__ldg(ids + r) * ld) + c);
    }
}

static int pow2_ceil(int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

// Scratch and schedule of the rows that are cut into units.  Without arrival counters the scratch is cleared here and
// finished by a kernel of its own.
static int take_units(SpmmArgs &a, const tango_spmm_plan *plan, cudaStream_t stream) {
    if (!plan) return TANGO_OK;
    a.row_order = plan->row_order;
    a.row_info = plan->row_order && aligned(plan->row_info, 16) ? reinterpret_cast<const int4 *>(plan->row_info) : nullptr;
    if (plan->n_units <= 0) return TANGO_OK;
    if (!plan->units || !plan->heavy_rows || !plan->ws || plan->ws_ld < a.f || plan->n_heavy <= 0) return TANGO_EINVAL;
    if (!aligned(plan->units, 16) || !aligned(plan->ws, 16) || plan->ws_ld % 4) return TANGO_EALIGN;
    a.units = plan->units; a.n_units = plan->n_units; a.heavy_rows = plan->heavy_rows;
    a.n_heavy = plan->n_heavy; a.ws = plan->ws; a.ws_ld = plan->ws_ld; a.split_threshold = plan->split_threshold;
    if (plan->arrivals) {
        if (a.nseg != 1 || plan->unit_slots <= 0 || plan->dense_a) return TANGO_EINVAL;
        a.arrivals = plan->arrivals; a.unit = plan->unit_slots;
    } else {
        TANGO_CUDA_TRY(cudaMemsetAsync(a.ws, 0, sizeof(int32_t) * (size_t)(a.n_heavy * a.nseg * a.ws_ld), stream));
    }
    return TANGO_OK;
}

static int finalize(const SpmmArgs &a, cudaStream_t stream) {
    const int64_t fb = ceil_div(a.n_heavy * ((a.f + 3) / 4), 256);
    spmm_finalize_kernel<<<(unsigned)fb, 256, 0, stream>>>(a);
    TANGO_LAUNCH_CHECK();
    return TANGO_OK;
}

template <int VEC, int MODE>
static int launch_rows(const SpmmArgs &a, unsigned blocks, cudaStream_t stream) {
    constexpr bool kDeep = VEC == 16;
    if (a.nseg > 1) spmm_kernel<VEC, MODE, false, true><<<blocks, kSpmmThreads, 0, stream>>>(a);
    else if (kDeep && a.G == 4) spmm_kernel<VEC, MODE, kDeep, false><<<blocks, kSpmmThreads, 0, stream>>>(a);
    else spmm_kernel<VEC, MODE, false, false><<<blocks, kSpmmThreads, 0, stream>>>(a);
    TANGO_LAUNCH_CHECK();
    return TANGO_OK;
}

template <int MODE>
static int launch_spmm(SpmmArgs &a, const tango_spmm_plan *plan, cudaStream_t stream) {
    if (a.n_rows == 0 || a.f == 0) return TANGO_OK;
    if (a.ld > 0x7fffffff) return TANGO_ESIZE;
    a.n_long = a.n_rows;
    const int rc = take_units(a, plan, stream);
    if (rc) return rc;
    const bool dense = plan && plan->dense_a && plan->dense_rows > 0 && plan->dense_n_cols > 0 && plan->dense_n_units > 0;
    if (dense) {
        // dense hub block: pack the block's feature rows, multiply on the tensor cores, add into the heavy rows'
        // int32 scratch (cleared above); the gather kernels below then cover only the edges outside the block
        if (MODE != MODE_COPY || a.nseg != 1 || plan->n_units < 0 || !plan->heavy_rows || !plan->ws ||
            plan->dense_rows > plan->n_heavy || !plan->dense_cols || !plan->dense_b || !plan->dense_units ||
            plan->dense_n_tiles <= 0 || plan->dense_rows % 128 || plan->dense_n_cols % 128 ||
            plan->n_skip_rows != plan->n_heavy || !plan->row_order || plan->ws_ld < a.f)
            return TANGO_EINVAL;
        if (a.ld % 16 || !aligned(a.feat, 16) || !aligned(plan->dense_a, 16) || !aligned(plan->dense_b, 16) ||
            !aligned(plan->dense_units, 16) || !aligned(plan->ws, 16) || plan->ws_ld % 4)
            return TANGO_EALIGN;
        if (plan->n_units == 0) {      // no unit set the scratch fields above
            a.heavy_rows = plan->heavy_rows; a.n_heavy = plan->n_heavy; a.ws = plan->ws; a.ws_ld = plan->ws_ld;
            a.split_threshold = plan->split_threshold;
            TANGO_CUDA_TRY(cudaMemsetAsync(a.ws, 0, sizeof(int32_t) * (size_t)(a.n_heavy * a.ws_ld), stream));
        }
        const int64_t ldb = round_up(a.f, 16);
        if (ldb > a.ld) return TANGO_EINVAL;
        {
            const int64_t pieces = plan->dense_n_cols * (ldb >> 4);
            int64_t gb = ceil_div(pieces, 256);
            if (gb > kNumSMs * 8) gb = kNumSMs * 8;
            if (ldb == a.ld) {
                gather_rows_kernel<<<(unsigned)gb, 256, 0, stream>>>(a.feat, a.ld, plan->dense_cols, plan->dense_n_cols,
                                                                    plan->dense_b);
            } else {
                return TANGO_EINVAL;   // feature rows wider than their padded width: not a layout the quantizers make
            }
            TANGO_LAUNCH_CHECK();
        }
        const int rc = igemm_accumulate_tiles_i32(plan->dense_a, plan->dense_n_tiles, plan->dense_units,
                                                  plan->dense_n_units, plan->dense_b, ldb, plan->dense_rows, a.f,
                                                  plan->dense_n_cols, a.ws, a.ws_ld, plan->dense_status, stream);
        if (rc) return rc;
    }
    if (plan && plan->n_skip_rows > 0) {
        // the leading rows of row_order belong to units + finalize: the row kernels start after them
        if (!plan->row_order || plan->n_skip_rows > a.n_rows || plan->n_long_rows < plan->n_skip_rows) return TANGO_EINVAL;
        a.row_order = plan->row_order + plan->n_skip_rows;
        if (a.row_info) a.row_info += plan->n_skip_rows;
        a.n_rows -= plan->n_skip_rows;
    }
    if (MODE == MODE_WEIGHT_LANE && a.H == 1) a.D = 1 << 20;  // one head: every byte shares the weight
    int vec = 1;
    if (a.ld % 16 == 0 && aligned(a.feat, 16)) vec = 16;
    else if (a.ld % 4 == 0 && aligned(a.feat, 4)) vec = 4;
    // narrow rows: prefer one lane per neighbour over mostly idle 16-byte lanes
    if (vec == 16 && a.f <= 4) vec = 4;
    a.f_pad = (int)round_up(a.f, vec);
    if (a.f_pad > a.ld) return TANGO_EINVAL;
    a.G = pow2_ceil((a.f_pad + vec - 1) / vec);
    if (a.G > 32) a.G = 32;
    if (MODE == MODE_WEIGHT_LANE && (a.D % vec) != 0) {
        // a lane's bytes must stay inside one head; fall back to narrower loads, else to the per-element mode
        if (vec == 16 && a.D % 4 == 0 && a.ld % 4 == 0) {
            vec = 4; a.f_pad = (int)round_up(a.f, 4); a.G = pow2_ceil(a.f_pad / 4); if (a.G > 32) a.G = 32;
        }
    }
    // short rows (the tail of the degree-sorted order) go to the lane-group kernel when one pass of G lanes covers a row
    const bool four = vec >= 4 && !(MODE == MODE_WEIGHT_LANE && (a.D % vec) != 0);
    const int64_t n_skip = plan ? plan->n_skip_rows : 0;
    if (plan && plan->row_order && plan->n_long_rows >= n_skip && plan->n_long_rows - n_skip <= a.n_rows && four &&
        a.f_pad <= 32 * vec)
        a.n_long = plan->n_long_rows - n_skip;
    else if (n_skip > 0) a.n_long = a.n_rows;
    const bool words = MODE == MODE_WEIGHT_LANE && (a.H == 1 || a.H == 2 || a.H == 4) && aligned(a.ew, a.H);
    // the few-neighbour form wants a lane per id and packed weights
    const int64_t over_few = plan ? plan->n_over_few - n_skip : 0, over_one = plan ? plan->n_over_one - n_skip : 0;
    const bool few = a.row_info && a.nseg == 1 && a.n_long < a.n_rows && four && a.G >= 4 && (MODE == MODE_COPY || words) &&
                     over_few >= a.n_long && over_one >= over_few && over_one <= a.n_rows;
    if (few) { a.n_few = over_few; a.n_one = over_one; }
    else { a.n_few = a.n_one = a.n_rows; }
    a.long_blocks = ceil_div(a.n_units + a.n_long, kSpmmThreads / 32);
    a.short_blocks = ceil_div((a.n_few - a.n_long) * a.G, kSpmmThreads);
    a.few_blocks = ceil_div(ceil_div(a.n_one - a.n_few, kFewRows) * a.G, kSpmmThreads);
    const int64_t blocks = a.long_blocks + a.short_blocks + a.few_blocks + ceil_div(ceil_div(a.n_rows - a.n_one, kOneRows) * a.G, kSpmmThreads);
    if (blocks > 0x7fffffff) return TANGO_ESIZE;
    int rc2 = TANGO_OK;
    if (blocks > 0) {
        const unsigned nb = (unsigned)blocks;
        if (MODE == MODE_WEIGHT_LANE && (a.D % vec) != 0) {
            if (vec == 16) rc2 = launch_rows<16, MODE_WEIGHT_ELEM>(a, nb, stream);
            else if (vec == 4) rc2 = launch_rows<4, MODE_WEIGHT_ELEM>(a, nb, stream);
            else rc2 = launch_rows<1, MODE_WEIGHT_LANE>(a, nb, stream);  // a lane holds one byte, always inside one head
        } else if (vec == 1) {
            rc2 = launch_rows<1, MODE>(a, nb, stream);
        } else if (words) {
            rc2 = vec == 16 ? launch_rows<16, MODE_WEIGHT_WORD>(a, nb, stream) : launch_rows<4, MODE_WEIGHT_WORD>(a, nb, stream);
        } else {
            rc2 = vec == 16 ? launch_rows<16, MODE>(a, nb, stream) : launch_rows<4, MODE>(a, nb, stream);
        }
    }
    if (rc2) return rc2;
    return (a.n_units > 0 && !a.arrivals) || dense ? finalize(a, stream) : TANGO_OK;
}

template <bool LISTED>
static void launch_incidence(const SpmmArgs &a, unsigned blocks, cudaStream_t stream) {
    switch (a.f) {
        case 1: incidence_kernel<1, LISTED><<<blocks, kSpmmThreads, 0, stream>>>(a); break;
        case 2: incidence_kernel<2, LISTED><<<blocks, kSpmmThreads, 0, stream>>>(a); break;
        case 4: incidence_kernel<4, LISTED><<<blocks, kSpmmThreads, 0, stream>>>(a); break;
        case 8: incidence_kernel<8, LISTED><<<blocks, kSpmmThreads, 0, stream>>>(a); break;
        default: incidence_kernel<16, LISTED><<<blocks, kSpmmThreads, 0, stream>>>(a); break;
    }
}

// Incidence sums over packed records (see incidence_kernel); returns false when the layout does not qualify.
static bool try_incidence(SpmmArgs &a, const tango_spmm_plan *plan, cudaStream_t stream, int &rc) {
    const int f = a.f;
    if (a.ld != f || !(f == 1 || f == 2 || f == 4 || f == 8 || f == 16) || !aligned(a.feat, a.indices ? f : 16)) return false;
    if (a.indices && plan && (plan->n_skip_rows > 0 || plan->dense_a)) return false;
    a.n_long = a.n_rows;
    rc = take_units(a, plan, stream);
    if (rc) return true;
    // rows with a handful of edges (the tail of the degree-sorted order) are cheaper with one lane group per row than
    // with a whole warp and its cross-lane reduction; that takes 4- or 16-byte pieces
    const int short_vec = (f == 16) ? 16 : (f == 4 || f == 8) ? 4 : 0;
    if (short_vec && plan && plan->row_order && plan->n_long_rows >= 0 && plan->n_long_rows <= a.n_rows) {
        a.n_long = plan->n_long_rows;
        a.f_pad = f;
        a.G = f / short_vec;          // 1 or 2 lanes per row
    }
    a.n_few = a.n_rows;
    a.long_blocks = ceil_div(a.n_units + a.n_long, kSpmmThreads / 32);
    const int64_t blocks = a.long_blocks + (short_vec ? ceil_div((a.n_rows - a.n_long) * a.G, kSpmmThreads) : 0);
    if (blocks > 0x7fffffff) { rc = TANGO_ESIZE; return true; }
    if (blocks > 0) {
        if (a.indices) launch_incidence<true>(a, (unsigned)blocks, stream);
        else launch_incidence<false>(a, (unsigned)blocks, stream);
        if (cudaPeekAtLastError() != cudaSuccess) { rc = TANGO_ECUDA; return true; }
    }
    if (a.n_units > 0 && !a.arrivals) rc = finalize(a, stream);
    return true;
}

}  // namespace tango

using namespace tango;

extern "C" int tango_spmm_copy_u(const int32_t *indptr, const int32_t *indices, int64_t n_rows, int nseg,
                                 const int8_t *nq, int64_t ldn, int64_t f, const float *scales, const float *row_scale,
                                 const float *bias, int relu, float *out, int64_t ldo, float *out_absmax,
                                 const tango_spmm_plan *plan, tango_stream_t stream) {
    if (n_rows < 0 || nseg < 1 || f < 0 || ldn < f || ldo < f || f > (1 << 20)) return TANGO_EINVAL;
    if (n_rows == 0 || f == 0) return TANGO_OK;
    if (!indptr || !indices || !nq || !scales || !out) return TANGO_EINVAL;
    SpmmArgs a{};
    a.indptr = indptr; a.indices = indices; a.edge_ids = nullptr; a.n_rows = n_rows; a.nseg = nseg;
    a.feat = nq; a.ld = ldn; a.f = (int)f; a.ew = nullptr; a.H = 1; a.D = (int)f;
    a.scales = scales; a.row_scale = row_scale; a.bias = bias; a.relu = relu;
    a.out = out; a.ldo = ldo; a.out_absmax = out_absmax;
    return launch_spmm<MODE_COPY>(a, plan, (cudaStream_t)stream);
}

extern "C" int tango_spmm_u_mul_e_bias(const int32_t *indptr, const int32_t *indices, const int32_t *edge_ids,
                                       int64_t n_rows, const int8_t *nq, int64_t ldn, int h, int d, const int8_t *eq,
                                       const float *scale, const float *bias, float *out, int64_t ldo, const tango_spmm_plan *plan,
                                       tango_stream_t stream) {
    if (n_rows < 0 || h < 1 || d < 1) return TANGO_EINVAL;
    const int64_t f = (int64_t)h * d;
    if (ldn < f || ldo < f || f > (1 << 20)) return TANGO_EINVAL;
    if (n_rows == 0) return TANGO_OK;
    if (!indptr || !indices || !nq || !eq || !scale || !out) return TANGO_EINVAL;
    SpmmArgs a{};
    a.indptr = indptr; a.indices = indices; a.edge_ids = edge_ids; a.n_rows = n_rows; a.nseg = 1;
    a.feat = nq; a.ld = ldn; a.f = (int)f; a.ew = eq; a.H = h; a.D = d;
    a.scales = scale; a.bias = bias; a.out = out; a.ldo = ldo;
    return launch_spmm<MODE_WEIGHT_LANE>(a, plan, (cudaStream_t)stream);
}

extern "C" int tango_spmm_u_mul_e(const int32_t *indptr, const int32_t *indices, const int32_t *edge_ids,
                                  int64_t n_rows, const int8_t *nq, int64_t ldn, int h, int d, const int8_t *eq,
                                  const float *scale, float *out, int64_t ldo, const tango_spmm_plan *plan,
                                  tango_stream_t stream) {
    return tango_spmm_u_mul_e_bias(indptr, indices, edge_ids, n_rows, nq, ldn, h, d, eq, scale, nullptr, out, ldo, plan, stream);
}

extern "C" int tango_spmm_incidence(const int32_t *indptr, const int32_t *edge_ids, int64_t n_rows, const int8_t *zq,
                                    int64_t ldz, int64_t f, const float *scale, float *out, int64_t ldo,
                                    const tango_spmm_plan *plan, tango_stream_t stream) {
    if (n_rows < 0 || f < 0 || ldz < f || ldo < f || f > (1 << 20)) return TANGO_EINVAL;
    if (n_rows == 0 || f == 0) return TANGO_OK;
    if (!indptr || !zq || !scale || !out) return TANGO_EINVAL;
    SpmmArgs a{};
    a.indptr = indptr; a.indices = edge_ids; a.edge_ids = nullptr; a.n_rows = n_rows; a.nseg = 1;
    a.feat = zq; a.ld = ldz; a.f = (int)f; a.H = 1; a.D = (int)f;
    a.scales = scale; a.out = out; a.ldo = ldo;
    int rc = TANGO_OK;
    if (try_incidence(a, plan, (cudaStream_t)stream, rc)) return rc;
    return launch_spmm<MODE_COPY>(a, plan, (cudaStream_t)stream);
}
