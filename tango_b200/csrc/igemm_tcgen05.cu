// int8 x int8 -> int32 GEMMs for the quantized linear layer on sm_100a:
// tcgen05.mma kind::i8 (M=128, N<=256, K=32 per instruction), operands staged in shared memory by TMA with the
// 128-byte swizzle, accumulators in tensor memory, read back with tcgen05.ld for the dequantising epilogue.
//
// One kernel serves the three products of the layer by choosing the operand "major" per call:
//   forward  Y [M,N]  = Xq[M,K]  . Wq[N,K]^T   A K-major,  B K-major
//   dX       dX[M,K]  = dYq[M,N] . Wq[N,K]     A K-major,  B MN-major (reduction index is the row of Wq)
//   dW       dW[N,K]  = dYq^T    . Xq[M,K]     A MN-major, B MN-major, split over the long reduction (M) with
//                                              int32 atomics into scratch; the CTA that completes a tile dequantises
//                                              it (callers with uncleared scratch: a small kernel does).
// so no transposed copies of the quantized tensors are ever written.
//
// One persistent kernel, one CTA of 18 warps per SM: warp 0 issues TMA loads, warp 1 owns tensor memory and issues the
// MMAs (one lane), warps 2-17 run the epilogue.  A CTA walks a static list of work items (output tiles, slices of the
// reduction of an output tile, or runs of stored hub tiles) and alternates between two TMEM accumulators, so that the
// epilogue of one item overlaps the loads and MMAs of the next.  B either stays resident in shared memory (one N-tile of
// it, all of K: the forward and dX products of layers up to a few hundred features wide) or streams through the ring
// beside A, from L2, where the CTAs that share an A tile run side by side.
//
// What bounds it: the fp32 output.  At 232,965 x 602 x 256 the forward moves 140 MB of A and 239 MB of Y (58 us at the
// measured HBM rate), dX 561 MB of output.  Earlier epilogues -- 64-byte boxes handed to the bulk-store engine, or 64-byte
// row pieces for pitches that are no multiple of 16 bytes -- took 112 and 351 us; the engine and the L2 work per row piece.
// A lane now stores 256 bits of its own row per instruction (whole 32-byte sectors, no staging, no fences), and other
// pitches go out as 128 contiguous bytes of a row per warp.
// Every mbarrier wait is bounded: after ~2 s without progress the kernel records TANGO_ETIMEOUT in the status word,
// lets outstanding copies land, frees its tensor memory and returns.
#include <cuda.h>

#include <mutex>

#include "common.cuh"

namespace tango {

constexpr int kBlockK = 128;          // bytes of reduction per pipeline stage
constexpr int kTileM = 128;           // UMMA M
constexpr int kABytes = kTileM * kBlockK;  // 16 KiB either major
constexpr int kMaxStages = 8;
constexpr uint64_t kWaitTimeoutNs = 2000000000ull;

constexpr int kEpilogueWarps = 16;
constexpr int kGemmThreads = 32 * (2 + kEpilogueWarps);
constexpr int kStageWords = 32 * 32;  // one epilogue warp's staging tile

// STORE: dequantise and store fp32.  ADD: int32 partial sums into ws with atomics.  SPLIT: the same, and the CTA that
// completes an output tile dequantises it.
enum { MODE_STORE = 0, MODE_ADD = 1, MODE_SPLIT = 2 };

struct GemmParams {
    int M, N, K;     // D is [M, N], reduction length K
    int n_tile;      // UMMA N: multiple of 16, <= 256
    int m_tiles, n_tiles, splits, n_work;
    int kb_total;    // ceil(K / 128)
    int kb_per_split;
    int a_mn, b_mn;  // 1 = the operand is stored with the reduction index as its row (MN-major)
    int b_boxes;     // MN-major B: number of 128-column TMA boxes per k block; K-major: 1
    int b_bytes;     // bytes of B per k block
    int one_item;    // no CTA has more than one work item
    int b_resident;  // one N-tile of B (blockIdx.y) stays in shared memory
    int stages;
    int mode;
    float *out;
    int64_t ldo;
    int32_t *ws;
    int64_t ldws;
    int *arrivals;   // SPLIT: one counter per output tile
    const float *sa, *sb, *bias;
    const float *out_row_scale;     // optional: output row r is multiplied by out_row_scale[r] after dequantisation
    int relu;
    float *absmax;                  // optional: receives max|output * absmax_row_scale[r]| / 127
    const float *absmax_row_scale;  // optional
    int *status;
    uint32_t tmem_cols;
    int wide_store;                 // output rows start on 32-byte boundaries and are whole sectors
    int pairs;                      // else: rows start on 8-byte boundaries and have an even number of columns
    int line_ld;                    // row pitch (words) of the tile of output lines in shared memory
    const int4 *tile_units;   // work item x = (row tile, first stored A tile, first k block, k blocks)
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when the wait was abandoned (timeout here or abort raised by another role).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    // hand-offs between the roles are short (a pipeline stage): poll for a while before starting to sleep
#pragma unroll 1
    for (int i = 0; i < 4096; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
#pragma unroll 1
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_timer_ns() - t0 > kWaitTimeoutNs) {
            *abort_flag = 1;
            return false;
        }
        __nanosleep(64);
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1 (sm_100).
// Bits [0,14) start address >> 4, [16,30) leading byte offset >> 4, [32,46) stride byte offset >> 4,
// [46,48) version, [61,64) layout type (2 = 128-byte swizzle).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 consecutive accumulator columns of the warp's 32 tensor-memory lanes: lane = row, register = column.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
          "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- one 32 x 32 chunk of an accumulator: lane = row, register = column, `width` columns exist
// 16-byte piece j of row `lane` goes to piece j ^ (lane & 7) of the staging tile: conflict-free both ways.
__device__ __forceinline__ void stage_chunk(uint32_t *tile, const uint32_t (&r)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4 *>(tile + lane * 32 + ((j ^ (lane & 7)) << 2)) =
            make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
    __syncwarp();
}
__device__ __forceinline__ const uint32_t *staged(const uint32_t *tile, int row, int col) {
    return tile + row * 32 + ((((col >> 2) ^ (row & 7)) << 2) | (col & 3));
}

// int32 partial sums into the scratch matrix: 32 neighbouring words of one row per step.
__device__ __forceinline__ void add_chunk(const GemmParams &p, const uint32_t (&r)[32], uint32_t *tile, int row0, int col0,
                                          int width) {
    const int lane = threadIdx.x & 31, n_rows = min(32, p.M - row0);
    stage_chunk(tile, r);
    if (lane < width) {
        int32_t *o = p.ws + (int64_t)row0 * p.ldws + col0 + lane;
#pragma unroll 8
        for (int rr = 0; rr < n_rows; ++rr, o += p.ldws) {
            const int v = (int)*staged(tile, rr, lane);
            if (v != 0) atomicAdd(o, v);
        }
    }
    __syncwarp();
}

// max(v, 0) that hands a NaN on, in one instruction (a compare and select in its place cost the plain form of the epilogue,
// which never runs it, 8 %: dX of 232,965 x 602 166 -> 180 us).
__device__ __forceinline__ float relu_nan(float v) {
    float t;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(t) : "f"(v));
    return t;
}

// Dequantise and store.  An epilogue warp is a dependent chain with few companions, so instructions count: the optional
// steps are compiled out of the plain form, and where the rows of the output start on 32-byte boundaries every lane stores
// its own row's chunk with four 256-bit stores.  Rows of any other pitch are laid out in shared memory first (`line_tile`,
// row pitch p.line_ld): see store_lines.
template <bool PLAIN>
__device__ __forceinline__ void store_chunk(const GemmParams &p, uint32_t (&r)[32], uint32_t *line_row, int row0, int col0,
                                            int width, float sc, float &amax) {
    const int lane = threadIdx.x & 31, row = row0 + lane;
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__fmul_rn((float)(int)r[i], sc));
    if (!PLAIN) {
        if (p.out_row_scale) {
            const float rs = row < p.M ? __ldg(p.out_row_scale + row) : 1.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__fmul_rn(__uint_as_float(r[i]), rs));
        }
        if (p.bias) {
            const float mine = __ldg(p.bias + min(col0 + lane, p.N - 1));
#pragma unroll
            for (int i = 0; i < 32; ++i)
                r[i] = __float_as_uint(__fadd_rn(__uint_as_float(r[i]), __shfl_sync(0xffffffffu, mine, i)));
        }
        if (p.relu) {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(relu_nan(__uint_as_float(r[i])));
        }
        if (p.absmax) {
            float m = 0.f;
            if (width == 32) {
#pragma unroll
                for (int i = 0; i < 32; ++i) m = fmaxf(m, fabsf(__uint_as_float(r[i])));
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) m = i < width ? fmaxf(m, fabsf(__uint_as_float(r[i]))) : m;
            }
            // rounding is monotonic: the largest product is the product of the largest value
            const float f = row < p.M ? (p.absmax_row_scale ? fabsf(__ldg(p.absmax_row_scale + row)) : 1.f) : 0.f;
            amax = fmaxf(amax, __fmul_rn(m, f));
        }
    }
    if (p.wide_store) {
        if (row < p.M) {
            float *o = p.out + (int64_t)row * p.ldo + col0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (8 * i < width) store_v8(o + 8 * i, r + 8 * i);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)          // (line_ld / 4 is odd: conflict-free)
            *reinterpret_cast<uint4 *>(line_row + 4 * j) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
    }
}

// The four warps of a 32-row quarter write its rows, each as the 128-byte lines it covers: a store instruction fills one
// line, and only the first and last sector of a row's stretch are written in part.  (2408-byte rows, 561 MB: writing the
// chunks one by one, two partial sectors in every five, took 246 us against 150 us for the same columns at a 2432-byte pitch,
// although the arithmetic alone takes 96 us.)
// V = float2 halves the instructions where rows and columns come in pairs.
template <class V>
__device__ __forceinline__ void store_lines(const GemmParams &p, const uint32_t *quarter, int group, int row0, int n0, int cols) {
    constexpr int kPer = sizeof(V) / 4;
    const int lane = threadIdx.x & 31, r0 = row0 + group * 8, n_rows = min(8, p.M - r0);
    if (n_rows <= 0) return;
    // row i's columns, shifted so that lane 0 of a step is at a line boundary: eight rows side by side hide each other's
    // shared-memory latency
    float *o[8];
    int c[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        o[i] = p.out + (int64_t)(r0 + i) * p.ldo + n0;
        c[i] = i < n_rows ? kPer * lane - ((int)(reinterpret_cast<uintptr_t>(o[i]) >> 2) & 31) : 1 << 30;
    }
    const uint32_t *t = quarter + group * 8 * p.line_ld;
    for (int j = 0; j < cols + 31; j += 32 * kPer) {
        V v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = (unsigned)(c[i] + j) < (unsigned)cols ? *reinterpret_cast<const V *>(t + i * p.line_ld + c[i] + j) : V();
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if ((unsigned)(c[i] + j) < (unsigned)cols) *reinterpret_cast<V *>(o[i] + c[i] + j) = v[i];
    }
}

// Whether every epilogue warp's (bounded) wait succeeded: the warps that meet again below must leave together.
__device__ __forceinline__ bool all_epilogue_warps(bool ok) {
    int all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 1, %2, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((int)ok), "n"(kEpilogueWarps * 32)
        : "memory");
    return all != 0;
}

// Work item w of a launch: an output tile, or one slice of the reduction of an output tile, or one run of stored hub tiles.
struct Work {
    int m0, n0, kb0, n_kb, a_tile;   // a_tile >= 0: the A tiles are stored one after the other, starting with that one
    int tile;                        // index of the output tile (for the arrival counters)
};
__device__ __forceinline__ Work work_item(const GemmParams &p, int w) {
    Work k;
    const int nt = p.b_resident ? blockIdx.y : w % p.n_tiles, rest = p.b_resident ? w : w / p.n_tiles;
    k.n0 = nt * p.n_tile;
    if (p.tile_units) {
        const int4 u = __ldg(p.tile_units + rest);
        k.m0 = u.x * kTileM; k.a_tile = u.y; k.kb0 = u.z; k.n_kb = u.w; k.tile = 0;
    } else {
        const int mt = rest % p.m_tiles, split = rest / p.m_tiles;
        k.m0 = mt * kTileM; k.a_tile = -1; k.kb0 = split * p.kb_per_split;
        k.n_kb = min(p.kb_total, k.kb0 + p.kb_per_split) - k.kb0;
        k.tile = mt * p.n_tiles + nt;
    }
    return k;
}

__global__ void __launch_bounds__(kGemmThreads, 1)
igemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kMaxStages];
    __shared__ __align__(8) uint64_t bar_empty[kMaxStages];
    __shared__ __align__(8) uint64_t bar_b;
    __shared__ __align__(8) uint64_t bar_acc_full[2];
    __shared__ __align__(8) uint64_t bar_acc_empty[2];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort, s_last;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;      // the swizzle needs 1024-byte aligned tiles
    const uint32_t b_base = smem_base;                                     // resident B, if any
    const uint32_t ring = b_base + (p.b_resident ? (uint32_t)p.kb_total * p.b_bytes : 0u);
    const uint32_t stage_bytes = kABytes + (p.b_resident ? 0u : (uint32_t)p.b_bytes);
    // epilogue staging; a CTA with one work item re-uses the ring, which is idle once its accumulator is complete
    const uint32_t st_off = ring - smem_u32(smem_raw) + (p.one_item ? 0u : p.stages * stage_bytes);
    const uint32_t acc_cols = p.tmem_cols >> 1;                            // two accumulators side by side

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_b), 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bar_acc_full[b]), 1);
            mbar_init(smem_u32(&bar_acc_empty[b]), kEpilogueWarps);        // one arrival per epilogue warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                     "r"(p.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = s_tmem_base;
    volatile int *abort_flag = &s_abort;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_a) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_b) : "memory");
            const auto load_b = [&](uint32_t dst, uint32_t bar, int n0, int kb) {
                if (!p.b_mn) {
                    tma_load_2d(dst, &tm_b, bar, kb * kBlockK, n0);
                } else {
                    for (int j = 0; j < p.b_boxes; ++j) tma_load_2d(dst + j * kABytes, &tm_b, bar, n0 + j * 128, kb * kBlockK);
                }
            };
            if (p.b_resident) {
                mbar_expect_tx(smem_u32(&bar_b), (uint32_t)p.kb_total * p.b_bytes);
                for (int kb = 0; kb < p.kb_total; ++kb)
                    load_b(b_base + kb * p.b_bytes, smem_u32(&bar_b), blockIdx.y * p.n_tile, kb);
            }
            int it = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < p.n_work && ok; w += gridDim.x) {
                const Work k = work_item(p, w);
                for (int i = 0; i < k.n_kb; ++i, ++it) {
                    const int s = it % p.stages;
                    if (!mbar_wait(smem_u32(&bar_empty[s]), ((uint32_t)(it / p.stages) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                    const uint32_t full = smem_u32(&bar_full[s]), a_dst = ring + s * stage_bytes;
                    const int kc = (k.kb0 + i) * kBlockK;
                    mbar_expect_tx(full, stage_bytes);
                    if (k.a_tile >= 0) tma_load_2d(a_dst, &tm_a, full, 0, (k.a_tile + i) * kTileM);
                    else if (!p.a_mn) tma_load_2d(a_dst, &tm_a, full, kc, k.m0);
                    else tma_load_2d(a_dst, &tm_a, full, k.m0, kc);
                    if (!p.b_resident) load_b(a_dst + kABytes, full, k.n0, k.kb0 + i);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            // Instruction descriptor: D = s32 (bits 4-5 = 2), A and B signed int8 (bits 7-9, 10-12 = 1),
            // operand majors (bits 15, 16), N >> 3 (bits 17-22), M >> 4 (bits 24-28).
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)p.a_mn << 15) |
                                   ((uint32_t)p.b_mn << 16) | ((uint32_t)(p.n_tile >> 3) << 17) |
                                   ((uint32_t)(kTileM >> 4) << 24);
            const uint32_t a_kstep = p.a_mn ? 32u * 128u : 32u, b_kstep = p.b_mn ? 32u * 128u : 32u;   // bytes per K=32 step
            const uint32_t a_lbo = p.a_mn ? (uint32_t)kABytes : 16u, b_lbo = p.b_mn ? (uint32_t)kABytes : 16u;
            bool ok = true;
            if (p.b_resident) ok = mbar_wait(smem_u32(&bar_b), 0u, abort_flag);
            int it = 0, t = 0;
            for (int w = blockIdx.x; w < p.n_work && ok; w += gridDim.x, ++t) {
                const Work k = work_item(p, w);
                const int buf = t & 1;
                if (!mbar_wait(smem_u32(&bar_acc_empty[buf]), ((uint32_t)(t >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tmem_d = tmem_base + buf * acc_cols;
                for (int i = 0; i < k.n_kb; ++i, ++it) {
                    const int s = it % p.stages, kb = k.kb0 + i;
                    if (!mbar_wait(smem_u32(&bar_full[s]), (uint32_t)(it / p.stages) & 1u, abort_flag)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_src = ring + s * stage_bytes;
                    const uint32_t b_src = p.b_resident ? b_base + kb * p.b_bytes : a_src + kABytes;
                    const int nk = min(4, (p.K - kb * kBlockK + 31) >> 5);
                    for (int q = 0; q < nk; ++q)
                        umma_i8(tmem_d, make_smem_desc(a_src + q * a_kstep, a_lbo, 1024u),
                                make_smem_desc(b_src + q * b_kstep, b_lbo, 1024u), idesc, (i > 0 || q > 0) ? 1u : 0u);
                    umma_commit(smem_u32(&bar_empty[s]));   // frees the stage once the MMAs above have read it
                }
                if (ok) umma_commit(smem_u32(&bar_acc_full[buf]));   // accumulator complete
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue (warps 2..17)
        // Warp w reads the 32 tensor-memory lanes 32 * (w % 4).. it may access and a quarter of the 32-column chunks.
        const int q = warp & 3, group = (warp - 2) >> 2;
        uint32_t *staging = reinterpret_cast<uint32_t *>(smem_raw + st_off), *tile = staging + (warp - 2) * kStageWords;
        const bool lines = p.mode == MODE_STORE && !p.wide_store;
        uint32_t *quarter = staging + q * 32 * p.line_ld;
        const bool want_max = p.absmax != nullptr;
        const bool plain = !p.out_row_scale && !p.bias && !p.relu && !want_max;
        const float sc = p.sa ? __fmul_rn(__ldg(p.sa), __ldg(p.sb)) : 0.f;
        float amax = 0.f;
        int t = 0;
        for (int w = blockIdx.x; w < p.n_work; w += gridDim.x, ++t) {
            const Work k = work_item(p, w);
            const int buf = t & 1;
            bool ok = mbar_wait(smem_u32(&bar_acc_full[buf]), (uint32_t)(t >> 1) & 1u, abort_flag);
            ok = p.mode == MODE_SPLIT || lines ? all_epilogue_warps(ok) : __all_sync(0xffffffffu, ok) != 0;
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row0 = k.m0 + q * 32;
            const uint32_t tbase = tmem_base + buf * acc_cols + ((uint32_t)(q * 32) << 16);
            const int end = min(p.n_tile, p.N - k.n0), per = ((p.n_tile + 127) >> 7) * 32;   // a stretch of whole chunks
            const int c_beg = group * per, c_end = min(end, c_beg + per);
            for (int c0 = c_beg; c0 < c_end; c0 += 32) {
                const int col0 = k.n0 + c0, width = min(32, c_end - c0);
                uint32_t r[32];
                tmem_ld32(tbase + (uint32_t)c0, r);
                if (p.mode != MODE_STORE) add_chunk(p, r, tile, row0, col0, width);
                else if (plain) store_chunk<true>(p, r, quarter + lane * p.line_ld + c0, row0, col0, width, sc, amax);
                else store_chunk<false>(p, r, quarter + lane * p.line_ld + c0, row0, col0, width, sc, amax);
            }
            // this warp has read its share of the accumulator: hand the buffer back to the MMA issuer
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar_acc_empty[buf])) : "memory");
            if (lines) {
                asm volatile("bar.sync %0, 128;" ::"r"(2 + q) : "memory");
                if (p.pairs) store_lines<float2>(p, quarter, group, row0, k.n0, end);
                else store_lines<float>(p, quarter, group, row0, k.n0, end);
                asm volatile("bar.sync %0, 128;" ::"r"(2 + q) : "memory");
            }
            if (p.mode == MODE_SPLIT) {
                // the CTA that adds the last slice of an output tile turns the finished sums into fp32
                __threadfence();
                asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueWarps * 32) : "memory");
                if (threadIdx.x == 64) s_last = atomicAdd(p.arrivals + k.tile, 1) == p.splits - 1;
                asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueWarps * 32) : "memory");
                if (s_last) {
                    __threadfence();
                    const int n_cols = min(p.n_tile, p.N - k.n0), n_rows = min(kTileM, p.M - k.m0);
                    for (int rr = warp - 2; rr < n_rows; rr += kEpilogueWarps)
                        for (int c = lane; c < n_cols; c += 32) {
                            const int64_t at = (int64_t)(k.m0 + rr);
                            const int v = __ldcg(p.ws + at * p.ldws + k.n0 + c);
                            p.out[at * p.ldo + k.n0 + c] = __fmul_rn((float)v, sc);
                        }
                }
            }
        }
        if (want_max) {
            amax = warp_max(amax);
            if (lane == 0 && amax > 0.f) {
                const float s = __fdiv_rn(amax, 127.0f);
                if (s > __ldcg(p.absmax)) atomic_max_nonneg(p.absmax, s);
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (s_abort) {
        // give copies that are still in flight time to land before the CTA's shared memory is released
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
        if (threadIdx.x == 0 && p.status) atomicExch(p.status, TANGO_ETIMEOUT);
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols)
                     : "memory");
    }
}

__global__ void __launch_bounds__(256) dequant_ws_kernel(const int32_t *__restrict__ ws, int64_t ldws, int64_t rows,
                                                         int64_t cols, const float *__restrict__ sa,
                                                         const float *__restrict__ sb, float *__restrict__ out,
                                                         int64_t ldo) {
    const float sc = __fmul_rn(__ldg(sa), __ldg(sb));
    const int64_t total = rows * cols;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / cols, c = i - r * cols;
        out[r * ldo + c] = __fmul_rn((float)ws[r * ldws + c], sc);
    }
}

// ------------------------------------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;  // benign race: every thread resolves the same pointer
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &qres) ==
                cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// 2-D uint8 tensor map over a row-major [outer, inner] byte matrix with leading dimension ld; 128-byte swizzle.
static int make_map(CUtensorMap *map, const void *base, int64_t inner, int64_t outer, int64_t ld, int box_inner,
                    int box_outer) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return TANGO_ECUDA;
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
    cuuint64_t strides[1] = {(cuuint64_t)ld};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda_error = (int)r;
        return TANGO_ECUDA;
    }
    return TANGO_OK;
}

struct GemmCall {
    const int8_t *a; int64_t lda; int a_mn;
    const int8_t *b; int64_t ldb; int b_mn;
    int64_t M, N, K;
    int mode; int splits;
    float *out; int64_t ldo; int32_t *ws; int64_t ldws; int *arrivals;
    const float *sa, *sb, *bias; float *absmax; int *status;
    const float *out_row_scale, *absmax_row_scale;
    int relu;
};

constexpr int kSmemBudget = 227 * 1024 - 2048;   // dynamic limit minus static barriers and alignment slack

// Tile shape, shared-memory layout, B's tensor map and the launch.  B: [rows, row bytes] with leading dimension ldb.
static int run_gemm(const CUtensorMap &tm_a, const int8_t *b, int64_t ldb, GemmParams &p, cudaStream_t stream) {
    // Shared memory beside the operands: one tile per epilogue warp for the atomics, a tile of output lines for rows that
    // 256-bit stores cannot take, nothing when a CTA has a single work item (its ring is idle by then).
    const int warp_tiles = kEpilogueWarps * kStageWords * 4;
    int gx;
    int64_t fit, stages, tile_bytes, b_all;
    for (p.n_tiles = (p.N + 255) / 256;; ++p.n_tiles) {
        p.n_tile = (int)round_up(ceil_div(p.N, p.n_tiles), 16);
        p.b_boxes = p.b_mn ? (int)ceil_div(p.n_tile, 128) : 1;
        p.b_bytes = p.b_mn ? p.b_boxes * kABytes : (int)round_up((int64_t)p.n_tile * kBlockK, 1024);
        p.line_ld = (int)round_up(p.n_tile, 32) + 4;
        const int64_t work = (int64_t)(p.tile_units ? p.n_work : p.m_tiles * (int64_t)p.splits) * p.n_tiles;
        if (work > 0x7fffffff) return TANGO_ESIZE;
        p.one_item = work <= kNumSMs;
        tile_bytes = p.mode != MODE_STORE ? warp_tiles : p.wide_store ? 0 : kTileM * p.line_ld * 4;
        const int64_t staging = p.one_item ? 0 : tile_bytes;
        b_all = (int64_t)p.kb_total * p.b_bytes;
        gx = kNumSMs / p.n_tiles < 1 ? 1 : kNumSMs / p.n_tiles;
        fit = (kSmemBudget - staging - b_all) / kABytes;
        stages = (kSmemBudget - staging) / (kABytes + p.b_bytes);
        if (fit >= 3 || stages >= 3 || p.n_tile <= 64) {      // narrower tiles only where a line tile leaves no room
            if (!p.tile_units) p.n_work = (int)work;
            else p.n_work *= p.n_tiles;
            break;
        }
    }
    const int64_t staging = p.one_item ? 0 : tile_bytes;
    // B stays in shared memory when one N-tile of it fits beside a ring of A tiles and a CTA has more than one tile to use
    // it on; else both operands stream (a single tile starts sooner that way)
    p.b_resident = p.mode == MODE_STORE && p.splits == 1 && !p.tile_units && !p.one_item && fit >= 3 && p.m_tiles > gx && p.n_tiles <= 65535;
    if (p.b_resident) stages = fit;
    if (stages > kMaxStages) stages = kMaxStages;
    if (stages < 2) return TANGO_ESIZE;
    p.stages = (int)stages;
    uint32_t cols = 32;
    while ((int)cols < p.n_tile) cols <<= 1;
    p.tmem_cols = cols * 2;
    size_t smem = 1024 + (p.b_resident ? (size_t)b_all + stages * kABytes : (size_t)stages * (kABytes + p.b_bytes)) + staging;
    if (smem < 1024 + (size_t)tile_bytes) smem = 1024 + (size_t)tile_bytes;
    dim3 grid;
    if (p.b_resident) {
        p.n_work = p.m_tiles;
        grid = dim3((unsigned)gx, (unsigned)p.n_tiles);
    } else {
        grid = dim3((unsigned)(p.n_work < kNumSMs ? p.n_work : kNumSMs));
    }
    // B: K-major [N rows, K bytes] box {128 k, n_tile};  MN-major [K rows, N bytes] boxes {128 n, 128 k}
    CUtensorMap tm_b;
    const int rc = p.b_mn ? make_map(&tm_b, b, p.N, p.K, ldb, 128, kBlockK) : make_map(&tm_b, b, p.K, p.N, ldb, kBlockK, p.n_tile);
    if (rc) return rc;
    // per-device attribute; setting it on every call keeps the entry point free of global state
    TANGO_CUDA_TRY(cudaFuncSetAttribute(igemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024));
    igemm_kernel<<<grid, kGemmThreads, smem, stream>>>(tm_a, tm_b, p);
    TANGO_LAUNCH_CHECK();
    return TANGO_OK;
}

static int launch_gemm(const GemmCall &c, cudaStream_t stream) {
    if (c.M <= 0 || c.N <= 0) return TANGO_OK;
    if (c.K <= 0) return TANGO_EINVAL;
    if (c.M > 0x7fffffff || c.N > 0x7fffffff || c.K > 0x7fffffff) return TANGO_ESIZE;
    if (!aligned(c.a, 16) || !aligned(c.b, 16) || c.lda % 16 || c.ldb % 16) return TANGO_EALIGN;
    GemmParams p{};
    p.M = (int)c.M; p.N = (int)c.N; p.K = (int)c.K;
    p.m_tiles = (int)ceil_div(c.M, kTileM);
    p.kb_total = (int)ceil_div(c.K, kBlockK);
    int splits = c.splits < 1 ? 1 : c.splits;
    if (splits > p.kb_total) splits = p.kb_total;
    p.kb_per_split = (int)ceil_div(p.kb_total, splits);
    p.splits = (int)ceil_div(p.kb_total, p.kb_per_split);
    p.a_mn = c.a_mn; p.b_mn = c.b_mn;
    p.mode = c.mode; p.out = c.out; p.ldo = c.ldo; p.ws = c.ws; p.ldws = c.ldws; p.arrivals = c.arrivals;
    p.sa = c.sa; p.sb = c.sb; p.bias = c.bias; p.absmax = c.absmax; p.status = c.status;
    p.out_row_scale = c.out_row_scale; p.absmax_row_scale = c.absmax_row_scale; p.relu = c.relu;
    p.wide_store = c.ldo % 8 == 0 && c.N % 8 == 0 && aligned(c.out, 32);
    p.pairs = c.ldo % 2 == 0 && c.N % 2 == 0 && aligned(c.out, 8);

    CUtensorMap tm_a;
    int rc;
    // A: K-major [M rows, K bytes] box {128 k, 128 m};  MN-major [K rows, M bytes] box {128 m, 128 k}
    if (!c.a_mn) rc = make_map(&tm_a, c.a, c.K, c.M, c.lda, kBlockK, kTileM);
    else rc = make_map(&tm_a, c.a, c.M, c.K, c.lda, 128, kBlockK);
    if (rc) return rc;
    return run_gemm(tm_a, c.b, c.ldb, p, stream);
}

int igemm_accumulate_tiles_i32(const int8_t *tiles, int64_t n_tiles, const int32_t *units, int64_t n_units,
                               const int8_t *b, int64_t ldb, int64_t m, int64_t n, int64_t k, int32_t *ws,
                               int64_t ldws, int *status, cudaStream_t stream) {
    if (n_units <= 0 || n <= 0) return TANGO_OK;
    if (m <= 0 || k <= 0 || n_tiles <= 0 || m % kTileM || k % kBlockK) return TANGO_EINVAL;
    if (m > 0x7fffffff || k > 0x7fffffff || n_tiles * kTileM > 0x7fffffff || n_units > 0x7fffffff) return TANGO_ESIZE;
    if (!aligned(tiles, 16) || !aligned(b, 16) || ldb % 16 || !aligned(units, 16)) return TANGO_EALIGN;
    GemmParams p{};
    p.M = (int)m; p.N = (int)n; p.K = (int)k;
    p.m_tiles = (int)(m / kTileM);
    p.kb_total = p.kb_per_split = (int)(k / kBlockK);
    p.splits = 1;
    p.n_work = (int)n_units;       // times the N-tiles that run_gemm decides on
    p.b_mn = 1;
    p.mode = MODE_ADD; p.ws = ws; p.ldws = ldws; p.status = status;
    p.tile_units = reinterpret_cast<const int4 *>(units);
    CUtensorMap tm_a;
    const int rc = make_map(&tm_a, tiles, kBlockK, n_tiles * kTileM, kBlockK, kBlockK, kTileM);   // one box = one stored tile
    if (rc) return rc;
    return run_gemm(tm_a, b, ldb, p, stream);
}

// Slices of the reduction of a weight gradient: as many as give every SM one work item.
static int dw_splits(int64_t m, int64_t n, int64_t k) {
    const int64_t tiles = ceil_div(n, kTileM) * ceil_div(k, 256);
    int64_t splits = kNumSMs / (tiles > 0 ? tiles : 1);
    if (splits > ceil_div(m, kBlockK)) splits = ceil_div(m, kBlockK);
    return (int)(splits < 1 ? 1 : splits);
}

}  // namespace tango

using namespace tango;

extern "C" int64_t tango_qgemm_dw_workspace_bytes(int64_t n, int64_t k) {
    if (n < 0 || k < 0) return 0;
    if (n == 0 || k == 0) return 0;
    // n * round_up(k, 4) * 4 must fit in int64: saturate instead of wrapping around
    if (k > INT64_MAX - 3) return INT64_MAX;
    const int64_t ldws = round_up(k, 4);
    if (n > INT64_MAX / 4 / ldws) return INT64_MAX;
    return n * ldws * (int64_t)sizeof(int32_t);
}

extern "C" int tango_qgemm_layer(const int8_t *xq, int64_t ldx, const int8_t *wq, int64_t ldw, int64_t m, int64_t n,
                                 int64_t k, const float *sx, const float *sw, const float *row_scale, const float *bias,
                                 int relu, float *y, int64_t ldy, float *scale_y, const float *scale_row_factor,
                                 int *status, tango_stream_t stream) {
    if (m < 0 || n < 0 || k <= 0 || ldx < k || ldw < k || ldy < n) return TANGO_EINVAL;
    if (m == 0 || n == 0) return TANGO_OK;
    if (!xq || !wq || !sx || !sw || !y) return TANGO_EINVAL;
    GemmCall c{};
    c.a = xq; c.lda = ldx; c.b = wq; c.ldb = ldw; c.M = m; c.N = n; c.K = k; c.mode = MODE_STORE; c.splits = 1;
    c.out = y; c.ldo = ldy; c.sa = sx; c.sb = sw; c.bias = bias; c.relu = relu; c.out_row_scale = row_scale;
    c.absmax = scale_y; c.absmax_row_scale = scale_row_factor; c.status = status;
    return launch_gemm(c, (cudaStream_t)stream);
}

extern "C" int tango_qgemm_nt(const int8_t *xq, int64_t ldx, const int8_t *wq, int64_t ldw, int64_t m, int64_t n,
                              int64_t k, const float *sx, const float *sw, const float *bias, float *y, int64_t ldy,
                              float *scale_y, int *status, tango_stream_t stream) {
    return tango_qgemm_layer(xq, ldx, wq, ldw, m, n, k, sx, sw, nullptr, bias, 0, y, ldy, scale_y, nullptr, status, stream);
}

extern "C" int tango_qgemm_forward(const float *x, int64_t ldx_f, const float *row_scale, const float *w,
                                   int64_t ldw_f, int64_t m, int64_t n, int64_t k, const float *sx, const float *sw,
                                   int8_t *xq, int64_t ldxq, int8_t *wq, int64_t ldwq, const float *bias, float *y,
                                   int64_t ldy, float *scale_y, int mode, uint64_t seed, uint64_t call,
                                   const uint64_t *step, int *status, tango_stream_t stream) {
    int rc = tango_quantize(x, m, k, ldx_f, row_scale, sx, xq, ldxq, mode, seed, call, step, stream);
    if (rc) return rc;
    rc = tango_quantize(w, n, k, ldw_f, nullptr, sw, wq, ldwq, mode, seed, call + 1, step, stream);
    if (rc) return rc;
    return tango_qgemm_nt(xq, ldxq, wq, ldwq, m, n, k, sx, sw, bias, y, ldy, scale_y, status, stream);
}

extern "C" int tango_qgemm_dx_layer(const int8_t *dyq, int64_t lddy, const int8_t *wq, int64_t ldw, int64_t m, int64_t n,
                                    int64_t k, const float *sdy, const float *sw, const float *row_scale, float *dx,
                                    int64_t lddx, float *scale_dx, int *status, tango_stream_t stream) {
    if (m < 0 || n <= 0 || k < 0 || lddy < n || ldw < k || lddx < k) return TANGO_EINVAL;
    if (m == 0 || k == 0) return TANGO_OK;
    if (!dyq || !wq || !sdy || !sw || !dx) return TANGO_EINVAL;
    // D[m, k] = A[m, n] . B[n, k]: reduction n; B is stored with the reduction index as its row
    GemmCall c{};
    c.a = dyq; c.lda = lddy; c.b = wq; c.ldb = ldw; c.b_mn = 1; c.M = m; c.N = k; c.K = n; c.mode = MODE_STORE; c.splits = 1;
    c.out = dx; c.ldo = lddx; c.sa = sdy; c.sb = sw; c.out_row_scale = row_scale; c.absmax = scale_dx; c.status = status;
    return launch_gemm(c, (cudaStream_t)stream);
}

extern "C" int tango_qgemm_dx(const int8_t *dyq, int64_t lddy, const int8_t *wq, int64_t ldw, int64_t m, int64_t n,
                              int64_t k, const float *sdy, const float *sw, const float *row_scale, float *dx,
                              int64_t lddx, int *status, tango_stream_t stream) {
    return tango_qgemm_dx_layer(dyq, lddy, wq, ldw, m, n, k, sdy, sw, row_scale, dx, lddx, nullptr, status, stream);
}

// D[n, k] = A[n, m] . B[m, k]: both operands are stored with the reduction index m as their row
static GemmCall dw_call(const int8_t *dyq, int64_t lddy, const int8_t *xq, int64_t ldx, int64_t m, int64_t n, int64_t k,
                        const float *sdy, const float *sx, int *status) {
    GemmCall c{};
    c.a = dyq; c.lda = lddy; c.a_mn = 1; c.b = xq; c.ldb = ldx; c.b_mn = 1; c.M = n; c.N = k; c.K = m;
    c.splits = dw_splits(m, n, k); c.sa = sdy; c.sb = sx; c.status = status;
    return c;
}

extern "C" int64_t tango_qgemm_dw_scratch_bytes(int64_t m, int64_t n, int64_t k) {
    if (m <= 0 || n <= 0 || k <= 0 || dw_splits(m, n, k) == 1) return 0;
    const int64_t sums = tango_qgemm_dw_workspace_bytes(n, k), tiles = ceil_div(n, kTileM) * ceil_div(k, 256);
    return sums > INT64_MAX - 4 * tiles ? INT64_MAX : sums + 4 * tiles;
}

extern "C" int tango_qgemm_dw_cleared(const int8_t *dyq, int64_t lddy, const int8_t *xq, int64_t ldx, int64_t m, int64_t n,
                                      int64_t k, const float *sdy, const float *sx, float *dw, int64_t lddw,
                                      void *scratch, int64_t scratch_bytes, int *status, tango_stream_t stream) {
    if (m <= 0 || n < 0 || k < 0 || lddy < n || ldx < k || lddw < k) return TANGO_EINVAL;
    if (n == 0 || k == 0) return TANGO_OK;
    if (!dyq || !xq || !sdy || !sx || !dw) return TANGO_EINVAL;
    const int64_t need = tango_qgemm_dw_scratch_bytes(m, n, k);
    if (scratch_bytes < need || (need > 0 && !scratch)) return TANGO_ESIZE;
    if (!aligned(scratch, 16)) return TANGO_EALIGN;
    GemmCall c = dw_call(dyq, lddy, xq, ldx, m, n, k, sdy, sx, status);
    c.mode = need > 0 ? MODE_SPLIT : MODE_STORE;
    c.out = dw; c.ldo = lddw;
    c.ws = static_cast<int32_t *>(scratch); c.ldws = round_up(k, 4);
    c.arrivals = c.ws + n * c.ldws;
    return launch_gemm(c, (cudaStream_t)stream);
}

extern "C" int tango_qgemm_dw(const int8_t *dyq, int64_t lddy, const int8_t *xq, int64_t ldx, int64_t m, int64_t n,
                              int64_t k, const float *sdy, const float *sx, float *dw, int64_t lddw, void *workspace,
                              int64_t workspace_bytes, int *status, tango_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (m <= 0 || n < 0 || k < 0 || lddy < n || ldx < k || lddw < k) return TANGO_EINVAL;
    if (n == 0 || k == 0) return TANGO_OK;
    if (!dyq || !xq || !sdy || !sx || !dw || !workspace) return TANGO_EINVAL;
    if (workspace_bytes < tango_qgemm_dw_workspace_bytes(n, k)) return TANGO_ESIZE;
    if (!aligned(workspace, 16)) return TANGO_EALIGN;
    const int64_t ldws = round_up(k, 4);
    TANGO_CUDA_TRY(cudaMemsetAsync(workspace, 0, (size_t)(n * ldws) * sizeof(int32_t), stream));
    GemmCall c = dw_call(dyq, lddy, xq, ldx, m, n, k, sdy, sx, status);
    c.mode = MODE_ADD; c.ws = (int32_t *)workspace; c.ldws = ldws;
    int rc = launch_gemm(c, stream);
    if (rc) return rc;
    int64_t blocks = ceil_div(n * k, 256);
    if (blocks > kNumSMs * 8) blocks = kNumSMs * 8;
    dequant_ws_kernel<<<(unsigned)blocks, 256, 0, stream>>>((const int32_t *)workspace, ldws, n, k, sdy, sx, dw, lddw);
    TANGO_LAUNCH_CHECK();
    return TANGO_OK;
}

// ------------------------------------------------------------------------------------------------ no-allocation dW
// Scratch for tango_qgemm_dw_noalloc: a fixed array inside the library image instead of caller-provided memory.
// Every GPU that loads the library keeps these 4 MiB until the process exits.
namespace tango {
constexpr int64_t kStaticDwScratchElems = 1 << 20;  // int32 elements: n * round_up(k, 4) must not exceed this
static __device__ __align__(256) int32_t g_dw_scratch[kStaticDwScratchElems];

constexpr int kMaxDevices = 64;
static std::mutex g_dw_scratch_mutex;
static void *g_dw_scratch_ptr[kMaxDevices] = {nullptr};

// Device address of g_dw_scratch on the current device.  In host code the array's name is only a handle, so the
// address is looked up once per device (with that device current) and cached.
static int dw_scratch_address(void **out) {
    int dev = -1;
    TANGO_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return TANGO_ESIZE;
    std::lock_guard<std::mutex> lock(g_dw_scratch_mutex);
    if (!g_dw_scratch_ptr[dev]) {
        void *p = nullptr;
        TANGO_CUDA_TRY(cudaGetSymbolAddress(&p, g_dw_scratch));
        if (!p) return TANGO_ECUDA;
        g_dw_scratch_ptr[dev] = p;
    }
    *out = g_dw_scratch_ptr[dev];
    return TANGO_OK;
}
}  // namespace tango

extern "C" int64_t tango_qgemm_dw_noalloc_max_elems(void) { return tango::kStaticDwScratchElems; }

extern "C" int tango_qgemm_dw_noalloc(const int8_t *dyq, int64_t lddy, const int8_t *xq, int64_t ldx, int64_t m,
                                      int64_t n, int64_t k, const float *sdy, const float *sx, float *dw,
                                      int64_t lddw, int *status, tango_stream_t stream) {
    if (n < 0 || k < 0) return TANGO_EINVAL;
    // compared in elements and by division, so that no product of caller-given sizes can wrap around
    if (k > tango::kStaticDwScratchElems) return TANGO_ESIZE;
    if (n > 0 && k > 0 && n > tango::kStaticDwScratchElems / round_up(k, 4)) return TANGO_ESIZE;
    void *scratch = nullptr;
    const int rc = tango::dw_scratch_address(&scratch);
    if (rc) return rc;
    // The regular entry point clears the part of the scratch it uses before accumulating into it.
    return tango_qgemm_dw(dyq, lddy, xq, ldx, m, n, k, sdy, sx, dw, lddw, scratch,
                          tango::kStaticDwScratchElems * (int64_t)sizeof(int32_t), status, stream);
}
