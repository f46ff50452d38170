// Products of the true 32-bit path on the fifth-generation tensor cores, for inner sizes from TC_MIN_K up.
//
//   C[t, n] = A[t, :] . W[n, :]   (dense, one of several independent products, or an expert's rows of a grouped one)
//
// A number x of 32 bits is taken as hi + lo: hi is x rounded to 11 bits of mantissa, lo = x - hi (exact, at most 2^-11 of x) is
// read to 11 bits, both operands of kind::tf32, and a product is hi hi + hi lo + lo hi.  What is left out, lo lo and lo's
// last bits, is at most 3 * 2^-21 of a term (on average a tenth of that) and of either sign; the tensor cores add without rounding to nearest, so 32 terms at most are added there (first the small products,
// then hi hi) and every such sum goes through registers, where it is added in 32 bits as any number is.  Against 64 bits the
// result is nearer than a chain of K fused multiply-adds, from K = 512 on (measured, relative to the result's norm, chain and
// here: see dense_f32.cu).
//
// Every output element is the same sums in the same order in every form below: chunks of 32 k in ascending order within
// each of four parts of the inner dimension, then the parts in ascending order.  So a row has the same bits however many
// rows share the step, in whichever tile and form, as the chains of the CUDA-core kernels have for smaller K.  A result that
// is not finite (an operand that is not, or a sum that overflows) is computed again as a chain of multiply-adds, so infinities and
// NaN reach exactly the elements that they reach there.
//
// Weights are the M operand (128 rows a tile; 64 gate rows and the up rows of the same outputs in a paired product) and lie in
// tensor memory, rows of activations are the N operand in shared memory.  Roles:
//   warps 0-3 and 4-7, chunks in turn: weights, ring -> hi and lo -> tensor memory
//   warps 8-15  the sums of a chunk: tensor memory -> registers, added up
//   warps 16, 17, chunks in turn: MMAs (12 a chunk; the tensor cores take them one by one as they come, so a single warp
//               would leave them idle while it waits for the next chunk's operands); warp 16 allocates tensor memory
//   warp 18     weights: memory -> ring (TMA; without it, where rows are not aligned for it, the warps that read them ask
//               for them with cp.async)
//   tiles of 64 and 128 rows: warp 19 brings hi and lo of the activations, which f32_split_rows_kernel has made (TMA)
//   tiles of 16 and 32: warps 19-22 bring the activations (cp.async, four chunks ahead) and make hi and lo of them in shared memory
// What bounds a chunk of a tile of 64 or 128 is shared memory: weights written and read, activations written, and read by
// every MMA.
// SPLIT: a cluster of 2 or 4 blocks shares a tile's parts and adds them up through distributed shared memory, where tiles
// alone would leave SMs without work (a decode step's few rows).
//
// Every wait on an mbarrier is bounded: one that runs out sets the status word, and all roles fall through to the exit.
#pragma once

#include "tcgen05.cuh"

namespace mi {
namespace f32tc {

using namespace tc;

constexpr int TC_MIN_K = 512;
constexpr int FK = 32;                                 // k per chunk: 32 floats are a swizzled row of 128 bytes
constexpr int PARTS = 4;
constexpr int OUT_WARP = 8, MMA_WARP = 16, W_WARP = 18, ROWS_WARP = 19;        // first warps of the roles
constexpr bool split_before(int nt) { return nt >= 64; }
constexpr int threads(int nt) { return 32 * (split_before(nt) ? 20 : 23); }
constexpr int T_SLOTS = 4, ROWS_AHEAD = 4;             // chunks of weights in tensor memory; of activations asked for
constexpr uint32_t SLOT_LIMIT = 65536;                 // bytes of part sums of a SPLIT block
// D float32, A and B tf32, both K-major, M = 128 (without N)
constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((128u >> 4) << 24);

// Rings, in chunks: weights; hi and lo of the activations (at most four: see the phases below; hi also holds what is on its
// way where the block splits it itself); sums in tensor memory
constexpr int w_slots(int nt, bool split) { return nt == 128 ? 4 : (nt == 64 ? 6 : 8) - (split ? 2 : 0); }
constexpr int lo_slots(int nt) { return nt == 128 ? 3 : 4; }
constexpr int hi_slots(int nt) { return split_before(nt) ? lo_slots(nt) : lo_slots(nt) + ROWS_AHEAD; }
constexpr int d_slots(int nt) { return nt == 128 ? 2 : 4; }
inline size_t smem_bytes(int nt, int split) {
    return 1024 + (size_t)w_slots(nt, split > 1) * 16384 + (size_t)(hi_slots(nt) + lo_slots(nt)) * nt * 128 +
           (size_t)(split > 1 ? PARTS / split : 1) * nt * 512;
}

// mbar_wait of tcgen05.cuh, by a whole warp
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
    bool there = false;
    for (uint32_t i = 0; i < WAIT_LIMIT && !there; ++i) {
        there = __all_sync(0xffffffffu, mbar_try_wait(bar, parity));
        if (!there && *abort_flag) return false;
    }
    if (!there) *abort_flag = code;
    return there;
}

struct Problem {
    const float* A; const float* W; float* C;
    const int* gather;                                 // grouped: row of A of a sorted row (or null)
    const int* offsets;                                // grouped: [E + 1]; dense: null
    int T, N, K, lda, ldc, E;                          // N: outputs (a paired product has 2 N rows of W an expert)
    int64_t sA, sW, sC;                                // dense: operands of product blockIdx.z
    int64_t split_rows;                                // rows of `hi` (those of `lo` come behind them), of products in turn
    GluForm glu;
    int* status;
};
struct RowMaps { CUtensorMap m[4]; };                  // hi and lo of the activations in boxes of 16, 32, 48 and 64 rows

__device__ __forceinline__ void umma_tf32_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void wait_tmem_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// hi and lo of x as operands of kind::tf32, which reads their upper 19 bits.  (x + 0x1000 may carry a NaN's bits into the sign:
// then lo is the NaN.)
__device__ __forceinline__ void split(uint32_t x, uint32_t& hi, uint32_t& lo) {
    hi = (x + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(__uint_as_float(x) - __uint_as_float(hi));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const char* src, bool there) {
    const int n = there ? 16 : 0;                      // nothing read: the bytes become zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool there) {
    const int n = there ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.402823466e38f); }

// an element once more, as the CUDA-core kernels compute it
__device__ __noinline__ float chain(const float* __restrict__ a, const float* __restrict__ w, int K) {
    float s = 0.f;
    for (int k = 0; k < K; ++k) s = fmaf(a[k], w[k], s);
    return s;
}

// An expert's rows are split evenly over its tiles of up to `nt` rows, whole groups of 16.  Uniform for the warp.
__device__ __forceinline__ int row_tile(const int* __restrict__ offsets, int E, int nt, int slot, int& e, int& row0) {
    const int lane = threadIdx.x & 31;
    for (int base = 0; base < E; base += 32) {
        const int i = base + lane;
        const int lo = i < E ? __ldg(offsets + i) : 0, cnt = i < E ? __ldg(offsets + i + 1) - lo : 0;
        const int own = (cnt + nt - 1) / nt;
        int through = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, through, d);
            if (lane >= d) through += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, through > slot);
        if (hit) {
            const int who = __ffs(hit) - 1;
            const int at = slot - __shfl_sync(0xffffffffu, through - own, who);
            const int n = __shfl_sync(0xffffffffu, cnt, who), tiles = __shfl_sync(0xffffffffu, own, who);
            const int per = ((n + tiles - 1) / tiles + 15) & ~15;
            e = base + who;
            row0 = __shfl_sync(0xffffffffu, lo, who) + at * per;
            return max(0, min(per, n - at * per));
        }
        slot -= __shfl_sync(0xffffffffu, through, 31);
    }
    return 0;
}

// hi and lo of rows of activations (K a multiple of 4): out[r] and out[rows + r] of x[gather ? gather[r] : r].  Grouped: only the
// rows that an expert has; beyond them `gather` need not be written.
__global__ void __launch_bounds__(256)
f32_split_rows_kernel(const float* __restrict__ x, const int* __restrict__ gather, const int* __restrict__ offsets, int E,
                      uint4* __restrict__ out, int rows, int lda, int K4, int64_t sA, int64_t all_rows) {
    const int r = blockIdx.x;
    if (offsets && r >= __ldg(offsets + E)) return;
    const uint4* src = reinterpret_cast<const uint4*>(x + blockIdx.y * sA + (int64_t)(gather ? __ldg(gather + r) : r) * lda);
    uint4* hi = out + ((int64_t)blockIdx.y * rows + r) * K4;
    for (int i = threadIdx.x; i < K4; i += 256) {
        const uint4 v = __ldg(src + i);
        uint4 h, l;
        split(v.x, h.x, l.x); split(v.y, h.y, l.y); split(v.z, h.z, l.z); split(v.w, h.w, l.w);
        hi[i] = h;
        hi[all_rows * K4 + i] = l;
    }
}

// NT: rows of activations per tile at most.  VEC: rows are 16-byte aligned, K is a multiple of 4 and `map_w` describes all
// rows of W (boxes of 32 floats x 128 rows, 64 in a paired product, 128-byte swizzle).
template <bool PAIRED, int NT, bool SPLIT, bool VEC>
__global__ void __launch_bounds__(threads(NT), 1)
f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ RowMaps map_rows, Problem g) {
    constexpr bool BEFORE = split_before(NT);
    static_assert(!BEFORE || VEC, "rows that are split before are aligned");
    constexpr int THREADS = threads(NT), W_SLOTS = w_slots(NT, SPLIT), LO_SLOTS = lo_slots(NT), HI_SLOTS = hi_slots(NT), D_SLOTS = d_slots(NT);
    constexpr int B_BYTES = NT * 128;
    constexpr int FEATS = PAIRED ? 64 : 128;           // outputs of a tile
    constexpr int OWN = NT / 2;                        // rows of activations of an adding warp
    constexpr int PER = NT / 16;                       // 16-byte pieces of activations per thread and chunk
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[4], done_bar[4], empty_bar[D_SLOTS], w_full[W_SLOTS], w_read[W_SLOTS], rows_full[LO_SLOTS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s;

    uint32_t rank = 0, ranks = 1;
    if (SPLIT) {
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    }
    const int n0 = (int)(blockIdx.x / ranks) * FEATS;
    int e = 0, row0, rows;
    if (g.offsets) {
        rows = row_tile(g.offsets, g.E, NT, blockIdx.y, e, row0);
        if (rows == 0) return;                         // uniform for the block and its cluster
    } else {
        row0 = blockIdx.y * NT;
        rows = min(NT, g.T - row0);
    }
    const float* A = g.A + blockIdx.z * g.sA;
    const float* W = g.W + blockIdx.z * g.sW + (int64_t)e * (PAIRED ? 2 : 1) * g.N * g.K;
    float* C = g.C + blockIdx.z * g.sC;
    const int n_mma = (rows + 15) & ~15;
    const int chunks = (g.K + FK - 1) / FK, per_part = (chunks + PARTS - 1) / PARTS;
    const int own_parts = PARTS / (int)ranks;
    const int first = min(chunks, (int)rank * own_parts * per_part), count = min(chunks, first + own_parts * per_part) - first;

    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* hi_ring = smem;                           // [slot][NT][128 bytes], swizzled
    uint8_t* lo_ring = hi_ring + HI_SLOTS * B_BYTES;
    uint8_t* w_ring = lo_ring + LO_SLOTS * B_BYTES;    // [slot][128 rows][128 bytes], swizzled
    float* sums = reinterpret_cast<float*>(w_ring + W_SLOTS * 16384);      // [part][NT][128]: SPLIT parts, otherwise their total
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    volatile int* abort_flag = &abort_s;

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int s = 0; s < 4; ++s) { mbar_init(&full_bar[s], BEFORE ? 4 : 8); mbar_init(&done_bar[s], 1); }
        for (int s = 0; s < D_SLOTS; ++s) mbar_init(&empty_bar[s], 8);
        for (int s = 0; s < LO_SLOTS; ++s) mbar_init(&rows_full[s], 1);
        for (int s = 0; s < W_SLOTS; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_read[s], 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;                 // columns 0-255: four chunks' sums; 256-511: four of weights

    // Phases of the barriers of four (full, done): whoever waits for chunk i there has itself to act before chunk i + 4
    // can complete, so a parity never stands for the phase after the next.
    if (warp < OUT_WARP) {
        const int turn = warp >> 2, quarter = warp & 3;
        // !VEC: this warp's 32 rows of chunk i, a row's lanes beside each other
        auto ask = [&](int i) {
            if (VEC) return;
            if (i < count) {
                const int k = (first + i) * FK + lane;
                const uint32_t at = smem_u32(w_ring) + (i % W_SLOTS) * 16384 + quarter * 4096;
#pragma unroll 4
                for (int r = 0; r < 32; ++r) {
                    const int f = quarter * 32 + r, n = n0 + f % FEATS;
                    const bool in = k < g.K && n < g.N;
                    cp_async4(at + r * 128 + ((((uint32_t)lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4,
                              in ? W + ((int64_t)(f / FEATS) * g.N + n) * g.K + k : g.W, in);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        constexpr int SLOTS = W_SLOTS / 2;             // of this turn
#pragma unroll 1
        for (int i = 0; i < SLOTS - 1; ++i) ask(turn + 2 * i);
        const uint8_t* w_lane = w_ring + quarter * 4096 + lane * 128;
        const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16) + 256;
#pragma unroll 1
        for (int i = turn; i < count; i += 2) {
            const int slot = i % W_SLOTS;
            if (VEC) {
                if (!wait_for(&w_full[slot], (i / W_SLOTS) & 1, abort_flag, 31)) break;
            } else {
                __syncwarp();                          // the whole warp has read its chunk before: that slot is asked for anew
                ask(i + 2 * (SLOTS - 1));
                asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory");
                __syncwarp();
            }
            // the MMAs of chunk i - T_SLOTS have read its place in tensor memory
            if (i >= T_SLOTS && !wait_for(&done_bar[i & 3], ((i - T_SLOTS) >> 2) & 1, abort_flag, 32)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint8_t* w = w_lane + slot * 16384;
            const uint32_t at = t_lane + (i % T_SLOTS) * 64;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const uint4 v = *reinterpret_cast<const uint4*>(w + (((4 * k + p) ^ (lane & 7)) << 4));
                    split(v.x, hi[4 * p], lo[4 * p]); split(v.y, hi[4 * p + 1], lo[4 * p + 1]);
                    split(v.z, hi[4 * p + 2], lo[4 * p + 2]); split(v.w, hi[4 * p + 3], lo[4 * p + 3]);
                }
                tmem_st16(at + 16 * k, hi);
                tmem_st16(at + 32 + 16 * k, lo);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full_bar[i & 3]);
                if (VEC) mbar_arrive(&w_read[slot]);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (warp < MMA_WARP) {
        // a warp's lanes are 32 features (rows of W) of the tile, its columns rows c_lo .. c_lo + OWN of the activations
        const int quarter = warp & 3, c_lo = ((warp - OUT_WARP) >> 2) * OWN, feat = quarter * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16) + c_lo;
        float* own = sums + c_lo * 128 + feat;         // of the first part; columns 128 apart
        float part[OWN];
#pragma unroll
        for (int i = 0; i < OWN; ++i) part[i] = 0.f;
        bool ok = true;
        int in_part = 0, parts = 0;
#pragma unroll 1
        for (int it = 0; it < count; ++it) {
            ok = wait_for(&done_bar[it & 3], (it >> 2) & 1, abort_flag, 37);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (c_lo < n_mma) {                        // uniform
                const uint32_t d = lane_addr + (it % D_SLOTS) * (256 / D_SLOTS);
                constexpr int GROUP = OWN < 32 ? OWN : OWN == 32 ? 32 : 16;
#pragma unroll
                for (int i0 = 0; i0 < OWN; i0 += GROUP) {
                    uint32_t v[GROUP];
                    if constexpr (GROUP == 32) tmem_ld32(d + i0, v);
                    else if constexpr (GROUP == 16) tmem_ld16(d + i0, v);
                    else tmem_ld8(d + i0, v);
                    wait_tmem_ld();
#pragma unroll
                    for (int i = 0; i < GROUP; ++i) part[i0 + i] += __uint_as_float(v[i]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_bar[it % D_SLOTS]);
            if (++in_part == per_part || it == count - 1) {
                float* to = own + (SPLIT ? parts * NT * 128 : 0);
                if (!SPLIT && parts > 0)
#pragma unroll
                    for (int i = 0; i < OWN; ++i) part[i] = to[i * 128] + part[i];
#pragma unroll
                for (int i = 0; i < OWN; ++i) {
                    to[i * 128] = 0.f + part[i];       // (a cluster's sums begin at +0, too)
                    part[i] = 0.f;
                }
                in_part = 0;
                ++parts;
            }
        }
        if (SPLIT)
            for (; parts < own_parts; ++parts)         // past the last chunk
#pragma unroll
                for (int i = 0; i < OWN; ++i) own[(parts * NT + i) * 128] = 0.f;
    } else if (warp < W_WARP) {
        const uint32_t idesc = IDESC | ((uint32_t)(n_mma >> 3) << 17);
        const uint64_t hi_desc = umma_desc(smem_u32(hi_ring)), lo_desc = umma_desc(smem_u32(lo_ring));
#pragma unroll 1
        for (int i = warp - MMA_WARP; i < count; i += 2) {
            if (!wait_for(&empty_bar[i % D_SLOTS], ((i / D_SLOTS) & 1) ^ 1, abort_flag, 35)) break;
            if (BEFORE && !wait_for(&rows_full[i % LO_SLOTS], (i / LO_SLOTS) & 1, abort_flag, 38)) break;
            if (!wait_for(&full_bar[i & 3], (i >> 2) & 1, abort_flag, 36)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t bh = hi_desc + (uint32_t)(((i % HI_SLOTS) * B_BYTES) >> 4), bl = lo_desc + (uint32_t)(((i % LO_SLOTS) * B_BYTES) >> 4);
            const uint32_t wh = tmem + 256 + (i % T_SLOTS) * 64, wl = wh + 32, d = tmem + (i % D_SLOTS) * (256 / D_SLOTS);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < FK / 8; ++k) {
                    umma_tf32_tmem_a(d, wl + k * 8, bh + k * 2, idesc, k > 0);
                    umma_tf32_tmem_a(d, wh + k * 8, bl + k * 2, idesc, 1);
                }
#pragma unroll
                for (int k = 0; k < FK / 8; ++k) umma_tf32_tmem_a(d, wh + k * 8, bh + k * 2, idesc, 1);
                umma_commit(&done_bar[i & 3]);
            }
            __syncwarp();
        }
    } else if (warp == W_WARP) {
        if (VEC && lane == 0) {
            const int row_w = (int)((blockIdx.z * g.sW) / g.K) + e * (PAIRED ? 2 : 1) * g.N + n0;          // (sW: whole rows)
            int i = 0;
#pragma unroll 1
            for (; i < count; ++i) {
                const int slot = i % W_SLOTS;
                if (!mbar_wait(&w_read[slot], ((i / W_SLOTS) & 1) ^ 1, abort_flag, 34)) break;
                mbar_expect_tx(&w_full[slot], 16384);
                uint8_t* to = w_ring + slot * 16384;
                tma_load_2d(to, &map_w, (first + i) * FK, row_w, &w_full[slot]);
                if (PAIRED) tma_load_2d(to + 8192, &map_w, (first + i) * FK, row_w + g.N, &w_full[slot]);
            }
            for (int j = max(0, i - W_SLOTS); j < i; ++j)          // nothing is on its way when the block ends, also after an abort
                for (uint32_t n = 0; n < WAIT_LIMIT && !mbar_try_wait(&w_full[j % W_SLOTS], (j / W_SLOTS) & 1); ++n) {}
        }
    } else if (BEFORE) {
        if (lane == 0) {
            const int y_hi = (int)(blockIdx.z * (int64_t)g.T + row0), y_lo = y_hi + (int)g.split_rows;
            const int n_rest = NT > 64 && n_mma > 64 ? n_mma - 64 : n_mma, at_rest = (n_mma - n_rest) * 128;
            const CUtensorMap* rest = &map_rows.m[n_rest / 16 - 1];
            int i = 0;
#pragma unroll 1
            for (; i < count; ++i) {
                // the MMAs of chunk i - LO_SLOTS have read its place
                if (i >= LO_SLOTS && !mbar_wait(&done_bar[(i - LO_SLOTS) & 3], ((i - LO_SLOTS) >> 2) & 1, abort_flag, 33)) break;
                const int slot = i % LO_SLOTS, k = (first + i) * FK;
                uint64_t* bar = &rows_full[slot];
                uint8_t *hi = hi_ring + slot * B_BYTES, *lo = lo_ring + slot * B_BYTES;
                mbar_expect_tx(bar, 2 * n_mma * 128);
                if (NT > 64 && n_mma > 64) {
                    tma_load_2d(hi, &map_rows.m[3], k, y_hi, bar);
                    tma_load_2d(lo, &map_rows.m[3], k, y_lo, bar);
                }
                tma_load_2d(hi + at_rest, rest, k, y_hi + n_mma - n_rest, bar);
                tma_load_2d(lo + at_rest, rest, k, y_lo + n_mma - n_rest, bar);
            }
            for (int j = max(0, i - LO_SLOTS); j < i; ++j)
                for (uint32_t n = 0; n < WAIT_LIMIT && !mbar_try_wait(&rows_full[j % LO_SLOTS], (j / LO_SLOTS) & 1); ++n) {}
        }
    } else {
        // this thread's pieces of a chunk are rows tid / 8 + 16 j at piece tid % 8; it alone reads what it asked for
        const int tid = threadIdx.x - 32 * ROWS_WARP, piece = tid & 7, r_lo = tid >> 3;
        const uint32_t pitch = (uint32_t)g.lda * 4u, b_lane = r_lo * 128 + ((piece ^ (r_lo & 7)) << 4);
        uint32_t row_of[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int r = r_lo + 16 * j;
            row_of[j] = r >= rows ? 0xffffffffu : g.gather ? (uint32_t)__ldg(g.gather + row0 + r) : (uint32_t)(row0 + r);
        }
        const uint32_t hi_at = smem_u32(hi_ring) + b_lane;
        auto ask = [&](int i) {
            if (i < count) {
                const int k = (first + i) * FK + piece * 4, left = g.K - k;
                const char* base = reinterpret_cast<const char*>(A + k);
                const uint32_t at = hi_at + (i % HI_SLOTS) * B_BYTES;
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    if (16 * j >= n_mma) break;        // uniform; no MMA reads these rows
                    const bool row = row_of[j] != 0xffffffffu;
                    const char* src = base + (uint64_t)row_of[j] * pitch;
                    if (VEC) {
                        const bool in = row && left > 0;
                        cp_async16(at + j * 2048, in ? src : reinterpret_cast<const char*>(g.W), in);
                    } else {
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            const bool in = row && left > x;
                            cp_async4(at + j * 2048 + 4 * x, in ? src + 4 * x : reinterpret_cast<const char*>(g.W), in);
                        }
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll 1
        for (int i = 0; i < ROWS_AHEAD; ++i) ask(i);
#pragma unroll 1
        for (int i = 0; i < count; ++i) {
            // the MMAs of chunk i - 4 have read its place in the ring of lo, and that of chunk i + 4 in the ring of hi
            if (i >= LO_SLOTS && !wait_for(&done_bar[i & 3], ((i - LO_SLOTS) >> 2) & 1, abort_flag, 33)) break;
            ask(i + ROWS_AHEAD);
            asm volatile("cp.async.wait_group %0;" ::"n"(ROWS_AHEAD) : "memory");
            uint8_t* hi_p = hi_ring + b_lane + (i % HI_SLOTS) * B_BYTES;
            uint8_t* lo_p = lo_ring + b_lane + (i % LO_SLOTS) * B_BYTES;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                if (16 * j >= n_mma) break;
                const uint4 v = *reinterpret_cast<const uint4*>(hi_p + j * 2048);
                uint4 hi, lo;
                split(v.x, hi.x, lo.x); split(v.y, hi.y, lo.y); split(v.z, hi.z, lo.z); split(v.w, hi.w, lo.w);
                *reinterpret_cast<uint4*>(hi_p + j * 2048) = hi;
                *reinterpret_cast<uint4*>(lo_p + j * 2048) = lo;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[i & 3]);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    // the outputs, by all warps: lanes along the features
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (SPLIT) asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    if (warp == MMA_WARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    if (abort_s == 0) {
        const uint32_t sums_at = smem_u32(sums);
        auto total = [&](int feat, int r) {
            if (!SPLIT) return sums[r * 128 + feat];
            float v = 0.f;
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
                uint32_t there;
                float s;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there)
                             : "r"(sums_at + (uint32_t)(((p % own_parts) * NT + r) * 128 + feat) * 4), "r"(p / own_parts));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(s) : "r"(there));
                v += s;
            }
            return v;
        };
        // rows rank, rank + ranks, ... of the tile are this block's
        for (int idx = threadIdx.x; idx < FEATS * ((rows - (int)rank + (int)ranks - 1) / (int)ranks); idx += THREADS) {
            const int feat = idx % FEATS, r = (idx / FEATS) * (int)ranks + (int)rank, n = n0 + feat, t = row0 + r;
            if (n >= g.N) continue;
            const float* a = A + (int64_t)(g.gather ? g.gather[t] : t) * g.lda;
            float v = total(feat, r);
            if (not_finite(v)) v = chain(a, W + (int64_t)n * g.K, g.K);
            if (PAIRED) {
                float up = total(feat + 64, r);
                if (not_finite(up)) up = chain(a, W + ((int64_t)g.N + n) * g.K, g.K);
                const float s = glu_row_scale(g.glu, t);
                v = glu_join(v * s, up * s, g.glu);
            }
            C[(int64_t)t * g.ldc + n] = v;
        }
    }
    if (SPLIT) {                                       // nobody leaves while its sums are read
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0 && abort_s != 0) atomicMax(g.status, abort_s);
}

}  // namespace f32tc
}  // namespace mi
