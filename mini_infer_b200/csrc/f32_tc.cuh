// Products of the true 32-bit path on the fifth-generation tensor cores, for inner sizes from TC_MIN_K up.
//
//   C[t, n] = A[t, :] . W[n, :]   (dense, one of several independent products, or an expert's rows of a grouped one)
//
// A number x of 32 bits is taken apart exactly, into three bfloat16 numbers: 2^24 x = h + m + l, each the rest rounded to 8 bits
// (the factor keeps the parts of the smallest x among the normal numbers).  Of the nine products of two numbers' parts all are formed but
// that of the two l, which is at most 2^-34 of the whole, in two sums: hh; and the others, which are 2^-8 of it and less.  The tensor
// cores add without rounding to nearest.  hh's terms have 16 bits, of which few are cut off, but 32 of them at most are added
// there: then the sum goes to registers and is added up in 32 bits as any number is.  The others stay for a part of the
// inner dimension.  Both meet in the output alone.  Measured error: see dense_f32.cu.  (Three bfloat16 parts instead of a float32:
// G. Henry, P. T. P. Tang, A. Heinecke, ARITH 2019.)
//
// Every output element is the same sums in the same order in every form below: chunks of 32 k in ascending order within
// each of four parts of the inner dimension, then the parts in ascending order.  So a row has the same bits however many
// rows share the step, in whichever tile and form, as the chains of the CUDA-core kernels have for smaller K.  A result that
// is not finite (an operand that is not, or one from 2^104 or a sum from 2^80 on) is computed again as a chain of multiply-adds, so
// infinities and NaN that operands bring reach exactly the elements that they reach there.
//
// Weights are the M operand (128 rows a tile; 64 gate rows and the up rows of the same outputs in a paired product) and lie in
// tensor memory, rows of activations are the N operand in shared memory.  Roles:
//   warps 0-7 or (tiles of 16 rows) 0-11, four for a chunk, in turn: weights, ring -> three parts -> tensor memory
//   warps 8-15 or 12-15  the sums of a chunk: tensor memory -> registers, added up
//   warps 16, 17, chunks in turn: MMAs, 16 a chunk (a warp takes 800 cycles for one in a busy SM, more than the MMAs' own time), the
//               others into a sum of its own; warp 16 allocates tensor memory.
//   warp 18     weights: memory -> ring (TMA; without it, where rows are not aligned for it, the warps that read them ask
//               for them with cp.async)
//   tiles of 64 rows: warp 19 brings the parts of the activations, which f32_split_rows_kernel has laid out as they stand here
//               (one plain copy a chunk; as boxes of rows of 64 bytes they held the tile up)
//   tiles of 16 and 32: warps 19-22, chunks in turn: activations, memory -> ring (cp.async, a warp's next two chunks ahead) ->
//               three parts in shared memory
// SPLIT: a cluster of 2 or 4 blocks shares a tile's parts and adds them up through distributed shared memory, where tiles
// alone would leave SMs without work (a decode step's few rows).
//
// Every wait on an mbarrier is bounded: one that runs out sets the status word, and all roles fall through to the exit.
#pragma once

#include "tcgen05.cuh"

#include <type_traits>

namespace mi {
namespace f32tc {

using namespace tc;

constexpr int TC_MIN_K = 512;
constexpr int FK = 32;                                 // k per chunk: 32 floats are a swizzled row of 128 bytes
constexpr int PARTS = 4;
constexpr int MMA_WARP = 16, W_WARP = 18, ROWS_WARP = 19;        // first warps of the roles
constexpr bool split_before(int nt) { return nt >= 64; }
constexpr int w_turns(int nt) { return nt == 16 ? 3 : 2; }                   // groups of four warps that take chunks of weights in turn
constexpr int threads(int nt) { return 32 * (split_before(nt) ? 20 : 23); }
constexpr int ROWS_WARPS = 4, ROWS_AHEAD = 2;          // of tiles that bring the activations themselves; a warp's chunks asked for
constexpr uint32_t SLOT_LIMIT = 65536;                 // bytes of part sums of a SPLIT block
constexpr float UP = 16777216.f, DOWN = 1.f / (UP * UP);       // factors of operands and results
// D float32, A and B bfloat16, both K-major, M = 128 (without N)
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);

// Rings, in chunks: weights; parts of the activations (at most four: see the phases below); activations on their way, where the
// block takes them apart; in tensor memory weights and sums of hh
constexpr int w_slots(int nt, bool split) { return nt == 64 ? (split ? 4 : 6) : w_turns(nt) == 3 || split ? 6 : 8; }       // (a multiple of w_turns)
constexpr int ROW_SLOTS = 4;
constexpr int raw_slots(int nt) { return split_before(nt) ? 0 : ROWS_WARPS * ROWS_AHEAD; }
constexpr int T_SLOTS = 4;
constexpr int h_slots(int nt) { return nt == 64 ? 3 : 4; }
inline size_t smem_bytes(int nt, int split) {
    return 1024 + (size_t)w_slots(nt, split > 1) * 16384 + (size_t)ROW_SLOTS * nt * 192 + (size_t)raw_slots(nt) * nt * 128 +
           (size_t)(split > 1 ? PARTS / split : 1) * 2 * nt * 512;
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
// ... for three at once: one behind the other they take 230 cycles each in a busy SM, also where nothing is left to wait for
__device__ __forceinline__ bool wait_for3(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb, uint64_t* c, uint32_t pc,
                                          volatile int* abort_flag, int code) {
    bool there = false;
    for (uint32_t i = 0; i < WAIT_LIMIT && !there; ++i) {
        const bool ta = mbar_try_wait(a, pa), tb = mbar_try_wait(b, pb), tc = mbar_try_wait(c, pc);
        there = __all_sync(0xffffffffu, ta & tb & tc);
        if (!there && *abort_flag) return false;
    }
    if (!there) *abort_flag = code;
    return there;
}

struct Problem {
    const float* A; const float* W; float* C;
    const int* gather;                                 // grouped: row of A of a sorted row (or null)
    const int* offsets;                                // grouped: [E + 1]; dense: null
    int N, K, lda, ldc, E;                             // N: outputs (a paired product has 2 N rows of W an expert)
    int64_t sA, sW, sC;                                // dense: operands of product blockIdx.z
    int row_begin, row_end;                            // the (sorted) rows of this launch
    uint8_t* parts;                                    // of their activations, tile by tile as tile_at says
    GluForm glu;
    int* status;
};

// (the descriptor's halves: only the lower one moves with the tile)
__device__ __forceinline__ void umma_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 b;\n setp.ne.b32 p, %5, 0;\n mov.b64 b, {%2, %3};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
// K-major tile in core matrices of 8 rows x 16 bytes, one behind the other along the rows, k_bytes apart along k
__device__ __forceinline__ uint64_t umma_desc_plain(uint32_t smem_addr, uint32_t k_bytes) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(k_bytes >> 4) << 16 | (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
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

// The parts of two neighbours, as pairs of bfloat16.  (Of an infinity, a NaN or a number whose h is an infinity, l is a NaN.)
__device__ __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float first_of(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float second_of(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ void add2(float& a, float& b, float x, float y) {
    asm("{\n .reg .b64 s, t;\n mov.b64 s, {%0, %1};\n mov.b64 t, {%2, %3};\n add.rn.f32x2 s, s, t;\n mov.b64 {%0, %1}, s;\n}"
        : "+f"(a), "+f"(b) : "f"(x), "f"(y));
}
// (a, b) - (x, y), exact here
__device__ __forceinline__ void less2(float& a, float& b, float x, float y) {
    asm("{\n .reg .b64 s, t, u;\n mov.b64 s, {%0, %1};\n mov.b64 t, {%2, %3};\n mov.b64 u, {%4, %4};\n fma.rn.f32x2 s, t, u, s;\n"
        " mov.b64 {%0, %1}, s;\n}" : "+f"(a), "+f"(b) : "f"(x), "f"(y), "f"(-1.f));
}
__device__ __forceinline__ void take_apart(uint32_t x0, uint32_t x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    float a = __uint_as_float(x0) * UP, b = __uint_as_float(x1) * UP;
    h = pack(a, b);
    less2(a, b, first_of(h), second_of(h));
    m = pack(a, b);
    less2(a, b, first_of(m), second_of(m));
    l = pack(a, b);
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

// An expert's rows among [begin, end) are split evenly over its tiles of up to `nt` rows, whole groups of 16.  Uniform for the warp.
__device__ __forceinline__ int row_tile(const int* __restrict__ offsets, int E, int begin, int end, int nt, int slot, int& e, int& row0) {
    const int lane = threadIdx.x & 31;
    for (int base = 0; base < E; base += 32) {
        const int i = base + lane;
        const int lo = i < E ? max(__ldg(offsets + i), begin) : 0, cnt = i < E ? max(0, min(__ldg(offsets + i + 1), end) - lo) : 0;
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

// The rows of tile `slot` of product z among the launch's: first and number.  Uniform for the warp.
__device__ __forceinline__ int tile_rows(const Problem& g, int nt, int slot, int& e, int& row0) {
    if (g.offsets) return row_tile(g.offsets, g.E, g.row_begin, g.row_end, nt, slot, e, row0);
    e = 0;
    row0 = g.row_begin + slot * nt;
    return min(nt, g.row_end - row0);
}
// Where its parts lie: chunks in turn, [8 k][part][n rows][16 bytes] each with n the tile's rows rounded up to 16 (hence room for
// 16 rows more than there are for every tile before it).
__device__ __forceinline__ int64_t tile_at(const Problem& g, int z, int slots, int slot, int row0, int chunks) {
    return ((int64_t)z * (g.row_end - g.row_begin + 16 * slots) + (row0 - g.row_begin) + 16 * slot) * chunks * (FK * 6);
}

// The parts of a tile's rows of activations, zeros from K to the end of its chunk.  Grouped: rows that no expert has are not read
// (`gather` need not be written there).  A warp's lanes are 32 rows: 32 bytes of each are read, 512 bytes of a part written.
// VEC: rows are 16-byte aligned, K is a multiple of 4.
constexpr int SPLIT_K = 64;                            // k of a block: 8 warps x 8
template <bool VEC>
__global__ void __launch_bounds__(256)
f32_split_rows_kernel(Problem g, int nt) {
    const int k = blockIdx.y * SPLIT_K + (threadIdx.x >> 5) * 8, chunks = (g.K + FK - 1) / FK;
    int e = 0, row0 = 0;
    const int rows = tile_rows(g, nt, blockIdx.x, e, row0), n = (rows + 15) & ~15;
    if (k >= chunks * FK) return;
    uint4* to = reinterpret_cast<uint4*>(g.parts + tile_at(g, blockIdx.z, gridDim.x, blockIdx.x, row0, chunks)) + (int64_t)(k / 8) * 3 * n;
    for (int r = threadIdx.x & 31; r < rows; r += 32) {
        const int64_t row = g.gather ? __ldg(g.gather + row0 + r) : row0 + r;
        const float* src = g.A + blockIdx.z * g.sA + row * g.lda + k;
        uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
        if (VEC) {
            if (k < g.K) a = __ldg(reinterpret_cast<const uint4*>(src));
            if (k + 4 < g.K) b = __ldg(reinterpret_cast<const uint4*>(src) + 1);
        } else {
            auto at = [&](int x) { return k + x < g.K ? __float_as_uint(__ldg(src + x)) : 0u; };
            a = make_uint4(at(0), at(1), at(2), at(3));
            b = make_uint4(at(4), at(5), at(6), at(7));
        }
        uint4 h, m, l;
        take_apart(a.x, a.y, h.x, m.x, l.x);
        take_apart(a.z, a.w, h.y, m.y, l.y);
        take_apart(b.x, b.y, h.z, m.z, l.z);
        take_apart(b.z, b.w, h.w, m.w, l.w);
        to[r] = h;
        to[n + r] = m;
        to[2 * n + r] = l;
    }
}

// NT: rows of activations per tile at most.  VEC: rows (of weights, and of activations that the block brings itself) are 16-byte
// aligned, K is a multiple of 4 and `map_w` describes all rows of W (boxes of 32 floats x 128 rows, 64 in a paired product,
// 128-byte swizzle).
template <bool PAIRED, int NT, bool SPLIT, bool VEC>
__global__ void __launch_bounds__(threads(NT), 1)
f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, Problem g) {
    constexpr bool BEFORE = split_before(NT);
    constexpr int THREADS = threads(NT), W_SLOTS = w_slots(NT, SPLIT), RAW_SLOTS = raw_slots(NT), H_SLOTS = h_slots(NT);
    constexpr int TURNS = w_turns(NT), OUT_WARP = 4 * TURNS;
    static_assert(W_SLOTS % TURNS == 0, "a turn's own slots");
    // columns of tensor memory: H_SLOTS chunks' hh; the others of either MMA warp; T_SLOTS chunks of weights, 16 columns a part
    constexpr int OTHERS_AT = 192, W_AT = 320;
    static_assert(H_SLOTS * NT <= OTHERS_AT && OTHERS_AT + 2 * NT <= W_AT && W_AT + T_SLOTS * 48 <= 512, "tensor memory");
    constexpr int ROW_BYTES = NT * 192;                // a chunk's activations: [8 k][part][rows][16 bytes]
    constexpr int FEATS = PAIRED ? 64 : 128;           // outputs of a tile
    constexpr int OWN = NT / ((MMA_WARP - OUT_WARP) / 4);                  // rows of activations of an adding warp
    constexpr int PER = NT / 4;                        // 16-byte pieces of activations per lane and chunk
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[4], done_bar[8], empty_bar[H_SLOTS], others_read, w_full[W_SLOTS], w_read[W_SLOTS], rows_full[ROW_SLOTS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s;

    uint32_t rank = 0, ranks = 1;
    if (SPLIT) {
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    }
    const int n0 = (int)(blockIdx.x / ranks) * FEATS;
    int e = 0, row0 = 0;
    const int rows = tile_rows(g, NT, blockIdx.y, e, row0);
    if (rows == 0) return;                             // uniform for the block and its cluster
    const float* A = g.A + blockIdx.z * g.sA;
    const float* W = g.W + blockIdx.z * g.sW + (int64_t)e * (PAIRED ? 2 : 1) * g.N * g.K;
    float* C = g.C + blockIdx.z * g.sC;
    const int n_mma = (rows + 15) & ~15;
    const int chunks = (g.K + FK - 1) / FK, per_part = (chunks + PARTS - 1) / PARTS;
    const int own_parts = PARTS / (int)ranks;
    const int first = min(chunks, (int)rank * own_parts * per_part), count = min(chunks, first + own_parts * per_part) - first;

    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* rows_ring = smem;
    uint8_t* raw_ring = rows_ring + ROW_SLOTS * ROW_BYTES;                 // [slot][NT][128 bytes]
    uint8_t* w_ring = raw_ring + RAW_SLOTS * NT * 128;                     // [slot][128 rows][128 bytes], swizzled
    float* sums = reinterpret_cast<float*>(w_ring + W_SLOTS * 16384);      // [part][hh, others][NT][128]: SPLIT parts, otherwise their total
    const uint32_t part_bytes = (uint32_t)n_mma * 16;  // of 8 k
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    volatile int* abort_flag = &abort_s;

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int s = 0; s < 4; ++s) mbar_init(&full_bar[s], BEFORE ? 4 : 5);
        for (int s = 0; s < 8; ++s) mbar_init(&done_bar[s], 1);
        for (int s = 0; s < H_SLOTS; ++s) mbar_init(&empty_bar[s], MMA_WARP - OUT_WARP);
        mbar_init(&others_read, MMA_WARP - OUT_WARP);
        for (int s = 0; s < ROW_SLOTS; ++s) mbar_init(&rows_full[s], 1);
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
    const uint32_t tmem = tmem_base_s;

    // Phases of full and done: whoever waits for chunk i there has itself to act before chunk i + 4 can complete, so a parity never
    // stands for the phase after the next.  Nor for the one before: done has eight barriers, since the two MMA warps' chunks complete
    // in either order and a warp of the weights, which waits for every third chunk, then knows of all chunks eight before alone.
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
        constexpr int SLOTS = W_SLOTS / TURNS;         // of this turn
#pragma unroll 1
        for (int i = 0; i < SLOTS - 1; ++i) ask(turn + TURNS * i);
        const uint8_t* w_lane = w_ring + quarter * 4096 + lane * 128;
        const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16) + W_AT;
#pragma unroll 1
        for (int i = turn; i < count; i += TURNS) {
            const int slot = i % W_SLOTS;
            if (VEC) {
                if (!wait_for(&w_full[slot], (i / W_SLOTS) & 1, abort_flag, 31)) break;
            } else {
                __syncwarp();                          // the whole warp has read its chunk before: that slot is asked for anew
                ask(i + TURNS * (SLOTS - 1));
                asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory");
                __syncwarp();
            }
            const uint8_t* w = w_lane + slot * 16384;
            const uint32_t at = t_lane + (i % T_SLOTS) * 48;
            uint32_t h[16], m[16], l[16];
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                const uint4 v = *reinterpret_cast<const uint4*>(w + ((p ^ (lane & 7)) << 4));
                take_apart(v.x, v.y, h[2 * p], m[2 * p], l[2 * p]);
                take_apart(v.z, v.w, h[2 * p + 1], m[2 * p + 1], l[2 * p + 1]);
            }
            if (VEC) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&w_read[slot]);
            }
            // the MMAs of chunk i - T_SLOTS have read its place in tensor memory
            if (i >= T_SLOTS && !wait_for(&done_bar[(i - T_SLOTS) & 7], ((i - T_SLOTS) >> 3) & 1, abort_flag, 32)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_st16(at, h);
            tmem_st16(at + 16, m);
            tmem_st16(at + 32, l);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[i & 3]);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (warp < MMA_WARP) {
        // a warp's lanes are 32 features (rows of W) of the tile, its columns rows c_lo .. c_lo + OWN of the activations
        const int quarter = warp & 3, c_lo = ((warp - OUT_WARP) >> 2) * OWN, feat = quarter * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16) + c_lo;
        float* own = sums + c_lo * 128 + feat;         // of the first part; columns 128 apart
        float part[OWN];                               // hh
#pragma unroll
        for (int i = 0; i < OWN; ++i) part[i] = 0.f;
        bool ok = true;
        int in_part = 0, parts = 0;
#pragma unroll 1
        for (int it = 0; it < count; ++it) {
            ok = wait_for(&done_bar[it & 7], (it >> 3) & 1, abort_flag, 37);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (c_lo < n_mma) {                        // uniform
                const uint32_t d = lane_addr + (it % H_SLOTS) * NT;
                uint32_t v[OWN];
                if constexpr (OWN == 32) tmem_ld32(d, v);
                else if constexpr (OWN == 16) tmem_ld16(d, v);
                else tmem_ld8(d, v);
                wait_tmem_ld();
#pragma unroll
                for (int i = 0; i < OWN; i += 2) add2(part[i], part[i + 1], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_bar[it % H_SLOTS]);
            if (++in_part == per_part || it == count - 1) {
                // the others of both MMA warps, the next part's may follow
                float* to = own + (SPLIT ? parts * 2 * NT * 128 : 0);
                constexpr int GROUP = OWN < 16 ? OWN : 16;
                float others[OWN];
#pragma unroll
                for (int i0 = 0; i0 < OWN; i0 += GROUP) {
                    const uint32_t d = lane_addr + OTHERS_AT + i0;
                    uint32_t x[GROUP], y[GROUP];
                    if constexpr (GROUP == 16) { tmem_ld16(d, x); tmem_ld16(d + NT, y); }
                    else { tmem_ld8(d, x); tmem_ld8(d + NT, y); }
                    wait_tmem_ld();
#pragma unroll
                    for (int i = 0; i < GROUP; ++i) others[i0 + i] = __uint_as_float(x[i]) + __uint_as_float(y[i]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&others_read);
                const bool more = !SPLIT && parts > 0;
#pragma unroll
                for (int i0 = 0; i0 < 2 * OWN; i0 += GROUP) {                // hh, others
                    const bool hh = i0 < OWN;
                    float* at = to + (hh ? i0 : NT + i0 - OWN) * 128;
                    float before[GROUP];               // (all loads ahead of the additions)
#pragma unroll
                    for (int i = 0; i < GROUP; ++i) before[i] = more ? at[i * 128] : 0.f;      // (a cluster's sums begin at +0, too)
#pragma unroll
                    for (int i = 0; i < GROUP; ++i) {
                        at[i * 128] = before[i] + (hh ? part[i0 + i] : others[i0 - OWN + i]);
                        if (hh) part[i0 + i] = 0.f;
                    }
                }
                in_part = 0;
                ++parts;
            }
        }
        if (SPLIT)
            for (; parts < own_parts; ++parts)         // past the last chunk
#pragma unroll
                for (int i = 0; i < OWN; ++i) own[(parts * 2 * NT + i) * 128] = own[((parts * 2 + 1) * NT + i) * 128] = 0.f;
    } else if (warp < W_WARP) {
        // The rows' number is a constant in here: with the operands formed from a variable one the warp took 450 cycles a chunk to
        // give the products out, and more than that to wait for what was there.
        auto give = [&](auto rows_c) {
            constexpr uint32_t n = decltype(rows_c)::value, DESC = IDESC | (n >> 3) << 17;
            constexpr uint32_t K_STEP = 6 * n;         // 16 k of rows; of weights 8 columns
            const uint64_t rows_desc = umma_desc_plain(smem_u32(rows_ring), 48 * n);
            const uint32_t desc_lo = (uint32_t)rows_desc, desc_hi = (uint32_t)(rows_desc >> 32);
            const uint32_t t = __reduce_max_sync(0xffffffffu, tmem);       // (the same in all lanes also for the compiler)
            // (every part has two chunks and more: inner sizes from 512 up)
            int in_part = warp - MMA_WARP, parts = 0;
            const uint32_t others = t + OTHERS_AT + in_part * NT;
#pragma unroll 1
            for (int i = in_part; i < count; i += 2) {
                if (in_part < 2 && parts > 0 && !wait_for(&others_read, (parts - 1) & 1, abort_flag, 36)) break;
                // room for the sums, rows (where no copy brings them: the room once more), weights (and rows)
                const uint32_t room = ((i / H_SLOTS) & 1) ^ 1;
                uint64_t* empty = &empty_bar[i % H_SLOTS];
                if (!wait_for3(empty, room, BEFORE ? &rows_full[i % ROW_SLOTS] : empty, BEFORE ? (i / ROW_SLOTS) & 1 : room,
                               &full_bar[i & 3], (i >> 2) & 1, abort_flag, 35)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t bh = desc_lo + (i % ROW_SLOTS) * (ROW_BYTES >> 4), bm = bh + n, bl = bm + n;
                const uint32_t wh = t + W_AT + (i % T_SLOTS) * 48, wm = wh + 16, wl = wm + 16, hh = t + (i % H_SLOTS) * NT;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < FK / 16; ++k) {
                        umma_tmem_a(hh, wh + k * 8, bh + k * K_STEP, desc_hi, DESC, k > 0);
                        umma_tmem_a(others, wh + k * 8, bm + k * K_STEP, desc_hi, DESC, in_part > 1 || k > 0);
                        umma_tmem_a(others, wm + k * 8, bh + k * K_STEP, desc_hi, DESC, 1);
                        umma_tmem_a(others, wh + k * 8, bl + k * K_STEP, desc_hi, DESC, 1);
                        umma_tmem_a(others, wm + k * 8, bm + k * K_STEP, desc_hi, DESC, 1);
                        umma_tmem_a(others, wl + k * 8, bh + k * K_STEP, desc_hi, DESC, 1);
                        umma_tmem_a(others, wm + k * 8, bl + k * K_STEP, desc_hi, DESC, 1);
                        umma_tmem_a(others, wl + k * 8, bm + k * K_STEP, desc_hi, DESC, 1);
                    }
                    umma_commit(&done_bar[i & 7]);
                }
                __syncwarp();
                in_part += 2;
                if (in_part >= per_part) in_part -= per_part, ++parts;
            }
        };
        if (NT == 16 || n_mma == 16) give(std::integral_constant<uint32_t, 16>());
        else if (NT == 32 || n_mma == 32) give(std::integral_constant<uint32_t, NT < 32 ? 16 : 32>());
        else if (n_mma == 48) give(std::integral_constant<uint32_t, NT < 64 ? 16 : 48>());
        else give(std::integral_constant<uint32_t, NT < 64 ? 16 : 64>());
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
    } else if constexpr (BEFORE) {
        if (lane == 0) {
            const uint32_t bytes = 12 * part_bytes;
            const uint8_t* from = g.parts + tile_at(g, blockIdx.z, gridDim.y, blockIdx.y, row0, chunks) + (int64_t)first * bytes;
            int i = 0;
#pragma unroll 1
            for (; i < count; ++i) {
                // the MMAs of chunk i - ROW_SLOTS have read its place
                if (i >= ROW_SLOTS && !mbar_wait(&done_bar[(i - ROW_SLOTS) & 7], ((i - ROW_SLOTS) >> 3) & 1, abort_flag, 33)) break;
                const int slot = i % ROW_SLOTS;
                mbar_expect_tx(&rows_full[slot], bytes);
                bulk_load(rows_ring + slot * ROW_BYTES, from + (int64_t)i * bytes, bytes, &rows_full[slot]);
            }
            for (int j = max(0, i - ROW_SLOTS); j < i; ++j)
                for (uint32_t n = 0; n < WAIT_LIMIT && !mbar_try_wait(&rows_full[j % ROW_SLOTS], (j / ROW_SLOTS) & 1); ++n) {}
        }
    } else {
        // a lane's pieces of a chunk are rows lane / 8 + 4 j at piece lane % 8; it alone reads what it asked for
        const int own = warp - ROWS_WARP, piece = lane & 7, r_lo = lane >> 3;
        const uint32_t pitch = (uint32_t)g.lda * 4u;
        const uint32_t rows_lane = (piece >> 1) * 3 * part_bytes + r_lo * 16 + (piece & 1) * 8;       // 8 bytes of each part
        uint32_t row_of[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int r = r_lo + 4 * j;
            row_of[j] = r >= rows ? 0xffffffffu : g.gather ? (uint32_t)__ldg(g.gather + row0 + r) : (uint32_t)(row0 + r);
        }
        const uint32_t raw_at = smem_u32(raw_ring) + lane * 16;
        auto ask = [&](int i) {
            if (i < count) {
                const int k = (first + i) * FK + piece * 4, left = g.K - k;
                const char* base = reinterpret_cast<const char*>(A + k);
                const uint32_t at = raw_at + (i % RAW_SLOTS) * (NT * 128);
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    if (4 * j >= n_mma) break;         // uniform; no MMA reads these rows
                    const bool row = row_of[j] != 0xffffffffu;
                    const char* src = base + (uint64_t)row_of[j] * pitch;
                    if (VEC) {
                        const bool in = row && left > 0;
                        cp_async16(at + j * 512, in ? src : reinterpret_cast<const char*>(g.W), in);
                    } else {
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            const bool in = row && left > x;
                            cp_async4(at + j * 512 + 4 * x, in ? src + 4 * x : reinterpret_cast<const char*>(g.W), in);
                        }
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll 1
        for (int i = 0; i < ROWS_AHEAD; ++i) ask(own + i * ROWS_WARPS);
#pragma unroll 1
        for (int i = own; i < count; i += ROWS_WARPS) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ROWS_AHEAD - 1) : "memory");
            // the MMAs of chunk i - ROW_SLOTS have read its place
            if (i >= ROW_SLOTS && !wait_for(&done_bar[(i - ROW_SLOTS) & 7], ((i - ROW_SLOTS) >> 3) & 1, abort_flag, 33)) break;
            const uint8_t* from = raw_ring + lane * 16 + (i % RAW_SLOTS) * (NT * 128);
            uint8_t* to = rows_ring + rows_lane + (i % ROW_SLOTS) * ROW_BYTES;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                if (4 * j >= n_mma) break;
                const uint4 v = *reinterpret_cast<const uint4*>(from + j * 512);
                uint2 h, m, l;
                take_apart(v.x, v.y, h.x, m.x, l.x);
                take_apart(v.z, v.w, h.y, m.y, l.y);
                *reinterpret_cast<uint2*>(to + j * 64) = h;
                *reinterpret_cast<uint2*>(to + j * 64 + part_bytes) = m;
                *reinterpret_cast<uint2*>(to + j * 64 + 2 * part_bytes) = l;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[i & 3]);
            ask(i + ROWS_AHEAD * ROWS_WARPS);          // into the place of this chunk, which this lane has read
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
        auto sum = [&](int feat, int r) {
            if (!SPLIT) return sums[r * 128 + feat];
            float v = 0.f;
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
                uint32_t there;
                float s;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there)
                             : "r"(sums_at + (uint32_t)(((p % own_parts) * 2 * NT + r) * 128 + feat) * 4), "r"(p / own_parts));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(s) : "r"(there));
                v += s;
            }
            return v;
        };
        auto total = [&](int feat, int r) { return (sum(feat, r) + sum(feat, NT + r)) * DOWN; };
        // rows rank, rank + ranks, ... of the tile are this block's
        constexpr int MOST = (FEATS * NT + THREADS - 1) / THREADS;
        const int outputs = FEATS * ((rows - (int)rank + (int)ranks - 1) / (int)ranks);
        auto place = [&](int j, int& feat, int& r) {
            const int idx = threadIdx.x + j * THREADS;
            feat = idx % FEATS;
            r = (idx / FEATS) * (int)ranks + (int)rank;
            return idx < outputs && n0 + feat < g.N;
        };
        auto put = [&](int feat, int r, float v, float up) {
            const int t = row0 + r;
            if (PAIRED) {
                const float s = glu_row_scale(g.glu, t);
                v = glu_join(v * s, up * s, g.glu);
            }
            C[(int64_t)t * g.ldc + n0 + feat] = v;
        };
        uint32_t again = 0, again_up = 0;              // of this thread's outputs, those that are not finite
        static_assert(MOST <= 32, "a bit each");
        for (int j = 0; j < MOST; ++j) {
            int feat, r;
            if (!place(j, feat, r)) continue;
            const float v = total(feat, r), up = PAIRED ? total(feat + 64, r) : 0.f;
            again |= (uint32_t)not_finite(v) << j;
            again_up |= (uint32_t)not_finite(up) << j;
            if (!(not_finite(v) || not_finite(up))) put(feat, r, v, up);
        }
        if (__syncthreads_or((again | again_up) != 0)) {
            // ... once more as the CUDA-core kernels compute them, the tile's operands by way of the rings.  512 rows against
            // [6144, 2048]: 0.11 ms; one of them NaN 0.28 ms; all of them 2.3 ms (43.7 with a thread's operands from memory).
            constexpr int PITCH = FK + 1;
            float* w_s = reinterpret_cast<float*>(smem);
            float* a_s = w_s + 128 * PITCH;
            float acc[MOST], acc_up[PAIRED ? MOST : 1];
#pragma unroll
            for (int j = 0; j < MOST; ++j) acc[j] = 0.f;
#pragma unroll
            for (int j = 0; j < (PAIRED ? MOST : 1); ++j) acc_up[j] = 0.f;
            for (int k0 = 0; k0 < g.K; k0 += FK) {
                __syncthreads();
                for (int i = threadIdx.x; i < 128 * FK; i += THREADS) {
                    const int f = i / FK, k = k0 + i % FK, n = n0 + f % FEATS;
                    w_s[f * PITCH + i % FK] = n < g.N && k < g.K ? W[((int64_t)(f / FEATS) * g.N + n) * g.K + k] : 0.f;
                }
                for (int i = threadIdx.x; i < rows * FK; i += THREADS) {
                    const int t = row0 + i / FK, k = k0 + i % FK;
                    a_s[i / FK * PITCH + i % FK] = k < g.K ? A[(int64_t)(g.gather ? g.gather[t] : t) * g.lda + k] : 0.f;
                }
                __syncthreads();
                const int n = min(FK, g.K - k0);
#pragma unroll
                for (int j = 0; j < MOST; ++j) {
                    int feat, r;
                    place(j, feat, r);
                    const float *a = a_s + r * PITCH, *w = w_s + feat * PITCH;
                    if (again >> j & 1)
                        for (int k = 0; k < n; ++k) acc[j] = fmaf(a[k], w[k], acc[j]);
                    if (PAIRED && (again_up >> j & 1))
                        for (int k = 0; k < n; ++k) acc_up[PAIRED ? j : 0] = fmaf(a[k], w[64 * PITCH + k], acc_up[PAIRED ? j : 0]);
                }
            }
#pragma unroll
            for (int j = 0; j < MOST; ++j) {
                int feat, r;
                if (!place(j, feat, r) || !((again | again_up) >> j & 1)) continue;
                put(feat, r, again >> j & 1 ? acc[j] : total(feat, r),
                    !PAIRED ? 0.f : again_up >> j & 1 ? acc_up[PAIRED ? j : 0] : total(feat + 64, r));
            }
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
