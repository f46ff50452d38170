// Prefill attention on the fifth-generation tensor cores (bfloat16, head size 64 or 128): portions
// of prompts of a ragged batch over the paged cache, flash-attention style, with both products on
// tcgen05.mma and their accumulators in tensor memory.
//
// Block = 256 queries of one head as two query tiles of 128 that read the same key tiles: one's softmax runs beside
// the other's tensor-core work.  Key tiles of 64, aligned to absolute positions, arrive page by page
// through TMA (128-byte swizzle) into rings of K and V tiles as deep as shared memory allows.  Per key and query tile:
//   S = Q K^T    A = Q tile (K-major), B = K tile (K-major), accumulator S[buf] in tensor memory
//   softmax      two threads per query row, 32 keys each (a row is a lane of tensor memory; the two
//                threads sit in two warps of the same lane quarter): the row of S comes to registers with
//                tcgen05.ld, P = exp2(s - reference) is rounded to bfloat16 and written over S in
//                place with tcgen05.st (two keys per 32-bit column); the reference follows the
//                running maximum only when that moved by more than 8 (P stays below 2^8), and only
//                then O is scaled in place (tcgen05.ld / .st).  The two halves' maxima meet in shared
//                memory, their sums once, at the end
//   O += P V     A = P straight from tensor memory, B = V tile as it lies in the cache (keys x head,
//                i.e. MN-major), accumulator O in tensor memory
//   warps 0-7, 8-15  softmax and epilogue of the first and the second query tile
//   warps 16, 17     TMA producers of K (and Q) and of V, one copy per page and 64 columns
//   warps 18, 19     issue the MMAs of the first and the second query tile (18 allocates tensor memory)
// What bounds it is the chain of one key tile (wait, load, maximum, exponentials, store, hand-over, product), so
// every part of the chain is kept off the producers' way: page numbers are looked up a tile ahead, K and V have a warp
// each, and a block that has the SM to itself keeps four and more tiles of each on their way (two blocks of one query
// tile per SM, with one producer and rings of three K and two V tiles: 1.9 us a key tile).
// S is double-buffered, so the next tile's S = Q K^T runs beside this tile's softmax.  Masking is positional: key j is visible from the
// query at position p iff j <= p and (window == 0 or j > p - window or j < keep_first) and j < kv_len; with chunks
// instead of a window iff j <= p and j lies in p's chunk (or j < keep_first): see AttnForm, which also gives the added
// key of `sink` a score per head and the output a gate per head.
//
// Every wait on an mbarrier is bounded: a wait that runs out sets an error status that the host
// reads, lets all roles fall through to the common exit, and the tensor memory is freed there.
//
// The reference computes prefill with one block per (request, head, query) and scalar dot
// products over every page of the request (src/kernels/paged_attn_kernel.cu:102-288).

#include "prefill_rules.h"
#include "tcgen05.cuh"

namespace mi {
namespace pt {

using namespace mi::tc;

constexpr int BN = 64;             // keys per tile
constexpr int HK = BN / 2;         // keys of a tile that a softmax thread takes
constexpr int THREADS = 640;       // 2 x 8 softmax warps, two producers, two that issue MMAs
constexpr int HALF_BYTES = 128 * 64 * 2;   // a tile of 128 rows x 64 columns: 16 KiB (Q)
constexpr int KV_HALF = BN * 64 * 2;       // a tile of BN keys x 64 columns: 8 KiB
// behind the tiles: barriers and words, then the halves' maxima of two tiles in turn, per query tile [2][2][BQ] floats
constexpr int WORDS = 512;
constexpr int tail(int dk) { return WORDS + query_tiles(dk) * 2 * 2 * BQ * 4; }
constexpr int SMEM_MAX = 227 * 1024;
// Stages of the rings: as many K and V tiles as fit beside the queries (8 of each at most).
constexpr int stages(int dk, int dv) {
    const int per = (dk / 64 + dv / 64) * KV_HALF, room = SMEM_MAX - tail(dk) - query_tiles(dk) * (dk / 64) * HALF_BYTES;
    return room / per < 8 ? room / per : 8;
}
constexpr size_t smem_bytes(int dk, int dv) {
    return (size_t)query_tiles(dk) * (dk / 64) * HALF_BYTES + (size_t)stages(dk, dv) * (dk / 64 + dv / 64) * KV_HALF + tail(dk);
}
static_assert(stages(256, 128) >= 3 && stages(192, 128) >= 3, "rings of three stages at the largest sizes");
// blocks along x: the query tiles of the longest portion, for every head
inline unsigned grid_x(int64_t rows, int heads, QueryTiles order) {
    const int64_t tiles = (rows + BQ - 1) / BQ;
    return (unsigned)((order == kSingle ? tiles : (tiles + 1) / 2) * heads);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// Matrix descriptor of an MN-major operand with 128-byte swizzle: rows of 128 bytes are steps of the
// contraction index, 8 of them 1024 B apart (stride byte offset); the next 64 elements of the
// non-contracted index lie `lbo_bytes` further (leading byte offset).
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t smem_addr, uint32_t lbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// tcgen05.mma with the A operand in tensor memory (lane = row, a 32-bit column holds two bfloat16 of
// consecutive k) and B in shared memory.
__device__ __forceinline__ void umma_bf16_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Barrier `id` of the two warps that share a lane quarter of a query tile; whether `ok` held for all of their threads.
__device__ __forceinline__ bool pair_and(int id, bool ok) {
    uint32_t all;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.and.pred q, %2, 64, p;\n selp.u32 %0, 1, 0, q;\n}"
                 : "=r"(all) : "r"((uint32_t)ok), "r"(id) : "memory");
    return all != 0;
}
// two multiply-adds, two additions in one instruction (each rounded as by itself)
__device__ __forceinline__ float2 fma_two(float2 a, float b, float c) {
    float2 r;
    asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n mov.b64 z, {%5, %5};\n"
        " fma.rn.f32x2 x, x, y, z;\n mov.b64 {%0, %1}, x;\n}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float2 add_two(float2 a, float2 b) {
    float2 r;
    asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x;\n}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

struct Maps {
    CUtensorMap q, k, v, kr;
};

// Keys and values that were formed from a latent before the call (UNFOLDED): token-major rows, all requests' contexts
// one after the other, [rows, nh * d] unrotated keys (map k), [rows, nh * e] values (map v) and the rotated key part
// that the heads share, [rows, r] (map kr).  A key tile is `d` columns of the head, in halves of 64, then the shared
// part in halves of its own; q [tokens, nh, DK] is laid out alike, with zeros between what the two parts fill.
struct Unfolded {
    int d16, r16;               // steps of 16 columns that the unrotated and the rotated part take
    int d, e;                   // columns of a head in the maps k and v
    const float* gate;          // null, or rows of `ldg` floats: out *= logistic(gate[t, gcol + h e + :])
    int ldg, gcol;
};

// DK, DV: key and value sizes in whole 64-column halves (a key row shorter than DK reads zeros beyond its end,
// in Q and in K alike).  hpq > 1 (with nh = nkv = 1): the heads of a query all read ONE key/value head, so the
// rows of a tile are (query, head) pairs, hpq consecutive rows a query: q and out are [tokens * hpq, .].
// CAPPED: every score becomes cap * tanh(score * scale / cap) before the mask and the softmax (`cap_in` =
// scale / cap, `cap_out` = cap / scale, so that what follows scales the capped number as it scales a plain one).
// `sink`: the softmax counts one key more, of score 0 and without a value: the reference of the exponentials
// starts at 0 and the running sum at 1.
// LOGISTIC: no softmax.  A visible key's weight is logistic(score * scale + head_bias[h]) by itself, not normalised
// over the keys: nothing follows a maximum, O is never rescaled and leaves as it is.
__device__ __forceinline__ float fast_tanh(float x) {
    return 1.0f - __fdividef(2.0f, fast_exp2(x * 2.8853900817779268f) + 1.0f);
}

template <int DK, int DV, bool CAPPED = false, bool LOGISTIC = false, bool UNFOLDED = false>
__global__ void __launch_bounds__(THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ Maps maps, const int* __restrict__ block_table,
                       const int* __restrict__ q_start, const int* __restrict__ kv_len,
                       __nv_bfloat16* __restrict__ out, int nh, int nkv, int page_size, int max_pages,
                       int window, float scale_log2, int* __restrict__ status, int keep_first, int hpq,
                       float cap_in, float cap_out, int sink, const float* __restrict__ head_bias, Unfolded uf, AttnForm form,
                       QueryTiles order) {
    constexpr int DKH = DK / 64, DVH = DV / 64;           // 64-column halves of a key and of a value row
    constexpr int NS = stages(DK, DV), QT = query_tiles(DK);
    constexpr uint32_t TMEM_COLS = 512;                   // per query tile S[0], S[1] (BN columns each), O (128)
    constexpr uint32_t COL_O = 2 * BN, COL_TILE = 256;
    // instruction descriptors: D float32, A and B bfloat16, M = 128
    constexpr uint32_t IDESC_S = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((128u >> 4) << 24);
    constexpr uint32_t IDESC_PV = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(DV >> 3) << 17) |
                                  ((128u >> 4) << 24);    // B (the V tile) MN-major
    extern __shared__ __align__(1024) uint8_t smem[];     // tiles first (the swizzle wants 1024-byte alignment)
    uint8_t* sQ = smem;                                   // per query tile DKH halves of [128 queries][64]
    uint8_t* sK = sQ + QT * DKH * HALF_BYTES;             // NS stages of DKH halves of [BN keys][64]
    uint8_t* sV = sK + NS * DKH * KV_HALF;                // NS stages of DVH halves for V
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + NS * DVH * KV_HALF);
    uint64_t* k_full = bars;
    uint64_t* v_full = k_full + NS;
    uint64_t* k_empty = v_full + NS;
    uint64_t* v_empty = k_empty + NS;
    uint64_t* q_full = v_empty + NS;                      // the rest per query tile
    uint64_t* s_full = q_full + QT;                       // [QT][2]
    uint64_t* p_full = s_full + QT * 2;                   // [QT][2] per S/P buffer: the softmax may be a tile ahead
    uint64_t* o_done = p_full + QT * 2;
    uint32_t* tmem_base_p = reinterpret_cast<uint32_t*>(o_done + QT);
    int* abort_p = reinterpret_cast<int*>(tmem_base_p + 1);
    float* halves = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + WORDS);      // [QT][2 in turn][2][BQ]
    static_assert((4 * 8 + QT * 6) * 8 + 8 <= WORDS, "barriers and words");

    // later queries see more keys: those of all heads are launched first, so that the short ones fill the tail
    const int b = blockIdx.z, h = blockIdx.x % nh, step = blockIdx.x / nh;
    const int q0 = q_start[b] * hpq, q_len = (q_start[b + 1] - q_start[b]) * hpq;      // in rows
    const int n_q = (q_len + BQ - 1) / BQ, n_blocks = order == kSingle ? n_q : (n_q + 1) / 2;
    if (step >= n_blocks) return;                         // uniform for the whole block
    const int kvl = kv_len[b];
    const bool bounded = window > 0 || form.chunk > 0;    // keys before some position are out of sight
    const int tile_a = order == kNeighbours ? 2 * (n_blocks - 1 - step) : n_q - 1 - step;
    const int tile_b = order == kSingle ? tile_a : min(order == kApart ? step : tile_a + 1, n_q - 1);
    const int tiles_q = tile_a == tile_b ? 1 : 2;
    const int hk = h / (nh / nkv);
    const int dh = UNFOLDED ? (uf.d16 + 3) / 4 : DKH;     // halves of the unrotated part
    int kv_base = 0;                                      // first row of the request's context in the maps
    if constexpr (UNFOLDED) for (int i = 0; i < b; ++i) kv_base += kv_len[i];
    const int pos0 = kvl - q_len / hpq;                   // position of the portion's first query (hpq divides BQ)
    auto row_of = [&](int t) { return (t ? tile_b : tile_a) * BQ; };                   // a query tile's first row,
    auto rows_of = [&](int t) { return min(BQ, q_len - row_of(t)); };                  // its number of rows,
    auto last_of = [&](int t) { return pos0 + (row_of(t) + rows_of(t) - 1) / hpq; };   // its last position
    const int blk_lo = pos0 + min(row_of(0), row_of(1)) / hpq, blk_hi = max(last_of(0), last_of(1));
    // Both query tiles read the same key tiles, each up to its last position.
    const int k_begin = (first_visible(blk_lo, window, form.chunk) / BN) * BN;
    const int k_end = min(kvl, blk_hi + 1);
    // Behind a window the first keep_first keys of a request stay visible: tiles over [0, sink_end) come
    // before the window's tiles.  Keys between the two are seen by no query of this block (k_begin is not
    // above any query's window).
    const int sink_end = bounded ? min(min(keep_first, k_begin), k_end) : 0;
    const int n_sink = (sink_end + BN - 1) / BN;
    const int n_tiles = n_sink + (k_end - k_begin + BN - 1) / BN;  // >= 1: the query's own key is visible
    auto tiles_of = [&](int t) { return n_sink + (min(kvl, last_of(t) + 1) - k_begin + BN - 1) / BN; };
    auto tile_start = [&](int j) { return j < n_sink ? j * BN : k_begin + (j - n_sink) * BN; };

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    volatile int* abort_flag = abort_p;

    if (threadIdx.x == 0) {
        *abort_p = (smem_u32(smem) & 1023u) ? 10 : 0;     // misplaced tiles: nothing is issued
        for (int s = 0; s < NS; ++s) {
            mbar_init(&k_full[s], 1); mbar_init(&v_full[s], 1);
            mbar_init(&k_empty[s], tiles_q); mbar_init(&v_empty[s], tiles_q);     // every query tile has read it
        }
        for (int t = 0; t < QT; ++t) {
            mbar_init(&q_full[t], 1);
            for (int s = 0; s < 2; ++s) { mbar_init(&s_full[2 * t + s], 1); mbar_init(&p_full[2 * t + s], 8); }
            mbar_init(&o_done[t], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Value stages start as zeros: rows that no copy fills (pages a window has released, the end of the last
    // tile) meet P = 0, and zero times a finite stale value is 0.  (What K holds there is masked in S.)
    for (int i = threadIdx.x; i < NS * DVH * KV_HALF / 16; i += THREADS)
        reinterpret_cast<uint4*>(sV)[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 18) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_base_p)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_base_p;

    if (warp == 16 || warp == 17) {
        // producers: warp 16 the K tiles (and Q), warp 17 the V tiles
        const bool is_k = warp == 16;
        if (is_k && lane == 0) {
            for (int t = 0; t < tiles_q; ++t) {
                mbar_expect_tx(&q_full[t], DKH * HALF_BYTES);
                for (int hh = 0; hh < DKH; ++hh)
                    tma_load_2d(sQ + (t * DKH + hh) * HALF_BYTES, &maps.q, h * DK + hh * 64, q0 + row_of(t), &q_full[t]);
            }
        }
        const int* table = block_table + (int64_t)b * max_pages;
        const int pages_per_tile = BN / page_size, halves_n = is_k ? DKH : DVH;
        const uint32_t page_bytes = (uint32_t)page_size * 128u;
        // one copy per page and 64-column half: lane = page * halves + half (at most 8 x 4)
        const int pg = lane / halves_n, hh = lane - pg * halves_n;
        const bool mine = pg < pages_per_tile;
        // the lane's page of tile j: inside the request and not released by a window, else -1
        auto page_of = [&](int j) {
            const int kpos = tile_start(j) + pg * page_size;
            return !mine || j >= n_tiles || kpos >= kvl ? -1 : (UNFOLDED ? 0 : __ldg(table + kpos / page_size));
        };
        uint64_t* full = is_k ? k_full : v_full;
        uint64_t* empty = is_k ? k_empty : v_empty;
        uint8_t* base = is_k ? sK : sV;
        int page = page_of(0);
        for (int j = 0; j < n_tiles; ++j) {
            const int next_page = page_of(j + 1);         // on its way while this tile's stage is waited for
            const int s = j % NS;
            bool ok = true;
            if (lane == 0) ok = mbar_wait(&empty[s], ((j / NS) & 1) ^ 1, abort_flag, is_k ? 11 : 21);
            if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            const unsigned have = __ballot_sync(0xffffffffu, page >= 0);
            if (lane == 0) mbar_expect_tx(&full[s], (uint32_t)__popc(have) * page_bytes);
            __syncwarp();
            if (page >= 0) {
                uint8_t* dst = base + (size_t)s * halves_n * KV_HALF + hh * KV_HALF + (size_t)pg * page_bytes;
                if constexpr (UNFOLDED) {
                    const int row = kv_base + tile_start(j) + pg * page_size;
                    if (!is_k) tma_load_2d(dst, &maps.v, h * uf.e + hh * 64, row, &full[s]);
                    else if (hh < dh) tma_load_2d(dst, &maps.k, h * uf.d + hh * 64, row, &full[s]);
                    else tma_load_2d(dst, &maps.kr, (hh - dh) * 64, row, &full[s]);
                } else {
                    tma_load_2d(dst, is_k ? &maps.k : &maps.v, hh * 64, (page * nkv + hk) * page_size, &full[s]);
                }
            }
            page = next_page;
        }
    } else if (warp >= 18) {
        // The whole warp walks through this, one lane issues: what describes the products stays in uniform registers
        // (a single lane's branch moved every descriptor there product by product: 850 cycles for the eight of S).
        const int t = warp - 18;
        if (t < tiles_q) {
            bool ok = *abort_flag == 0 && mbar_wait(&q_full[t], 0, abort_flag, 12);
            ok = __all_sync(0xffffffffu, ok);             // the loops below are the whole warp's
            const int n_mine = tiles_of(t);
            const uint32_t tmem_t = tmem_base + t * COL_TILE;
            // descriptors of the tile origins; an offset of b bytes inside a tile adds b / 16 to the address field
            const uint64_t dq = umma_desc(smem_u32(sQ + (size_t)t * DKH * HALF_BYTES));
            const uint64_t dk0 = umma_desc(smem_u32(sK)), dv0 = umma_desc_mn(smem_u32(sV), KV_HALF);
            // S of tile j goes to buffer j & 1.  P of tile j overwrites S of tile j in place (bfloat16, two
            // keys per 32-bit column) and is the A operand of O += P V straight from tensor memory; S of
            // tile j + 2 goes to the same buffer and is issued once O += P V of tile j is complete.
            auto issue_s = [&](int j) {                   // its K tile is there
                const int s = j % NS, buf = j & 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t dks = dk0 + (uint32_t)((s * DKH * KV_HALF) >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < DK / 16; ++kk) {
                        // columns that neither part fills are left out (what lies in K there is another head's)
                        if (UNFOLDED && !(kk < dh * 4 ? kk < uf.d16 : kk - dh * 4 < uf.r16)) continue;
                        const uint32_t sub = (uint32_t)(kk & 3) * 32;
                        umma_bf16(tmem_t + buf * BN, dq + (((uint32_t)(kk >> 2) * HALF_BYTES + sub) >> 4),
                                  dks + (((uint32_t)(kk >> 2) * KV_HALF + sub) >> 4), IDESC_S, kk > 0 ? 1u : 0u);
                    }
                    umma_commit(&s_full[2 * t + buf]);
                    umma_commit(&k_empty[s]);             // this query tile has read the K stage once these MMAs have run
                }
                __syncwarp();
            };
            auto k_there = [&](int j) { return mbar_wait(&k_full[j % NS], (j / NS) & 1, abort_flag, 13); };
            for (int j = 0; j < 2 && j < n_mine && ok; ++j) {
                ok = __all_sync(0xffffffffu, k_there(j));
                if (ok) issue_s(j);
            }
            for (int j = 0; j < n_mine && ok; ++j) {
                const int s = j % NS, buf = j & 1;
                ok = mbar_wait(&v_full[s], (j / NS) & 1, abort_flag, 16) &&
                     mbar_wait(&p_full[2 * t + buf], (j >> 1) & 1, abort_flag, 15);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t dvs = dv0 + (uint32_t)((s * DVH * KV_HALF) >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < BN / 16; ++ks) // 16 keys of P are 8 columns of tensor memory
                        umma_bf16_tmem_a(tmem_t + COL_O, tmem_t + buf * BN + ks * 8,
                                         dvs + (((uint32_t)ks * 2048) >> 4), IDESC_PV, (j > 0 || ks > 0) ? 1u : 0u);
                    umma_commit(&o_done[t]);              // O holds tile j
                    umma_commit(&v_empty[s]);             // ... and has read the V stage
                }
                __syncwarp();
                if (j + 2 < n_mine) {
                    ok = k_there(j + 2) && mbar_wait(&o_done[t], j & 1, abort_flag, 14);
                    ok = __all_sync(0xffffffffu, ok);
                    if (ok) issue_s(j + 2);
                }
            }
            // key tiles that only the other query tile reads: passed on as they arrive
            for (int j = n_mine; j < n_tiles && ok; ++j) {
                const int s = j % NS;
                ok = k_there(j) && mbar_wait(&v_full[s], (j / NS) & 1, abort_flag, 16);
                ok = __all_sync(0xffffffffu, ok);
                if (ok && elect_one()) { mbar_arrive(&k_empty[s]); mbar_arrive(&v_empty[s]); }
                __syncwarp();
            }
        }
    } else if ((warp >> 3) < tiles_q) {
        // softmax and epilogue: two threads to a query row (= lane of tensor memory), one half of a tile's keys each
        const int t = warp >> 3, quarter = warp & 3, half = (warp >> 2) & 1, my0 = half * HK;
        const int r = quarter * 32 + lane, pair_id = 1 + 4 * t + quarter;
        const uint32_t lane_addr = tmem_base + t * COL_TILE + ((uint32_t)(quarter * 32) << 16);
        const int tile_row0 = row_of(t), nq = rows_of(t), n_mine = tiles_of(t);
        const int p_lo = pos0 + tile_row0 / hpq;          // position of the tile's first query
        const int p_hi = p_lo + (nq - 1) / hpq;
        const int p_row = p_lo + r / hpq;                 // position of this thread's query
        const int vis_hi = min(p_row, kvl - 1);           // last visible key
        const int vis_lo = first_visible(p_row, window, form.chunk);   // first visible key
        const int tile_vis_lo = first_visible(p_hi, window, form.chunk);
        float* meet = halves + t * 4 * BQ;                // [2 in turn][2 halves][BQ]
        float m_ref = sink ? (form.sink_score ? form.sink_score[h] * 1.4426950408889634f : 0.f) : -INFINITY;   // reference of the exponentials, in log2 units
        float l_run = sink && half == 0 ? 1.f : 0.f;
        bool ok = true, together = true;                  // until both halves leave early, at a meeting
        for (int j = 0; j < n_mine; ++j) {
            const int buf = j & 1;
            const int k0 = tile_start(j) + my0;
            ok = ok && mbar_wait(&s_full[2 * t + buf], (j >> 1) & 1, abort_flag, 17);
            ok = __all_sync(0xffffffffu, ok);             // tcgen05.ld and .st are warp-wide: all lanes or none
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // the half's row of S to registers; once both halves have it, its place may take P
            uint32_t v[HK];
            const uint32_t s_addr = lane_addr + buf * BN;
            if (ok) {
                tmem_ld32(s_addr + my0, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            } else {
#pragma unroll
                for (int i = 0; i < HK; ++i) v[i] = 0u;
            }
            if constexpr (CAPPED) {
#pragma unroll
                for (int i = 0; i < HK; ++i)
                    v[i] = __float_as_uint(fast_tanh(__uint_as_float(v[i]) * cap_in) * cap_out);
            }
            // does any (row, key) of this half need the mask?
            const bool masked = (k0 + HK - 1 > p_lo) || (k0 + HK > kvl) || (bounded && k0 < tile_vis_lo);
            // below a row's window only kept first keys are visible: of a tile of kept first keys those below
            // sink_end (such a tile lies below every window, so it is always masked key by key), of a window's
            // tile those below keep_first
            const int keep_lim = j < n_sink ? sink_end : keep_first;
            uint32_t pk[HK / 2];
            float alpha = 1.f;
            if constexpr (LOGISTIC) {
                ok = together = pair_and(pair_id, ok);    // both halves have read S (or one gave up: both leave)
                if (!ok) break;
                // logistic(x) = 1 / (1 + 2^(-x log2 e)); the exponent is bounded so that the power stays finite
                const float hb = head_bias[h] * 1.4426950408889634f;
#pragma unroll
                for (int i = 0; i < HK; i += 2) {
                    float w0 = __fdividef(1.0f, 1.0f + fast_exp2(fminf(-fmaf(__uint_as_float(v[i]), scale_log2, hb), 80.f)));
                    float w1 = __fdividef(1.0f, 1.0f + fast_exp2(fminf(-fmaf(__uint_as_float(v[i + 1]), scale_log2, hb), 80.f)));
                    if (masked) {
                        const int kj = k0 + i;
                        if (kj > vis_hi || (kj < vis_lo && kj >= keep_lim)) w0 = 0.f;
                        if (kj + 1 > vis_hi || (kj + 1 < vis_lo && kj + 1 >= keep_lim)) w1 = 0.f;
                    }
                    pk[i >> 1] = pack_bf16(w0, w1);
                }
            } else {
                float mxs[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four chains, not one of HK steps
                if (masked) {
#pragma unroll
                    for (int i = 0; i < HK; ++i) {
                        const int kj = k0 + i;
                        if (kj > vis_hi || (kj < vis_lo && kj >= keep_lim)) v[i] = 0xff800000u;   // -inf
                    }
                }
#pragma unroll
                for (int i = 0; i < HK; ++i) mxs[i & 3] = fmaxf(mxs[i & 3], __uint_as_float(v[i]));
                // the scale is positive: the maximum of the scaled scores is the scaled maximum
                const float mine = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])) * scale_log2;
                float* at = meet + buf * 2 * BQ + r;      // (the other half has read this place two barriers ago)
                at[half * BQ] = mine;
                ok = together = pair_and(pair_id, ok);    // both halves have read S and left their maxima (or one gave
                if (!ok) break;                           // up: both leave)
                const float mx = fmaxf(mine, at[(half ^ 1) * BQ]);
                // the reference follows the maximum only when that moved by more than 8: exponentials stay
                // below 2^8, and O needs scaling only then
                if (mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY)) {
                    alpha = m_ref == -INFINITY ? 0.f : fast_exp2(m_ref - mx);
                    m_ref = mx;
                }
                const float base = m_ref == -INFINITY ? 0.f : m_ref;
                float2 sums[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int i = 0; i < HK; i += 2) {
                    float2 e = fma_two(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), scale_log2, -base);
                    e.x = fast_exp2(e.x); e.y = fast_exp2(e.y);
                    sums[(i >> 1) & 1] = add_two(sums[(i >> 1) & 1], e);
                    pk[i >> 1] = pack_bf16(e.x, e.y);
                }
                l_run = l_run * alpha + ((sums[0].x + sums[0].y) + (sums[1].x + sums[1].y));
            }
            // O is scaled only after O += P V of tile j - 1, and the last tile waits for that product in any case: see
            // follows_product.
            const bool rescale = !LOGISTIC && j > 0 && !__all_sync(0xffffffffu, alpha == 1.f);
            if (follows_product(j, n_mine, rescale)) {
                ok = mbar_wait(&o_done[t], (j - 1) & 1, abort_flag, rescale ? 18 : 19);
                ok = __all_sync(0xffffffffu, ok);
            }
            if (ok && rescale) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c0 = half * (DV / 2); c0 < (half + 1) * (DV / 2); c0 += 32) {
                    uint32_t o[32];
                    tmem_ld32(lane_addr + COL_O + c0, o);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tmem_st32(lane_addr + COL_O + c0, o);
                }
            }
            // P over S in place: 64 keys are 32 columns of two bfloat16 each
            if (ok) {
                tmem_st16(s_addr + half * (HK / 2), pk);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full[2 * t + buf]);
            }
        }
        if (together) {
            // the product before was seen complete ahead of the last hand-over: the barrier is in phase n - 1 or n
            ok = ok && mbar_wait(&o_done[t], (n_mine - 1) & 1, abort_flag, 20);
            ok = __all_sync(0xffffffffu, ok);
            // the halves' sums meet where the maxima of a tile more would
            float* at = meet + (n_mine & 1) * 2 * BQ + r;
            at[half * BQ] = l_run;
            ok = pair_and(pair_id, ok);
            l_run = at[0] + at[BQ];
        }
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float inv = LOGISTIC ? 1.f : (l_run > 0.f ? 1.f / l_run : 0.f);
            if (form.gate && r < nq) inv *= head_gate(form, q0 + tile_row0 + r, h);
            const int ev = UNFOLDED ? uf.e : DV;          // columns of a value (a multiple of 8)
            __nv_bfloat16* dst = out + ((int64_t)(q0 + tile_row0 + r) * nh + h) * ev;
            const float* gt = UNFOLDED && uf.gate && r < nq
                                  ? uf.gate + (int64_t)(q0 + tile_row0 + r) * uf.ldg + uf.gcol + h * ev : nullptr;
#pragma unroll 1
            for (int c0 = half * (DV / 2); c0 < (half + 1) * (DV / 2); c0 += 32) {
                uint32_t o[32];
                tmem_ld32(lane_addr + COL_O + c0, o);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (r < nq) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        if (UNFOLDED && c0 + i >= ev) continue;
                        if (UNFOLDED && gt) {
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                o[i + k] = __float_as_uint(__fdividef(__uint_as_float(o[i + k]), 1.0f + __expf(-__ldg(gt + c0 + i + k))));
                        }
                        uint4 w;
                        w.x = pack_bf16(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
                        w.y = pack_bf16(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
                        w.z = pack_bf16(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
                        w.w = pack_bf16(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + c0 + i) = w;
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 18) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    if (threadIdx.x == 0 && *abort_p != 0) atomicMax(status, *abort_p);
}

// Row-major bfloat16 matrix [rows, cols] with a row pitch of `pitch` elements, box of 64 columns x
// box_rows rows, 128-byte swizzle.
static bool make_map_pitched(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch,
                             uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {pitch * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace pt
}  // namespace mi

using namespace mi;

extern "C" {

// 1 if the tcgen05 prefill attention takes this geometry: head size 64 or 128; pages of 8, 16, 32 or 64
// tokens (a page is one TMA box of whole 8-row swizzle groups, and pages tile a key tile).
int mi_attn_prefill_tc_supported(int d, int page_size) {
    const bool ps_ok = page_size >= 8 && page_size <= pt::BN && (page_size & (page_size - 1)) == 0;
    return ((d == 64 || d == 128) && ps_ok) ? 1 : 0;
}

// q [T, nh, d], out [T, nh, d] bfloat16; k_cache, v_cache one layer's [num_pages, nkv, page_size, d].
// `status` (device int, zero before the first call) receives a non-zero code if a wait inside the
// kernel ran out.
int mi_attn_prefill_tc(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                       const int* q_start, const int* kv_len, void* out, int* status, int T, int B, int max_q_len,
                       int nh, int nkv, int d, int page_size, int num_pages, int max_pages, int window, float scale,
                       int keep_first, float cap, int sink, int chunk, const float* sink_score, const float* gate,
                       int64_t ld_gate, cudaStream_t stream) {
    if (B <= 0 || max_q_len <= 0 || T <= 0) return kOk;
    if (chunk < 0 || (chunk > 0 && window > 0) || (sink_score && !sink)) {
        set_last_error("prefill attention (tcgen05): chunks of %d go without a window (%d), a sink's scores with a sink", chunk, window);
        return kBadShape;
    }
    const AttnForm form = {chunk, sink_score, gate, ld_gate};
    if (cap < 0.f || !(scale > 0.f)) {
        set_last_error("prefill attention (tcgen05): a cap of %g on scores scaled by %g", (double)cap, (double)scale);
        return kBadShape;
    }
    if (keep_first < 0) { set_last_error("prefill attention (tcgen05): %d kept first keys", keep_first); return kBadShape; }
    if (!mi_attn_prefill_tc_supported(d, page_size)) {
        set_last_error("prefill attention (tcgen05): head_dim %d with pages of %d tokens is not taken", d, page_size);
        return kBadShape;
    }
    if (nkv < 1 || nh % nkv != 0) {
        set_last_error("attention: %d query heads are not a multiple of %d key/value heads", nh, nkv);
        return kBadShape;
    }
    if (B > 65535 || nh > 65535) {
        set_last_error("attention: batch %d or head count %d exceeds the grid limit 65535", B, nh);
        return kBadShape;
    }
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
         reinterpret_cast<uintptr_t>(out)) & 15) {
        set_last_error("prefill attention (tcgen05): operands must be 16-byte aligned");
        return kBadShape;
    }
    pt::Maps maps = {};
    const uint64_t cache_rows = (uint64_t)num_pages * nkv * page_size;
    bool ok = pt::make_map_pitched(&maps.q, q, (uint64_t)T, (uint64_t)nh * d, (uint64_t)nh * d, pt::BQ) &&
              pt::make_map_pitched(&maps.k, k_cache, cache_rows, (uint64_t)d, (uint64_t)d, (uint32_t)page_size) &&
              pt::make_map_pitched(&maps.v, v_cache, cache_rows, (uint64_t)d, (uint64_t)d, (uint32_t)page_size);
    if (!ok) {
        set_last_error("prefill attention (tcgen05): cuTensorMapEncodeTiled failed");
        return kLaunchFailed;
    }
    const pt::QueryTiles order = pt::query_order(max_q_len, T, nh, B, d, window > 0 || chunk > 0);
    const dim3 grid(pt::grid_x(max_q_len, nh, order), 1, B);
    const float scale_log2 = scale * 1.4426950408889634f;
    const size_t smem = d == 64 ? pt::smem_bytes(64, 64) : pt::smem_bytes(128, 128);
    const float cap_in = cap > 0.f ? scale / cap : 0.f, cap_out = cap > 0.f ? cap / scale : 0.f;
#define MI_PT(DD, CC)                                                                                     \
    do {                                                                                                  \
        auto kern = pt::attn_prefill_tc_kernel<DD, DD, CC>;                                               \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);               \
        kern<<<grid, pt::THREADS, smem, stream>>>(maps, block_table, q_start, kv_len, (__nv_bfloat16*)out, nh,    \
                                          nkv, page_size, max_pages, window, scale_log2, status,          \
                                          keep_first, 1, cap_in, cap_out, sink, nullptr, pt::Unfolded{}, form, order);           \
    } while (0)
    if (cap > 0.f) { if (d == 64) MI_PT(64, true); else MI_PT(128, true); }
    else { if (d == 64) MI_PT(64, false); else MI_PT(128, false); }
#undef MI_PT
    return finish_launch("attn_prefill_tc");
}

// The same kernel with logistic key weights that are not normalised (see LOGISTIC above): key and value heads of
// 64 or 128 numbers each, not necessarily alike; q [T, nh, dk], out [T, nh, dv]; head_bias float [nh].
int mi_attn_prefill_tc_logistic_supported(int dk, int dv, int page_size) {
    return (dk == 64 || dk == 128) && (dv == 64 || dv == 128) && mi_attn_prefill_tc_supported(64, page_size);
}

int mi_attn_prefill_tc_logistic(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                                const int* q_start, const int* kv_len, void* out, int* status, int T, int B,
                                int max_q_len, int nh, int nkv, int dk, int dv, int page_size, int num_pages,
                                int max_pages, int window, float scale, const float* head_bias, cudaStream_t stream) {
    if (B <= 0 || max_q_len <= 0 || T <= 0) return kOk;
    if (!mi_attn_prefill_tc_logistic_supported(dk, dv, page_size) || !head_bias || !(scale > 0.f)) {
        set_last_error("prefill attention with logistic weights (tcgen05): keys of %d, values of %d, pages of %d tokens "
                       "are not taken, or the heads' biases are missing", dk, dv, page_size);
        return kBadShape;
    }
    if (nkv < 1 || nh % nkv != 0 || B > 65535 || nh > 65535) {
        set_last_error("attention: %d query heads over %d key/value heads, batch %d", nh, nkv, B);
        return kBadShape;
    }
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
         reinterpret_cast<uintptr_t>(out)) & 15) {
        set_last_error("prefill attention (tcgen05): operands must be 16-byte aligned");
        return kBadShape;
    }
    pt::Maps maps = {};
    const uint64_t cache_rows = (uint64_t)num_pages * nkv * page_size;
    bool ok = pt::make_map_pitched(&maps.q, q, (uint64_t)T, (uint64_t)nh * dk, (uint64_t)nh * dk, pt::BQ) &&
              pt::make_map_pitched(&maps.k, k_cache, cache_rows, (uint64_t)dk, (uint64_t)dk, (uint32_t)page_size) &&
              pt::make_map_pitched(&maps.v, v_cache, cache_rows, (uint64_t)dv, (uint64_t)dv, (uint32_t)page_size);
    if (!ok) {
        set_last_error("prefill attention (tcgen05): cuTensorMapEncodeTiled failed");
        return kLaunchFailed;
    }
    const pt::QueryTiles order = pt::query_order(max_q_len, T, nh, B, dk, window > 0);
    const dim3 grid(pt::grid_x(max_q_len, nh, order), 1, B);
    const float scale_log2 = scale * 1.4426950408889634f;
#define MI_PTL(KK, VV)                                                                                    \
    do {                                                                                                  \
        auto kern = pt::attn_prefill_tc_kernel<KK, VV, false, true>;                                      \
        const size_t smem = pt::smem_bytes(KK, VV);                                                       \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);               \
        kern<<<grid, pt::THREADS, smem, stream>>>(maps, block_table, q_start, kv_len, (__nv_bfloat16*)out, nh,    \
                                          nkv, page_size, max_pages, window, scale_log2, status, 0, 1,    \
                                          0.f, 0.f, 0, head_bias, pt::Unfolded{}, AttnForm{}, order);                            \
    } while (0)
    if (dk == 64) { if (dv == 64) MI_PTL(64, 64); else MI_PTL(64, 128); }
    else { if (dv == 64) MI_PTL(128, 64); else MI_PTL(128, 128); }
#undef MI_PTL
    return finish_launch("attn_prefill_tc");
}

// The same kernel for heads that all read ONE key/value head whose values are the first `dv` numbers of its key
// rows (attention through a latent with the key matrices folded into the queries): q [T, H, dk], cache one layer's
// [num_pages, 1, page_size, dk], out [T, H, dv] bfloat16.  The rows of a query tile are (query, head) pairs, so
// a key tile is fetched once for all heads.  Takes H a divisor of 128, dv 64 or 128, dk a multiple of 8 of at
// most 256 (rounded up to whole 64-column halves that read zeros beyond dk) and the page sizes of the kernel.
int mi_attn_prefill_tc_shared_supported(int H, int dk, int dv, int page_size) {
    return H >= 1 && H <= 128 && 128 % H == 0 && (dv == 64 || dv == 128) && dk >= dv && dk <= 256 && dk % 8 == 0 &&
           mi_attn_prefill_tc_supported(64, page_size);
}

int mi_attn_prefill_tc_shared(const void* q, const void* cache, const int* block_table, const int* q_start,
                              const int* kv_len, void* out, int* status, int T, int B, int max_q_len, int H, int dk,
                              int dv, int page_size, int num_pages, int max_pages, int window, float scale,
                              int keep_first, cudaStream_t stream) {
    if (B <= 0 || max_q_len <= 0 || T <= 0) return kOk;
    if (!mi_attn_prefill_tc_shared_supported(H, dk, dv, page_size) || keep_first < 0) {
        set_last_error("prefill attention over a shared head (tcgen05): %d heads, rows of %d, values of %d, pages of %d "
                       "tokens are not taken", H, dk, dv, page_size);
        return kBadShape;
    }
    if (B > 65535) { set_last_error("attention: batch %d exceeds the grid limit 65535", B); return kBadShape; }
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15) {
        set_last_error("prefill attention (tcgen05): operands must be 16-byte aligned");
        return kBadShape;
    }
    pt::Maps maps = {};
    const uint64_t cache_rows = (uint64_t)num_pages * page_size;
    bool ok = pt::make_map_pitched(&maps.q, q, (uint64_t)T * H, (uint64_t)dk, (uint64_t)dk, pt::BQ) &&
              pt::make_map_pitched(&maps.k, cache, cache_rows, (uint64_t)dk, (uint64_t)dk, (uint32_t)page_size) &&
              pt::make_map_pitched(&maps.v, cache, cache_rows, (uint64_t)dv, (uint64_t)dk, (uint32_t)page_size);
    if (!ok) {
        set_last_error("prefill attention (tcgen05): cuTensorMapEncodeTiled failed");
        return kLaunchFailed;
    }
    const int DKr = (dk + 63) / 64 * 64;
    const pt::QueryTiles order = pt::query_order((int64_t)max_q_len * H, (int64_t)T * H, 1, B, DKr, window > 0);
    const dim3 grid(pt::grid_x((int64_t)max_q_len * H, 1, order), 1, B);
    const float scale_log2 = scale * 1.4426950408889634f;
#define MI_PTS(KK, VV)                                                                                    \
    do {                                                                                                  \
        auto kern = pt::attn_prefill_tc_kernel<KK, VV>;                                                   \
        const size_t smem = pt::smem_bytes(KK, VV);                                                       \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);               \
        kern<<<grid, pt::THREADS, smem, stream>>>(maps, block_table, q_start, kv_len, (__nv_bfloat16*)out, 1, 1,  \
                                          page_size, max_pages, window, scale_log2, status, keep_first, H,  \
                                          0.f, 0.f, 0, nullptr, pt::Unfolded{}, AttnForm{}, order);                                \
    } while (0)
    if (dv == 64) {
        if (DKr == 64) MI_PTS(64, 64); else if (DKr == 128) MI_PTS(128, 64); else if (DKr == 192) MI_PTS(192, 64); else MI_PTS(256, 64);
    } else {
        if (DKr == 128) MI_PTS(128, 128); else if (DKr == 192) MI_PTS(192, 128); else MI_PTS(256, 128);
    }
#undef MI_PTS
    return finish_launch("attn_prefill_tc");
}

// The same kernel over keys and values that were formed from latents before the call (see Unfolded): q [T, nh, DK] with
// DK = 64 (ceil(d / 64) + ceil(r / 64)), the rotated part from column 64 ceil(d / 64) on, zeros up to the next multiple
// of 16 behind each part; kv [rows, kv_pitch] with the unrotated keys of the heads from column 0 and their values from
// column v_col on; k_rot [rows, r_pitch]; out [T, nh, e].  `kv_len` gives the contexts that follow one another in the
// rows.  Takes d and e multiples of 8, values up to 128, DK up to 256.
int mi_attn_prefill_tc_unfolded_supported(int d, int r, int e) {
    if (d < 8 || d % 8 || r < 2 || r % 2 || e < 8 || e % 8 || e > 128) return 0;
    return (d + 63) / 64 + (r + 63) / 64 <= 4;
}

int mi_attn_prefill_tc_unfolded(const void* q, const void* kv, const void* k_rot, const int* q_start,
                                const int* kv_len, void* out, int* status, int T, int B, int max_q_len, int nh, int d,
                                int r, int e, int rows, int kv_pitch, int v_col, int r_pitch, int window, float scale,
                                const float* gate, int ldg, int gcol, cudaStream_t stream) {
    if (B <= 0 || max_q_len <= 0 || T <= 0) return kOk;
    if (!mi_attn_prefill_tc_unfolded_supported(d, r, e) || nh < 1 || nh > 65535 || B > 65535 || rows < 1 ||
        kv_pitch % 8 || v_col % 8 || v_col < nh * d || kv_pitch < v_col + nh * e || r_pitch % 8 || r_pitch < r ||
        !(scale > 0.f) || window < 0 || (gate && (gcol < 0 || gcol + nh * e > ldg))) {
        set_last_error("prefill attention over unfolded latents (tcgen05): %d heads of %d + %d, values of %d are not taken",
                       nh, d, r, e);
        return kBadShape;
    }
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kv) | reinterpret_cast<uintptr_t>(k_rot) |
         reinterpret_cast<uintptr_t>(out)) & 15) {
        set_last_error("prefill attention (tcgen05): operands must be 16-byte aligned");
        return kBadShape;
    }
    const int DKr = ((d + 63) / 64 + (r + 63) / 64) * 64, DVr = (e + 63) / 64 * 64;
    pt::Maps maps = {};
    const __nv_bfloat16* kvp = (const __nv_bfloat16*)kv;
    bool ok = pt::make_map_pitched(&maps.q, q, (uint64_t)T, (uint64_t)nh * DKr, (uint64_t)nh * DKr, pt::BQ) &&
              pt::make_map_pitched(&maps.k, kvp, (uint64_t)rows, (uint64_t)nh * d, (uint64_t)kv_pitch, pt::BN) &&
              pt::make_map_pitched(&maps.v, kvp + v_col, (uint64_t)rows, (uint64_t)nh * e, (uint64_t)kv_pitch, pt::BN) &&
              pt::make_map_pitched(&maps.kr, k_rot, (uint64_t)rows, (uint64_t)r, (uint64_t)r_pitch, pt::BN);
    if (!ok) {
        set_last_error("prefill attention (tcgen05): cuTensorMapEncodeTiled failed");
        return kLaunchFailed;
    }
    const pt::Unfolded uf = {(d + 15) / 16, (r + 15) / 16, d, e, gate, ldg, gcol};
    const pt::QueryTiles order = pt::query_order(max_q_len, T, nh, B, DKr, window > 0);
    const dim3 grid(pt::grid_x(max_q_len, nh, order), 1, B);
    const float scale_log2 = scale * 1.4426950408889634f;
#define MI_PTU(KK, VV)                                                                                    \
    do {                                                                                                  \
        const size_t smem = pt::smem_bytes(KK, VV);                                                       \
        auto kern = pt::attn_prefill_tc_kernel<KK, VV, false, false, true>;                               \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);               \
        kern<<<grid, pt::THREADS, smem, stream>>>(maps, nullptr, q_start, kv_len, (__nv_bfloat16*)out, nh, nh, \
                                          pt::BN, 0, window, scale_log2, status, 0, 1, 0.f, 0.f, 0,       \
                                          nullptr, uf, AttnForm{}, order);                                                   \
    } while (0)
    if (DVr == 64) {
        if (DKr == 128) MI_PTU(128, 64); else if (DKr == 192) MI_PTU(192, 64); else MI_PTU(256, 64);
    } else {
        if (DKr == 128) MI_PTU(128, 128); else if (DKr == 192) MI_PTU(192, 128); else MI_PTU(256, 128);
    }
#undef MI_PTU
    return finish_launch("attn_prefill_tc");
}

}  // extern "C"
