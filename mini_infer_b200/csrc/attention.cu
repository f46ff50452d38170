// Attention over the paged cache for a ragged batch: every request brings
// q_len new query tokens (a portion of a prompt, or one decoded token) that sit
// at the tail of its kv_len cached keys.
//
// The reference runs one block per (request, head, query token) and walks all
// pages of the request with scalar dot products, for prefill and decode alike
// (src/kernels/paged_attn_kernel.cu:102-288), accepts head sizes 64 and 128
// only (:313-315) and masks causally only in "prefill" mode (:228-231).
// Here: a tiled kernel for any head size up to 256 (float arithmetic, used by
// the 32-bit path and as the fallback of the bfloat16 path) and a split-KV
// decode kernel with a merge step.  Masking is positional in all cases:
// key j is visible from the query at absolute position p iff j <= p and
// (window == 0 or j > p - window)  (same rule as :228-236); the decode kernel
// also knows chunks, an added key with a score per head and a gate per head (AttnForm).
//
// Cache layout per layer: [page, kv_head, page_size, d]; block_table[b, i] is
// the page of keys [i*page_size, (i+1)*page_size) of request b, or -1 once a
// window has passed it.

#include "f32_tiles.cuh"

namespace mi {

// ---------------------------------------------------------------------------
// Tiled kernel.  Block = 128 threads, 16 queries of one head, key tiles of 32
// aligned to absolute positions (so the order of a row's additions does not
// depend on where a portion starts, up to the first tile under a window).
// ---------------------------------------------------------------------------
constexpr int TQ = 16;   // queries per block
constexpr int TK = 32;   // keys per tile

template <typename AT, int ND>  // ND = ceil(d / 8) accumulators per thread
__global__ void __launch_bounds__(128)
attn_tiled_kernel(const AT* __restrict__ q, const AT* __restrict__ k_cache, const AT* __restrict__ v_cache,
                  const int* __restrict__ block_table, const int* __restrict__ q_start,
                  const int* __restrict__ kv_len, AT* __restrict__ out, int nh, int nkv, int d,
                  int page_size, int max_pages, int window, float scale) {
    extern __shared__ float smem[];
    const int b = blockIdx.z, h = blockIdx.y, qt = blockIdx.x;
    const int q0 = q_start[b], q_len = q_start[b + 1] - q0;
    if (qt * TQ >= q_len) return;
    const int kvl = kv_len[b];
    const int hk = h / (nh / nkv);
    const int tid = threadIdx.x;
    const int dp = d + 1;
    float* Qs = smem;                       // [TQ][d+1]
    float* Ks = Qs + TQ * dp;               // [TK][d+1]
    float* Vs = Ks + TK * dp;               // [TK][d]
    float* Ss = Vs + TK * d;                // [TQ][TK+1]
    __shared__ int64_t row_off[TK];

    const int nq = min(TQ, q_len - qt * TQ);
    // absolute position of local query i of this tile
    const int p_lo = kvl - q_len + qt * TQ;
    const int p_hi = p_lo + nq - 1;

    for (int idx = tid; idx < TQ * d; idx += 128) {
        const int i = idx / d, c = idx - i * d;
        float v = 0.f;
        if (i < nq) v = to_float(q[((int64_t)(q0 + qt * TQ + i) * nh + h) * d + c]) * scale;
        Qs[i * dp + c] = v;
    }

    const int qi = tid >> 3;       // query row of this thread (0..15)
    const int sub = tid & 7;       // position among the 8 threads of the row
    const int my_pos = p_lo + qi;  // meaningful when qi < nq
    float m_run = -INFINITY, l_run = 0.f;
    float acc[ND];
#pragma unroll
    for (int j = 0; j < ND; ++j) acc[j] = 0.f;

    int k_begin = 0;
    if (window > 0) k_begin = max(0, p_lo - window + 1);
    k_begin = (k_begin / TK) * TK;
    const int k_end = min(kvl, p_hi + 1);
    const int* table = block_table + (int64_t)b * max_pages;

    for (int kt = k_begin; kt < k_end; kt += TK) {
        __syncthreads();  // previous tile fully consumed (and Qs written, first time)
        if (tid < TK) {
            const int kj = kt + tid;
            int64_t off = -1;
            if (kj < k_end) {
                const int page = table[kj / page_size];
                if (page >= 0)
                    off = ((int64_t)page * nkv + hk) * page_size * d + (int64_t)(kj % page_size) * d;
            }
            row_off[tid] = off;
        }
        __syncthreads();
        for (int idx = tid; idx < TK * d; idx += 128) {
            const int r = idx / d, c = idx - r * d;
            const int64_t off = row_off[r];
            float kv = 0.f, vv = 0.f;
            if (off >= 0) { kv = to_float(k_cache[off + c]); vv = to_float(v_cache[off + c]); }
            Ks[r * dp + c] = kv;
            Vs[r * d + c] = vv;
        }
        __syncthreads();
        // scores: this thread owns keys sub, sub+8, sub+16, sub+24 of row qi
        float s[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int kr = sub + 8 * j;
            const int kj = kt + kr;
            float dot = 0.f;
            const float* qrow = Qs + qi * dp;
            const float* krow = Ks + kr * dp;
            for (int c = 0; c < d; ++c) dot += qrow[c] * krow[c];
            const bool vis = (qi < nq) && (kj <= my_pos) && (window == 0 || kj > my_pos - window) &&
                             (row_off[kr] >= 0);
            s[j] = vis ? dot : -INFINITY;
        }
        float tmax = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        const float m_new = fmaxf(m_run, tmax);
        float alpha = 1.f, psum = 0.f;
        if (m_new == -INFINITY) {
#pragma unroll
            for (int j = 0; j < 4; ++j) Ss[qi * (TK + 1) + sub + 8 * j] = 0.f;
        } else {
            alpha = expf(m_run - m_new);  // m_run = -inf gives 0
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = expf(s[j] - m_new);
                Ss[qi * (TK + 1) + sub + 8 * j] = p;
                psum += p;
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
        l_run = l_run * alpha + psum;
        m_run = m_new;
        __syncwarp();  // the 8 threads of a row live in one warp: their Ss writes are visible
        const float* prow = Ss + qi * (TK + 1);
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            const int c = sub + 8 * j;
            if (c < d) {
                float a = acc[j] * alpha;
                for (int kr = 0; kr < TK; ++kr) a += prow[kr] * Vs[kr * d + c];
                acc[j] = a;
            }
        }
    }
    if (qi < nq) {
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        AT* o = out + ((int64_t)(q0 + qt * TQ + qi) * nh + h) * d;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            const int c = sub + 8 * j;
            if (c < d) o[c] = from_float<AT>(acc[j] * inv);
        }
    }
}

// ---------------------------------------------------------------------------
// The same in 32 bits for heads of 64 and 128: 32 queries of one head per block of 2 x 4 warps, key tiles of 32 at the same
// absolute positions, one order of additions for every row whatever its step: a dot product is one chain of fused
// multiply-adds over the head's numbers, an output one chain over the keys of a tile after its scaling; the tiles of even
// and of odd number are walked side by side, by four warps each, and the two walks' rows meet at the end.  A warp owns 8
// queries through both products (no block-wide barrier between them), with 2 x 4 scores and then 4 x (D / 16) outputs a
// thread, two of these per instruction; it passes over tiles that none of its queries sees.  512 queries of 16 heads of
// 128 behind 700 keys: 196 us in one walk of four warps with two buffers, 184 us in two with a buffer each (16 queries a
// warp, with a third fewer reads of shared memory per product, 187 us); 876 us with the kernel above, which reads a pair of
// operands per multiply-add.
// ---------------------------------------------------------------------------
constexpr int FQ = 32, FK = 32;

template <int D> constexpr size_t rows_f32_smem() {
    return sizeof(float) * (FQ * (D + 4) + 2 * (FK * (D + 4) + FK * D) + 2 * (FQ * FK + FQ)) + sizeof(int) * 2 * FK;
}

template <int D>
__global__ void __launch_bounds__(256, 2)
attn_rows_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                     const int* __restrict__ block_table, const int* __restrict__ q_start, const int* __restrict__ kv_len,
                     float* __restrict__ out, int nh, int nkv, int page_size, int max_pages, int window, float scale) {
    extern __shared__ __align__(16) float smem[];
    constexpr int QP = D + 4, NC = D / 64;         // row pitch of queries and keys; 16-byte groups of outputs a thread
    const int b = blockIdx.z, h = blockIdx.y, qt = gridDim.x - 1 - blockIdx.x;    // the longest rows first
    const int q0 = q_start[b], q_len = q_start[b + 1] - q0;
    if (qt * FQ >= q_len) return;
    const int kvl = kv_len[b], hk = h / (nh / nkv);
    const int walk = threadIdx.x >> 7, tid = threadIdx.x & 127, warp = tid >> 5, lane = tid & 31;
    float* Qs = smem;                              // [FQ][QP]
    float* Ks = Qs + FQ * QP + walk * FK * (QP + D);      // the walk's [FK][QP]
    float* Vs = Ks + FK * QP;                      // ... and [FK][D]
    float* behind = Qs + FQ * QP + 2 * FK * (QP + D);
    float* Ps = behind + (walk * 4 + warp) * 8 * FK;      // the warp's [FK][8]: key, query
    float* As = behind + 2 * FQ * FK + (walk * 4 + warp) * 8;     // the warp's 8 factors
    int* there = reinterpret_cast<int*>(behind + 2 * FQ * FK + 2 * FQ) + walk * FK;      // [FK]: the key has a page
    auto walk_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + walk) : "memory"); };

    const int nq = min(FQ, q_len - qt * FQ);
    const int p_lo = kvl - q_len + qt * FQ;        // position of the block's first query
    const int k_end = min(kvl, p_lo + nq);
    int k_begin = window > 0 ? max(0, p_lo - window + 1) : 0;
    k_begin = (k_begin / FK) * FK;
    const int* table = block_table + (int64_t)b * max_pages;

    auto ask = [&](int kt) {              // 4 threads a key row
        const int r = tid >> 2, kj = kt + r;
        int page = -1;
        if (kj < k_end) page = __ldg(table + kj / page_size);
        const bool in = page >= 0;
        const int64_t off = in ? (((int64_t)page * nkv + hk) * page_size + kj % page_size) * D : 0;
        if ((tid & 3) == 0) there[r] = in;
        const uint32_t kd = (uint32_t)__cvta_generic_to_shared(Ks + r * QP);
        const uint32_t vd = (uint32_t)__cvta_generic_to_shared(Vs + r * D);
        const int n = in ? 16 : 0;                 // nothing read: zeros
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
            const int c = ((tid & 3) + 4 * i) * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(kd + c * 4), "l"(k_cache + off + c), "r"(n) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(vd + c * 4), "l"(v_cache + off + c), "r"(n) : "memory");
        }
    };

    for (int idx = threadIdx.x; idx < FQ * (D / 4); idx += 256) {
        const int i = idx / (D / 4), c = idx - i * (D / 4);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < nq) v = __ldg(reinterpret_cast<const float4*>(q + ((int64_t)(q0 + qt * FQ + i) * nh + h) * D) + c);
        v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
        *reinterpret_cast<float4*>(Qs + i * QP + c * 4) = v;
    }

    // scores: queries sr, sr + 1 of the warp, keys sub + 8 j; outputs: queries orow .. orow + 3, 4 numbers from each oc + 64 i
    const int sub = lane & 7, sr = (lane >> 3) * 2, orow = (lane >> 4) * 4, oc = (lane & 15) * 4;
    const int wq = warp * 8;                       // the warp's first query
    const int pos = p_lo + wq + sr;                // position of the thread's first score row
    const int w_last = p_lo + min(wq + 8, nq) - 1, w_first = p_lo + wq;
    const bool busy = wq < nq;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    unsigned long long acc[4][2 * NC];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2 * NC; ++j) acc[i][j] = 0ull;

    __syncthreads();                               // the queries are there
    // the walk's tiles: those whose number has its parity
    for (int kt = k_begin + ((k_begin / FK ^ walk) & 1) * FK; kt < k_end; kt += 2 * FK) {
        walk_sync();                               // the tile before has been used
        ask(kt);
        asm volatile("cp.async.wait_all;" ::: "memory");
        walk_sync();                               // this tile is there
        if (!busy || kt > w_last || (window > 0 && kt + FK <= w_first - window + 1)) continue;     // uniform for the warp
        float s[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
        const float* qrow = Qs + (wq + sr) * QP;
        const float* krow = Ks + sub * QP;
        float4 kv[2][4], qv[2][2];                 // the next four numbers are on their way while these are used
        auto pull = [&](int c, int at) {
#pragma unroll
            for (int j = 0; j < 4; ++j) kv[at][j] = *reinterpret_cast<const float4*>(krow + 8 * j * QP + c);
#pragma unroll
            for (int i = 0; i < 2; ++i) qv[at][i] = *reinterpret_cast<const float4*>(qrow + i * QP + c);
        };
        pull(0, 0);
#pragma unroll
        for (int c = 0; c < D; c += 4) {
            const int at = (c >> 2) & 1;
            if (c + 4 < D) pull(c + 4, at ^ 1);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        s[i][j] = fmaf((&qv[at][i].x)[u], (&kv[at][j].x)[u], s[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int p_i = pos + i;
            float tmax = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int kj = kt + sub + 8 * j;
                const bool vis = wq + sr + i < nq && kj <= p_i && (window == 0 || kj > p_i - window) &&
                                 there[sub + 8 * j];
                s[i][j] = vis ? s[i][j] : -INFINITY;
                tmax = fmaxf(tmax, s[i][j]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
            const float m_new = fmaxf(m_run[i], tmax);
            float alpha = 1.f, psum = 0.f;
            if (m_new != -INFINITY) alpha = expf(m_run[i] - m_new);          // a running maximum of -inf gives 0
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = m_new == -INFINITY ? 0.f : expf(s[i][j] - m_new);
                Ps[(sub + 8 * j) * 8 + sr + i] = p;
                psum += p;
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
            l_run[i] = fmaf(l_run[i], alpha, psum);
            m_run[i] = m_new;
            if (sub == 0) As[sr + i] = alpha;
        }
        __syncwarp();
        {
            const float4 f = *reinterpret_cast<const float4*>(As + orow);
            const float fs[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2 * NC; ++j) {
                    const float2 a = f32t::halves_of(acc[i][j]);
                    acc[i][j] = f32t::pair_of(__fmul_rn(a.x, fs[i]), __fmul_rn(a.y, fs[i]));
                }
        }
        const float* vrow = Vs + oc;
        float4 pn = *reinterpret_cast<const float4*>(Ps + orow);
        ulonglong2 vn[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) vn[c] = *reinterpret_cast<const ulonglong2*>(vrow + 64 * c);
        // Keys behind the warp's last query are left out: their weights are zeros, but values that are not finite must not
        // meet those of queries before them.
        const int n_keys = min(FK, w_last - kt + 1);
#pragma unroll
        for (int kr = 0; kr < FK; ++kr) {
            if (kr >= n_keys) break;
            const unsigned long long pp[4] = {f32t::pair_of(pn.x, pn.x), f32t::pair_of(pn.y, pn.y),
                                              f32t::pair_of(pn.z, pn.z), f32t::pair_of(pn.w, pn.w)};
            ulonglong2 v[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) v[c] = vn[c];
            if (kr + 1 < FK) {
                pn = *reinterpret_cast<const float4*>(Ps + (kr + 1) * 8 + orow);
#pragma unroll
                for (int c = 0; c < NC; ++c) vn[c] = *reinterpret_cast<const ulonglong2*>(vrow + (kr + 1) * D + 64 * c);
            }
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    f32t::fma2(acc[i][2 * c], pp[i], v[c].x);
                    f32t::fma2(acc[i][2 * c + 1], pp[i], v[c].y);
                }
        }
        __syncwarp();                              // the weights have been read
    }
    // The second walk leaves its rows where its tiles were: [FQ][D] outputs, then maxima and sums; the first takes them in.
    __syncthreads();
    float* theirs = Qs + FQ * QP + FK * (QP + D);
    float* m_theirs = theirs + FQ * D;
    float* l_theirs = m_theirs + FQ;
    if (walk == 1 && busy) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (sub == 0) { m_theirs[wq + sr + i] = m_run[i]; l_theirs[wq + sr + i] = l_run[i]; }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < NC; ++c)
                *reinterpret_cast<ulonglong2*>(theirs + (wq + orow + i) * D + oc + 64 * c) = make_ulonglong2(acc[i][2 * c], acc[i][2 * c + 1]);
    }
    __syncthreads();
    if (walk == 1 || !busy) return;
    // factors of the two walks' rows: exp(m - common maximum) over the common sum
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (sub == 0) {
            const float mt = m_theirs[wq + sr + i], lt = l_theirs[wq + sr + i], m = fmaxf(m_run[i], mt);
            const float a = m == -INFINITY ? 0.f : expf(m_run[i] - m), b = m == -INFINITY ? 0.f : expf(mt - m);
            const float l = fmaf(l_run[i], a, __fmul_rn(lt, b)), inv = l > 0.f ? 1.f / l : 0.f;
            As[sr + i] = a * inv;
            Ps[sr + i] = b * inv;
        }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (wq + orow + i >= nq) break;
        const float a = As[orow + i], b = Ps[orow + i];
        const float* r = theirs + (wq + orow + i) * D + oc;
        float* o = out + ((int64_t)(q0 + qt * FQ + wq + orow + i) * nh + h) * D + oc;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const float2 lo = f32t::halves_of(acc[i][2 * c]), hi = f32t::halves_of(acc[i][2 * c + 1]);
            const float4 y = *reinterpret_cast<const float4*>(r + 64 * c);
            *reinterpret_cast<float4*>(o + 64 * c) = make_float4(fmaf(lo.x, a, __fmul_rn(y.x, b)), fmaf(lo.y, a, __fmul_rn(y.y, b)),
                                                                 fmaf(hi.x, a, __fmul_rn(y.z, b)), fmaf(hi.y, a, __fmul_rn(y.w, b)));
        }
    }
}

// ---------------------------------------------------------------------------
// Split-KV decode: one query token per request (q_len == 1).  Block = (request,
// head, split of SPLIT keys); 16 groups of 8 threads, each group walks every
// 16th key of the split with its own running (m, l, acc); groups are merged in
// shared memory in group order, splits by the merge kernel in split order.
// The number of splits of a request depends on its own kv_len only.
// Partials: part_o [B, nh, max_splits, D], part_ml [B, nh, max_splits, 2].
// ---------------------------------------------------------------------------
// E consecutive elements (E a multiple of 8, 16-byte aligned) as floats, with 16-byte loads
template <typename AT, int E> __device__ __forceinline__ void load_vec(const AT* p, float (&out)[E]);
template <> __device__ __forceinline__ void load_vec<float, 8>(const float* p, float (&out)[8]) {
    const float4* v = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 0; i < 2; ++i) { const float4 x = __ldg(v + i); out[4*i] = x.x; out[4*i+1] = x.y; out[4*i+2] = x.z; out[4*i+3] = x.w; }
}
template <> __device__ __forceinline__ void load_vec<float, 16>(const float* p, float (&out)[16]) {
    const float4* v = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float4 x = __ldg(v + i); out[4*i] = x.x; out[4*i+1] = x.y; out[4*i+2] = x.z; out[4*i+3] = x.w; }
}
template <> __device__ __forceinline__ void load_vec<float, 32>(const float* p, float (&out)[32]) {
    const float4* v = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) { const float4 x = __ldg(v + i); out[4*i] = x.x; out[4*i+1] = x.y; out[4*i+2] = x.z; out[4*i+3] = x.w; }
}
__device__ __forceinline__ void unpack8(const uint4 x, float* out) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); out[2*i] = f.x; out[2*i+1] = f.y; }
}
template <> __device__ __forceinline__ void load_vec<__nv_bfloat16, 8>(const __nv_bfloat16* p, float (&out)[8]) {
    unpack8(__ldg(reinterpret_cast<const uint4*>(p)), out);
}
template <> __device__ __forceinline__ void load_vec<__nv_bfloat16, 16>(const __nv_bfloat16* p, float (&out)[16]) {
    const uint4* v = reinterpret_cast<const uint4*>(p);
    unpack8(__ldg(v), out); unpack8(__ldg(v + 1), out + 8);
}
template <> __device__ __forceinline__ void load_vec<__nv_bfloat16, 32>(const __nv_bfloat16* p, float (&out)[32]) {
    const uint4* v = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) unpack8(__ldg(v + i), out + 8 * i);
}

// E consecutive elements held as they were loaded (16-byte words), unpacked to float when used
template <typename AT, int E> struct RawVec;
template <int E> struct RawVec<float, E> {
    float4 w[E / 4];
    __device__ __forceinline__ void load(const float* p) {
#pragma unroll
        for (int i = 0; i < E / 4; ++i) w[i] = __ldg(reinterpret_cast<const float4*>(p) + i);
    }
    __device__ __forceinline__ void unpack(float (&out)[E]) const {
#pragma unroll
        for (int i = 0; i < E / 4; ++i) { out[4*i] = w[i].x; out[4*i+1] = w[i].y; out[4*i+2] = w[i].z; out[4*i+3] = w[i].w; }
    }
};
template <int E> struct RawVec<__nv_bfloat16, E> {
    uint4 w[E / 8];
    __device__ __forceinline__ void load(const __nv_bfloat16* p) {
#pragma unroll
        for (int i = 0; i < E / 8; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
    }
    __device__ __forceinline__ void unpack(float (&out)[E]) const {
#pragma unroll
        for (int i = 0; i < E / 8; ++i) unpack8(w[i], &out[8 * i]);
    }
};

// Splits of a request with `kvl` keys: SPLIT keys each; a tail of up to a quarter of a split joins
// the split before it instead of making a block of its own.  A function of the request's own length only.
template <int SPLIT>
__device__ __forceinline__ int decode_splits(int kvl) {
    return max(1, (kvl + SPLIT - SPLIT / 4 - 1) / SPLIT);
}

// tanh of a capped score: the library's for float32 scores; for a bfloat16 cache, whose scores carry the rounding
// of their operands, 1 - 2 / (e^{2x} + 1) with the hardware's exponential and division (exact at both ends:
// e^{2x} = inf gives 1, 0 gives -1).
template <typename AT>
__device__ __forceinline__ float capped_tanh(float x) {
    if (sizeof(AT) == 4) return tanhf(x);
    return 1.0f - __fdividef(2.0f, __expf(2.0f * x) + 1.0f);
}

constexpr int DEC_SPLIT = 512;      // keys per split by default; smaller splits spread one or two requests over the device
constexpr int DEC_GROUPS = 16;
constexpr int DEC_JOIN_MAX = 8, DEC_JOIN_PER_SM = 4;

// JOIN: the splits of a head are a cluster of at most DEC_JOIN_MAX blocks, and the first of them adds the others' results up
// from their shared memory, as the merge kernel below does from the scratch (which is then not touched): one launch instead of
// two, and no trip through memory between them.  Clusters wait for room for all of their blocks, so this pays while the device
// holds all blocks at once (4 an SM).  The same bits either way.  One request of 300 keys, 8 heads over 2: 8.9 us in two
// launches, 6.8 joined; 8 of up to 2,048 keys, 16 over 16 (512 blocks): 24.4 and 23.1; 64 of up to 3,000 (6,144 blocks): 166 and
// 216.
// The scores of a round of keys are formed side by side and share one rescaling (a chain of two exchanges and two exponentials a
// key held the rounds up): the three above 6.0, 18.8 and 154 us.
template <typename AT, int D, int SPLIT, bool JOIN = false>
__global__ void __launch_bounds__(128)
attn_decode_split_kernel(const AT* __restrict__ q, const AT* __restrict__ k_cache, const AT* __restrict__ v_cache,
                         const int* __restrict__ block_table, const int* __restrict__ q_start,
                         const int* __restrict__ kv_len, float* __restrict__ part_o,
                         float* __restrict__ part_ml, int nh, int nkv, int page_size, int max_pages,
                         int max_splits, int window, float scale, float cap, AT* __restrict__ out, int sink, AttnForm form) {
    static_assert(!JOIN || D == 128, "a thread per column");
    constexpr int E = D / 8;  // elements per thread
    const int chunk = form.chunk;
    wait_for_earlier_kernels();
    const int b = blockIdx.z, h = blockIdx.y, sp = blockIdx.x;
    const int kvl = kv_len[b];
    const int pos = kvl - 1;
    const int k_first = first_visible(pos, window, chunk);
    // never more splits than the caller's scratch holds (a caller whose max_splits is too small for its
    // longest request gets a result over fewer keys, never an access outside the scratch)
    const int n_splits = min(decode_splits<SPLIT>(kvl), max_splits);
    const int first_split = min(k_first / SPLIT, n_splits - 1);
    if (sp < first_split || sp >= n_splits) return;
    const int hk = h / (nh / nkv);
    const int tid = threadIdx.x, grp = tid >> 3, sub = tid & 7;
    // the 8 threads of a group stay together; groups of one warp may diverge
    const unsigned gmask = 0xFFu << ((tid & 31) & ~7);
    const int t = q_start[b];
    float qr[E];
    load_vec<AT, E>(q + ((int64_t)t * nh + h) * D + sub * E, qr);
#pragma unroll
    for (int i = 0; i < E; ++i) qr[i] *= scale;
    float m_run = -INFINITY, l_run = 0.f;
    const float inv_cap = cap > 0.f ? 1.0f / cap : 0.f;
    float acc[E];
#pragma unroll
    for (int i = 0; i < E; ++i) acc[i] = 0.f;
    constexpr int SPAN = SPLIT + SPLIT / 4;                   // the last split may hold a short tail too
    const int k_lo = max(sp * SPLIT, k_first);
    const int k_hi = sp == n_splits - 1 ? min(kvl, sp * SPLIT + SPAN) : (sp + 1) * SPLIT;
    const int span = k_hi - sp * SPLIT;
    // the pages of this split, looked up once
    __shared__ int64_t key_off[SPAN];
    {
        const int* table = block_table + (int64_t)b * max_pages;
        for (int i = tid; i < span; i += 128) {
            const int kj = sp * SPLIT + i;
            int64_t off = -1;
            if (kj >= k_lo && kj < k_hi) {
                const int page = table[kj / page_size];
                if (page >= 0) off = ((int64_t)page * nkv + hk) * page_size * D + (int64_t)(kj % page_size) * D;
            }
            key_off[i] = off;
        }
    }
    __syncthreads();
    // KPR keys per round: all their loads are issued before any is used
    constexpr int KPR = (sizeof(AT) == 2 || E <= 16) ? 4 : 2;
    using Raw = RawVec<AT, E>;
    struct Round { Raw k[KPR], v[KPR]; bool in[KPR]; };
    auto ask = [&](int i0, Round& r) {
#pragma unroll
        for (int u = 0; u < KPR; ++u) {
            const int i = i0 + u * DEC_GROUPS;
            const int64_t off = i < span ? key_off[i] : -1;
            r.in[u] = off >= 0;
            if (r.in[u]) { r.k[u].load(k_cache + off + sub * E); r.v[u].load(v_cache + off + sub * E); }
        }
    };
    // the scores of a round side by side, then one rescaling for its keys
    auto use = [&](const Round& r) {
        float p[KPR], m_new = m_run;
#pragma unroll
        for (int u = 0; u < KPR; ++u) {
            float kf[E];
            r.k[u].unpack(kf);
            p[u] = 0.f;
#pragma unroll
            for (int i = 0; i < E; ++i) p[u] += qr[i] * kf[i];
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < KPR; ++u) p[u] += __shfl_xor_sync(gmask, p[u], o);
#pragma unroll
        for (int u = 0; u < KPR; ++u) {
            if (cap > 0.f) p[u] = cap * capped_tanh<AT>(p[u] * inv_cap);
            if (!r.in[u]) p[u] = -INFINITY;
            m_new = fmaxf(m_new, p[u]);
        }
        const float ref = m_new == -INFINITY ? 0.f : m_new;          // (the group has seen no key)
        const float alpha = expf(m_run - ref);
        l_run *= alpha;
#pragma unroll
        for (int i = 0; i < E; ++i) acc[i] *= alpha;
#pragma unroll
        for (int u = 0; u < KPR; ++u) {
            if (!r.in[u]) continue;
            const float w = expf(p[u] - ref);
            l_run += w;
            float vf[E];
            r.v[u].unpack(vf);
#pragma unroll
            for (int i = 0; i < E; ++i) acc[i] += w * vf[i];
        }
        m_run = m_new;
    };
    constexpr int STEP = KPR * DEC_GROUPS;
    for (int i0 = grp; i0 < span; i0 += STEP) {
        Round r;
        ask(i0, r);
        use(r);
    }
    // merge the 16 groups in group order
    __shared__ float sm_m[DEC_GROUPS], sm_l[DEC_GROUPS];
    __shared__ __align__(16) float sm_o[DEC_GROUPS][D];
    __shared__ float own_o[JOIN ? D : 1], own_ml[2];
    if (sub == 0) { sm_m[grp] = m_run; sm_l[grp] = l_run; }
#pragma unroll
    for (int i = 0; i < E; i += 4)
        *reinterpret_cast<float4*>(&sm_o[grp][sub * E + i]) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    __syncthreads();
    float m_all = -INFINITY, l_all = 0.f, w[DEC_GROUPS];
#pragma unroll
    for (int g = 0; g < DEC_GROUPS; ++g) m_all = fmaxf(m_all, sm_m[g]);
#pragma unroll
    for (int g = 0; g < DEC_GROUPS; ++g) {
        w[g] = (sm_m[g] == -INFINITY) ? 0.f : expf(sm_m[g] - m_all);
        l_all += w[g] * sm_l[g];
    }
    const int64_t pidx = ((int64_t)b * nh + h) * max_splits + sp;
    for (int c = tid; c < D; c += 128) {
        float o = 0.f;
#pragma unroll
        for (int g = 0; g < DEC_GROUPS; ++g) o += w[g] * sm_o[g][c];
        if (JOIN) own_o[c] = o;
        else part_o[pidx * D + c] = o;
    }
    if (tid == 0) {
        if (JOIN) { own_ml[0] = m_all; own_ml[1] = l_all; }
        else { part_ml[pidx * 2] = m_all; part_ml[pidx * 2 + 1] = l_all; }
    }
    if constexpr (JOIN) {
        // (blocks without keys of this request have left: a cluster's barriers wait for those that are there)
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (sp == first_split) {
            auto of = [](const float* own, int block) {
                uint32_t there;
                float v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(own)), "r"(block));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(there));
                return v;
            };
            const float s0 = form.sink_score ? form.sink_score[h] : 0.f;
            float ms[DEC_JOIN_MAX], ls[DEC_JOIN_MAX], os[DEC_JOIN_MAX], m_head = -INFINITY;
#pragma unroll
            for (int x = 0; x < DEC_JOIN_MAX; ++x) {
                const bool there = first_split + x < n_splits;
                ms[x] = there ? of(&own_ml[0], first_split + x) : -INFINITY;
                ls[x] = there ? of(&own_ml[1], first_split + x) : 0.f;
                os[x] = there ? of(&own_o[tid], first_split + x) : 0.f;
                m_head = fmaxf(m_head, ms[x]);
            }
            if (sink) m_head = fmaxf(m_head, s0);
            float l = sink ? expf(s0 - m_head) : 0.f, o = 0.f;
#pragma unroll
            for (int x = 0; x < DEC_JOIN_MAX; ++x) {
                if (first_split + x >= n_splits) break;
                const float w = ms[x] == -INFINITY ? 0.f : expf(ms[x] - m_head);
                l += w * ls[x];
                o += w * os[x];
            }
            const float inv = (l > 0.f ? 1.f / l : 0.f) * head_gate(form, t, h);
            out[((int64_t)t * nh + h) * D + tid] = from_float<AT>(o * inv);
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// One launch for a decode step's attention: splits in clusters.
template <typename AT, int D, int SPLIT, typename... A>
static void launch_decode_joined(dim3 grid, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid;
    lc.blockDim = dim3(128);
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = grid.x;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = dependent_launch_enabled() ? 2 : 1;
    (void)cudaLaunchKernelEx(&lc, attn_decode_split_kernel<AT, D, SPLIT, true>, args...);
}

// Merge of a (request, head)'s splits in split order.  The splits' maxima and sums are fetched by all
// threads at once and their weights exp(m_s - m) kept in shared memory (up to MERGE_CAP splits; more
// are re-read from global memory), so the block waits for global memory twice, not once per split.
constexpr int MERGE_CAP = 512;

template <typename AT, int D, int SPLIT>
__global__ void attn_decode_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                         const int* __restrict__ q_start, const int* __restrict__ kv_len,
                                         AT* __restrict__ out, int nh, int max_splits, int window, int sink,
                                         AttnForm form) {
    const int chunk = form.chunk;
    __shared__ float sm_w[MERGE_CAP], sm_l[MERGE_CAP], sm_red[4];
    wait_for_earlier_kernels();
    const int b = blockIdx.y, h = blockIdx.x;
    const int kvl = kv_len[b];
    const int pos = kvl - 1;
    const int k_first = first_visible(pos, window, chunk);
    const int n_splits = min(decode_splits<SPLIT>(kvl), max_splits);
    const int first_split = min(k_first / SPLIT, n_splits - 1);
    const int64_t base = ((int64_t)b * nh + h) * max_splits;
    const int t = q_start[b];
    const int n = n_splits - first_split;
    const float s0 = form.sink_score ? form.sink_score[h] : 0.f;
    const float hg = head_gate(form, t, h);
    if (n <= MERGE_CAP) {
        const float2* ml = reinterpret_cast<const float2*>(part_ml) + base + first_split;
        float mx = -INFINITY;
        for (int s = threadIdx.x; s < n; s += blockDim.x) {
            const float2 v = ml[s];
            sm_w[s] = v.x;
            sm_l[s] = v.y;
            mx = fmaxf(mx, v.x);
        }
        mx = warp_max(mx);
        if ((threadIdx.x & 31) == 0) sm_red[threadIdx.x >> 5] = mx;
        __syncthreads();
        float m_all = -INFINITY;
        for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) m_all = fmaxf(m_all, sm_red[w]);
        // one key more, without a value: it joins the reference and the sum, not the rows
        if (sink) m_all = fmaxf(m_all, s0);
        for (int s = threadIdx.x; s < n; s += blockDim.x) {
            const float m = sm_w[s];
            sm_w[s] = m == -INFINITY ? 0.f : expf(m - m_all);
        }
        __syncthreads();
        float l = sink ? expf(s0 - m_all) : 0.f;
        for (int s = 0; s < n; ++s) l += sm_w[s] * sm_l[s];
        const float inv = (l > 0.f ? 1.f / l : 0.f) * hg;
        const float* po = part_o + (base + first_split) * D;
        for (int c = threadIdx.x; c < D; c += blockDim.x) {
            float o = 0.f;
#pragma unroll 4
            for (int s = 0; s < n; ++s) o += sm_w[s] * po[(int64_t)s * D + c];
            out[((int64_t)t * nh + h) * D + c] = from_float<AT>(o * inv);
        }
        return;
    }
    float m_all = -INFINITY;
    for (int s = first_split; s < n_splits; ++s) m_all = fmaxf(m_all, part_ml[(base + s) * 2]);
    if (sink) m_all = fmaxf(m_all, s0);
    float l = sink ? expf(s0 - m_all) : 0.f;
    for (int s = first_split; s < n_splits; ++s) {
        const float m = part_ml[(base + s) * 2];
        l += (m == -INFINITY ? 0.f : expf(m - m_all)) * part_ml[(base + s) * 2 + 1];
    }
    const float inv = (l > 0.f ? 1.f / l : 0.f) * hg;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
        float o = 0.f;
        for (int s = first_split; s < n_splits; ++s) {
            const float m = part_ml[(base + s) * 2];
            o += (m == -INFINITY ? 0.f : expf(m - m_all)) * part_o[(base + s) * D + c];
        }
        out[((int64_t)t * nh + h) * D + c] = from_float<AT>(o * inv);
    }
}

template <typename AT>
static int launch_tiled(const void* q, const void* kc, const void* vc, const int* block_table,
                        const int* q_start, const int* kv_len, void* out, int B, int max_q_len, int nh,
                        int nkv, int d, int page_size, int max_pages, int window, float scale,
                        cudaStream_t stream) {
    const dim3 grid((max_q_len + TQ - 1) / TQ, nh, B);
    const size_t smem = sizeof(float) * ((size_t)TQ * (d + 1) + (size_t)TK * (d + 1) + (size_t)TK * d + TQ * (TK + 1));
#define MI_TILED(ND)                                                                                   \
    do {                                                                                               \
        auto kern = attn_tiled_kernel<AT, ND>;                                                         \
        if (smem > 40 * 1024) /* (48 KiB with what the kernel has beside it) */                        \
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);        \
        kern<<<grid, 128, smem, stream>>>((const AT*)q, (const AT*)kc, (const AT*)vc, block_table,     \
                                          q_start, kv_len, (AT*)out, nh, nkv, d, page_size, max_pages, \
                                          window, scale);                                              \
    } while (0)
    if (d <= 16) MI_TILED(2);
    else if (d <= 32) MI_TILED(4);
    else if (d <= 64) MI_TILED(8);
    else if (d <= 128) MI_TILED(16);
    else MI_TILED(32);
#undef MI_TILED
    return finish_launch("attn_tiled");
}

}  // namespace mi

using namespace mi;

extern "C" {

// Attention for any mix of portions and single tokens.  max_q_len bounds the
// longest portion in the batch (grid size).
int mi_attn_tiled(const void* q, const void* k_cache, const void* v_cache, int adtype, const int* block_table,
                  const int* q_start, const int* kv_len, void* out, int B, int max_q_len, int nh, int nkv,
                  int d, int page_size, int max_pages, int window, float scale, cudaStream_t stream) {
    if (B <= 0 || max_q_len <= 0) return kOk;
    if (d < 1 || d > 256) {
        set_last_error("attention: head_dim %d is outside [1, 256]", d);
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
    if (adtype == kF32 && (d == 64 || d == 128) &&
        ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
          reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
        const dim3 grid((max_q_len + FQ - 1) / FQ, nh, B);
        const size_t smem = d == 64 ? rows_f32_smem<64>() : rows_f32_smem<128>();
        auto kernel = d == 64 ? attn_rows_f32_kernel<64> : attn_rows_f32_kernel<128>;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kernel<<<grid, 256, smem, stream>>>((const float*)q, (const float*)k_cache, (const float*)v_cache, block_table,
                                            q_start, kv_len, (float*)out, nh, nkv, page_size, max_pages, window, scale);
        return finish_launch("attn_rows_f32");
    }
    MI_DISPATCH_1(adtype, AT,
        return launch_tiled<AT>(q, k_cache, v_cache, block_table, q_start, kv_len, out, B, max_q_len, nh,
                                nkv, d, page_size, max_pages, window, scale, stream));
    return kOk;
}

// 1 if the split-KV decode kernel is built for this head size.
int mi_attn_decode_supported(int d) { return (d == 64 || d == 128 || d == 256) ? 1 : 0; }

int mi_attn_decode_split_size() { return DEC_SPLIT; }

// 1 if `split` keys per split is built (128, 256, 512).
int mi_attn_decode_split_supported(int split) { return (split == 128 || split == 256 || split == 512) ? 1 : 0; }

// 1 if the splits of a decode attention over a bfloat16 cache go as clusters, in one launch: heads of `d` numbers, `heads` of all
// requests together, up to `splits` each.
int mi_attn_decode_joined(int d, int64_t heads, int splits) {
    return d == 128 && splits <= DEC_JOIN_MAX && heads * splits <= DEC_JOIN_PER_SM * (int64_t)sm_count() ? 1 : 0;
}

// Decode attention: every request has exactly one query token.  `part_o` needs
// B*nh*max_splits*d floats, `part_ml` B*nh*max_splits*2, with max_splits >= ceil(max_kv_len / split).
// cap > 0: every scaled score becomes cap * tanh(score / cap); sink: the softmax counts one key more, of score
// 0 and without a value.
int mi_attn_decode_split_form(const void* q, const void* k_cache, const void* v_cache, int adtype,
                              const int* block_table, const int* q_start, const int* kv_len, void* out,
                              float* part_o, float* part_ml, int B, int nh, int nkv, int d, int page_size,
                              int max_pages, int max_splits, int split, int window, float scale, float cap, int sink,
                              int chunk, const float* sink_score, const float* gate, int64_t ld_gate,
                              cudaStream_t stream) {
    if (B <= 0) return kOk;
    if (chunk < 0 || (chunk > 0 && window > 0) || (sink_score && !sink)) {
        set_last_error("decode attention: chunks of %d go without a window (%d), a sink's scores with a sink", chunk, window);
        return kBadShape;
    }
    const AttnForm form = {chunk, sink_score, gate, ld_gate};
    if (cap < 0.f) { set_last_error("decode attention: a cap of %g", (double)cap); return kBadShape; }
    if (!mi_attn_decode_supported(d)) {
        set_last_error("decode attention: head_dim %d is not built (64, 128, 256)", d);
        return kBadShape;
    }
    if (!mi_attn_decode_split_supported(split)) {
        set_last_error("decode attention: splits of %d keys are not built (128, 256, 512)", split);
        return kBadShape;
    }
    if (nkv < 1 || nh % nkv != 0) {
        set_last_error("attention: %d query heads are not a multiple of %d key/value heads", nh, nkv);
        return kBadShape;
    }
    if (B > 65535 || nh > 65535 || max_splits < 1) {
        set_last_error("decode attention: bad grid (B=%d, nh=%d, max_splits=%d)", B, nh, max_splits);
        return kBadShape;
    }
    const dim3 grid(max_splits, nh, B);
    const dim3 mgrid(nh, B);
#define MI_DEC(DD, SS)                                                                                    \
    do {                                                                                                  \
        if constexpr (DD == 128 && sizeof(AT) == 2) {                                                     \
            if (mi_attn_decode_joined(d, (int64_t)nh * B, max_splits)) {                                   \
                launch_decode_joined<AT, DD, SS>(grid, stream, (const AT*)q, (const AT*)k_cache, (const AT*)v_cache, \
                    block_table, q_start, kv_len, part_o, part_ml, nh, nkv, page_size, max_pages, max_splits, window, \
                    scale, cap, (AT*)out, sink, form);                                                    \
                return finish_launch("attn_decode");                                                      \
            }                                                                                             \
        }                                                                                                 \
        launch_dependent(attn_decode_split_kernel<AT, DD, SS>, grid, dim3(128), 0, stream,                \
            (const AT*)q, (const AT*)k_cache, (const AT*)v_cache, block_table, q_start, kv_len, part_o,  \
            part_ml, nh, nkv, page_size, max_pages, max_splits, window, scale, cap, (AT*)nullptr, 0, form); \
        launch_behind(attn_decode_merge_kernel<AT, DD, SS>, mgrid, dim3(DD <= 128 ? DD : 128), 0, stream, \
            part_o, part_ml, q_start, kv_len, (AT*)out, nh, max_splits, window, sink, form);              \
    } while (0)
#define MI_DEC_D(SS) do { if (d == 64) MI_DEC(64, SS); else if (d == 128) MI_DEC(128, SS); else MI_DEC(256, SS); } while (0)
    MI_DISPATCH_1(adtype, AT,
        if (split == 128) MI_DEC_D(128); else if (split == 256) MI_DEC_D(256); else MI_DEC_D(512));
#undef MI_DEC_D
#undef MI_DEC
    return finish_launch("attn_decode", 2);
}

int mi_attn_decode_split(const void* q, const void* k_cache, const void* v_cache, int adtype, const int* block_table,
                         const int* q_start, const int* kv_len, void* out, float* part_o, float* part_ml, int B,
                         int nh, int nkv, int d, int page_size, int max_pages, int max_splits, int split, int window,
                         float scale, cudaStream_t stream) {
    return mi_attn_decode_split_form(q, k_cache, v_cache, adtype, block_table, q_start, kv_len, out, part_o, part_ml,
                                     B, nh, nkv, d, page_size, max_pages, max_splits, split, window, scale, 0.f, 0, 0,
                                     nullptr, nullptr, 0, stream);
}

// The same with the default split size.
int mi_attn_decode(const void* q, const void* k_cache, const void* v_cache, int adtype, const int* block_table,
                   const int* q_start, const int* kv_len, void* out, float* part_o, float* part_ml, int B,
                   int nh, int nkv, int d, int page_size, int max_pages, int max_splits, int window,
                   float scale, cudaStream_t stream) {
    return mi_attn_decode_split(q, k_cache, v_cache, adtype, block_table, q_start, kv_len, out, part_o, part_ml, B, nh,
                                nkv, d, page_size, max_pages, max_splits, DEC_SPLIT, window, scale, stream);
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// The same decode attention for callers that must not allocate (see attention_noalloc.h): the
// split partials live in an array that is part of the library image instead of caller scratch.
// ---------------------------------------------------------------------------------------------
#include "attention_noalloc.h"

namespace mi {

static __device__ __align__(256) unsigned char g_noalloc_scratch[MI_ATTN_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
// Device address of g_noalloc_scratch per device.  In host code the array's name is only a
// handle for cudaGetSymbolAddress, never a pointer a kernel could use.
static float* g_noalloc_ptr[kMaxDevices] = {nullptr};

// Looks the address up once per device, with that device current.  Returns nullptr on failure.
static float* noalloc_scratch_for_current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        set_last_error("decode attention (no allocation): cannot identify the current device");
        return nullptr;
    }
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            set_last_error("decode attention (no allocation): cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return nullptr;
        }
        g_noalloc_ptr[dev] = static_cast<float*>(p);
    }
    return g_noalloc_ptr[dev];
}

}  // namespace mi

extern "C" {

unsigned int mi_attn_decode_noalloc_capacity(void) { return MI_ATTN_NOALLOC_SCRATCH_BYTES; }

int mi_attn_decode_noalloc(const void* q, const void* k_cache, const void* v_cache, int adtype,
                           const int* block_table, const int* q_start, const int* kv_len, void* out, int B,
                           int nh, int nkv, int d, int page_size, int max_pages, int max_splits, int window,
                           float scale, cudaStream_t stream) {
    if (B <= 0) return kOk;
    if (max_splits < 1 || nh < 1 || d < 1) {
        set_last_error("decode attention (no allocation): bad sizes (nh=%d, d=%d, max_splits=%d)", nh, d, max_splits);
        return kBadShape;
    }
    const unsigned long long n_part = (unsigned long long)B * nh * max_splits;
    const unsigned long long need = n_part * ((unsigned long long)d + 2ull) * sizeof(float);
    if (need > MI_ATTN_NOALLOC_SCRATCH_BYTES) {
        set_last_error("decode attention (no allocation): B=%d, heads=%d, splits=%d, head_dim=%d need %llu bytes of "
                       "scratch, the built-in array holds %u", B, nh, max_splits, d, need,
                       (unsigned)MI_ATTN_NOALLOC_SCRATCH_BYTES);
        return kBadShape;
    }
    float* scratch = noalloc_scratch_for_current_device();
    if (!scratch) return kLaunchFailed;
    float* part_o = scratch;                       // [B, nh, max_splits, d]
    float* part_ml = scratch + n_part * d;         // [B, nh, max_splits, 2]
    return mi_attn_decode(q, k_cache, v_cache, adtype, block_table, q_start, kv_len, out, part_o, part_ml, B, nh,
                          nkv, d, page_size, max_pages, max_splits, window, scale, stream);
}

}  // extern "C"
