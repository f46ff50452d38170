// Tiles of products in true 32 bits on the CUDA cores: what the dense and the grouped float32 products share (inner sizes
// below 512; larger ones go to the tensor cores, f32_tc.cuh).
//
// Every output element is ONE chain of fused multiply-adds over k in ascending order, in every form below, so a
// result has the same bits whichever form, tile or row of a tile computes it.  Two forms:
//
//   WideTile   64 rows x BN columns by 128 threads, 8 x (BN / 16) outputs a thread.  Bound by the FMA pipes: two
//              multiply-adds go in one instruction (fma.rn.f32x2, the same rounding as two), which leaves issue slots
//              for the loads from shared memory and for making pairs (a, a); the next k tile is on its way from
//              memory in registers meanwhile.  A warp covers 16 rows and is idle where its rows lie past the end; a
//              block's warps take their rows in an order that turns with the block, so that the idle ones of several
//              blocks do not all belong to one quarter of the SM.
//   NarrowTile 16 rows x 32 columns by 128 threads, 4 rows a warp, one column (or gate and up column) a lane.
//              Bound by reading W: four tiles of 64 k arrive through cp.async while one is used.
//
// Measured when larger inner sizes came here: 512 rows against [6144, 2048] and [2048, 2048] (a q/k/v and an output product): 629 us with 64 x 64 tiles of 4 x 4
// outputs a thread, 415 us with these (43 and 35 TFLOP/s; the FMA pipes are 70 % busy where every SM has blocks).
#pragma once

#include "common.cuh"

namespace mi {
namespace f32t {

constexpr int THREADS = 128;
constexpr int BM = 64, BK = 16;            // WideTile
constexpr int NM = 16, NN = 32, NK = 64;   // NarrowTile
constexpr int NSTAGES = 4, NPITCH = NK + 4;

__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 halves_of(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// four values from k on (zeros past K, and for a row that is not there)
template <bool VEC>
__device__ __forceinline__ float4 load4(const float* __restrict__ row, int k, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!row) return v;
    if (VEC) {
        if (k < K) v = __ldg(reinterpret_cast<const float4*>(row + k));
    } else {
        if (k < K) v.x = __ldg(row + k);
        if (k + 1 < K) v.y = __ldg(row + k + 1);
        if (k + 2 < K) v.z = __ldg(row + k + 2);
        if (k + 3 < K) v.w = __ldg(row + k + 3);
    }
    return v;
}

// The thread's columns of a WideTile: TN / 2 from c_lo on, TN / 2 from BN / 2 + c_lo on; its rows: 8 from r_lo on.
template <int BN> struct WidePlace {
    static constexpr int TN = BN / 16;
    int r_lo, c_lo;
    __device__ __forceinline__ explicit WidePlace(int turn) {
        const int warp = ((threadIdx.x >> 5) + turn) & 3, lane = threadIdx.x & 31;
        r_lo = warp * 16 + (lane >> 4) * 8;
        c_lo = (lane & 15) * (TN / 2);
    }
};

// acc[i][j]: outputs of row r_lo + i; pairs j of the thread's columns in order.  a_row(r), w_row(n): row r of the tile's
// BM rows (n of its BN columns) or null.  K > 0.
template <int BN, bool VEC, typename ARow, typename WRow>
__device__ __forceinline__ void wide_tile(unsigned long long (&acc)[8][BN / 32], ARow a_row, WRow w_row, int rows, int K,
                                          const WidePlace<BN>& at) {
    constexpr int TN = BN / 16, LA = BM * 4 / THREADS, LW = BN * 4 / THREADS;
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Ws[2][BK][BN + 4];
    const int tid = threadIdx.x, kc = (tid & 3) * 4;
    const float* ap[LA];
    const float* wp[LW];
#pragma unroll
    for (int i = 0; i < LA; ++i) ap[i] = a_row((tid >> 2) + 32 * i);
#pragma unroll
    for (int i = 0; i < LW; ++i) wp[i] = w_row((tid >> 2) + 32 * i);
    float4 av[LA], wv[LW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; ++i) av[i] = load4<VEC>(ap[i], k0 + kc, K);
#pragma unroll
        for (int i = 0; i < LW; ++i) wv[i] = load4<VEC>(wp[i], k0 + kc, K);
    };
    auto put = [&](int buf) {
        const int r = tid >> 2;
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            As[buf][kc][r + 32 * i] = av[i].x; As[buf][kc + 1][r + 32 * i] = av[i].y;
            As[buf][kc + 2][r + 32 * i] = av[i].z; As[buf][kc + 3][r + 32 * i] = av[i].w;
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            Ws[buf][kc][r + 32 * i] = wv[i].x; Ws[buf][kc + 1][r + 32 * i] = wv[i].y;
            Ws[buf][kc + 2][r + 32 * i] = wv[i].z; Ws[buf][kc + 3][r + 32 * i] = wv[i].w;
        }
    };
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    const bool busy = (at.r_lo & ~15) < rows;          // uniform for a warp
    fetch(0);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
        if (busy) {
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {          // k beyond K holds zeros: fma(0, 0, acc) == acc
                const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][at.r_lo]);
                const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][at.r_lo + 4]);
                unsigned long long w[TN / 2];
                if constexpr (TN == 8) {
                    const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(&Ws[buf][kk][at.c_lo]);
                    const ulonglong2 hi = *reinterpret_cast<const ulonglong2*>(&Ws[buf][kk][BN / 2 + at.c_lo]);
                    w[0] = lo.x; w[1] = lo.y; w[2] = hi.x; w[3] = hi.y;
                } else {
                    w[0] = *reinterpret_cast<const unsigned long long*>(&Ws[buf][kk][at.c_lo]);
                    w[1] = *reinterpret_cast<const unsigned long long*>(&Ws[buf][kk][BN / 2 + at.c_lo]);
                }
                const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned long long aa = pair_of(a[i], a[i]);
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, w[j]);
                }
            }
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool there) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = there ? 16 : 0;                      // nothing read: the 16 bytes become zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// bytes of dynamic shared memory of a NarrowTile with W rows of `halves` matrices
inline size_t narrow_smem(int halves) { return (size_t)NSTAGES * (NM + halves * NN) * NPITCH * 4; }

// acc[h][i]: row warp * 4 + i, column `lane` of half h.  Rows must be 16-byte aligned and K a multiple of 4;
// `any`: an address that may be named (not read) for what is not there.
template <int HALVES, typename ARow, typename WRow>
__device__ __forceinline__ void narrow_tile(float (&acc)[HALVES][4], ARow a_row, WRow w_row, int rows, int K,
                                            const float* any) {
    extern __shared__ __align__(16) float smem_f[];
    constexpr int STAGE = (NM + HALVES * NN) * NPITCH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row_l = tid >> 4, kc = (tid & 15) * 4;   // 8 rows of 64 floats per round of the block's copies
    const float* ap[NM / 8];
    const float* wp[HALVES * NN / 8];
#pragma unroll
    for (int i = 0; i < NM / 8; ++i) ap[i] = a_row(row_l + 8 * i);
#pragma unroll
    for (int i = 0; i < HALVES * NN / 8; ++i) wp[i] = w_row(row_l + 8 * i);
    const int tiles = (K + NK - 1) / NK;
    auto ask = [&](int t) {
        if (t < tiles) {
            float* s = smem_f + (t % NSTAGES) * STAGE;
            const int k = t * NK + kc;
#pragma unroll
            for (int i = 0; i < NM / 8; ++i) {
                const bool in = ap[i] && k < K;
                cp16(s + (row_l + 8 * i) * NPITCH + kc, in ? ap[i] + k : any, in);
            }
#pragma unroll
            for (int i = 0; i < HALVES * NN / 8; ++i) {
                const bool in = wp[i] && k < K;
                cp16(s + (NM + row_l + 8 * i) * NPITCH + kc, in ? wp[i] + k : any, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int h = 0; h < HALVES; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[h][i] = 0.f;
#pragma unroll
    for (int t = 0; t < NSTAGES - 1; ++t) ask(t);
    const bool busy = warp * 4 < rows;
    for (int t = 0; t < tiles; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NSTAGES - 2) : "memory");
        __syncthreads();                               // tile t is there, and tile t - 1 has been used
        ask(t + NSTAGES - 1);
        if (busy) {
            const float* s = smem_f + (t % NSTAGES) * STAGE;
#pragma unroll 4
            for (int k = 0; k < NK; k += 4) {
                float4 w[HALVES];
#pragma unroll
                for (int h = 0; h < HALVES; ++h)
                    w[h] = *reinterpret_cast<const float4*>(s + (NM + h * NN + lane) * NPITCH + k);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(s + (warp * 4 + i) * NPITCH + k);
#pragma unroll
                    for (int h = 0; h < HALVES; ++h) {
                        acc[h][i] = fmaf(a.x, w[h].x, acc[h][i]);
                        acc[h][i] = fmaf(a.y, w[h].y, acc[h][i]);
                        acc[h][i] = fmaf(a.z, w[h].z, acc[h][i]);
                        acc[h][i] = fmaf(a.w, w[h].w, acc[h][i]);
                    }
                }
            }
        }
    }
}

}  // namespace f32t
}  // namespace mi
