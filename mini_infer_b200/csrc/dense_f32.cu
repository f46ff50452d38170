// Dense product of the true 32-bit path: C[T, N] = A[T, K] . W[N, K]^T, float in, float out.
//
// Every output element is one chain of fused multiply-adds over k in ascending order, whatever the number
// of rows and wherever a row lies in its tile, so a token's result does not depend on how many other
// tokens share its step: the float32 path gives the same bits for every way of cutting and batching the
// work.  (A library product picks other kernels, and other orders of summation, for other row counts.)
// CUDA cores only, no reduced-precision mode: this path exists to show faults that bfloat16 hides.
// The reference runs every dense product in FP16 through cuBLAS (src/layers/mlp.cpp:120-130).

#include "f32_tiles.cuh"

namespace mi {

// One of several independent products (a head, say) is blockIdx.z; its operands lie sA, sW, sC apart.
struct DenseF32 {
    const float* A; const float* W; float* C;
    int T, N, K, lda, ldc;
    int64_t sA, sW, sC;
};

template <int BN, bool VEC>
__global__ void __launch_bounds__(f32t::THREADS, 3)
dense_f32_wide_kernel(DenseF32 g) {
    constexpr int TN = BN / 16;
    const float* A = g.A + blockIdx.z * g.sA;
    const float* W = g.W + blockIdx.z * g.sW;
    float* C = g.C + blockIdx.z * g.sC;
    const int row0 = blockIdx.y * f32t::BM, n0 = blockIdx.x * BN;
    const f32t::WidePlace<BN> at(blockIdx.x + blockIdx.y);
    unsigned long long acc[8][TN / 2];
    const int rows = min(f32t::BM, g.T - row0);
    f32t::wide_tile<BN, VEC>(
        acc, [&](int r) { return r < rows ? A + (int64_t)(row0 + r) * g.lda : nullptr; },
        [&](int n) { return n0 + n < g.N ? W + (int64_t)(n0 + n) * g.K : nullptr; }, rows, g.K, at);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (at.r_lo + i >= rows) break;
        float* c = C + (int64_t)(row0 + at.r_lo + i) * g.ldc;
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
            const float2 v = f32t::halves_of(acc[i][j]);
            const int n = n0 + (j < TN / 4 ? at.c_lo + 2 * j : BN / 2 + at.c_lo + 2 * (j - TN / 4));
            if (n < g.N) c[n] = v.x;
            if (n + 1 < g.N) c[n + 1] = v.y;
        }
    }
}

__global__ void __launch_bounds__(f32t::THREADS)
dense_f32_narrow_kernel(DenseF32 g) {
    const float* A = g.A + blockIdx.z * g.sA;
    const float* W = g.W + blockIdx.z * g.sW;
    float* C = g.C + blockIdx.z * g.sC;
    const int n0 = blockIdx.x * f32t::NN, row0 = blockIdx.y * f32t::NM;
    const int rows = min(f32t::NM, g.T - row0);
    float acc[1][4];
    f32t::narrow_tile<1>(
        acc, [&](int r) { return r < rows ? A + (int64_t)(row0 + r) * g.lda : nullptr; },
        [&](int n) { return n0 + n < g.N ? W + (int64_t)(n0 + n) * g.K : nullptr; }, rows, g.K, A);
    const int r = (threadIdx.x >> 5) * 4, n = n0 + (threadIdx.x & 31);
    if (n >= g.N) return;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (r + i < rows) C[(int64_t)(row0 + r + i) * g.ldc + n] = acc[0][i];
}

// Which form: up to DF_NARROW_ROWS rows a product is bound by reading W, and the narrow tiles keep more of it in flight
// (against [6144, 2048], narrow and wide: 16 rows 39 and 61 us, 32 rows 53 and 61, 48 rows 65 and 66; against [2048, 5632]:
// 32 rows 66 and 163 us); above, wide tiles of 128 columns, or of 64 where those of 128 would leave SMs without one.
constexpr int DF_NARROW_ROWS = 32, DF_SMS = 148;

static int dense_f32_launch(const DenseF32& g, int batch, bool vec, cudaStream_t stream, const char* what) {
    const int64_t tiles_y = ((int64_t)g.T + f32t::BM - 1) / f32t::BM;
    if (tiles_y > 65535) { set_last_error("dense product (float32): %d rows exceed the grid limit", g.T); return kBadShape; }
    if (vec && g.T <= DF_NARROW_ROWS) {
        const size_t smem = f32t::narrow_smem(1);
        cudaFuncSetAttribute(dense_f32_narrow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        dense_f32_narrow_kernel<<<dim3((g.N + f32t::NN - 1) / f32t::NN, (g.T + f32t::NM - 1) / f32t::NM, batch), f32t::THREADS, smem, stream>>>(g);
        return finish_launch(what);
    }
    const int64_t wide = tiles_y * ((g.N + 127) / 128) * batch;
    const bool half = wide < DF_SMS;
    const int bn = half ? 64 : 128;
    const dim3 grid((g.N + bn - 1) / bn, (unsigned)tiles_y, batch);
    if (half) {
        if (vec) dense_f32_wide_kernel<64, true><<<grid, f32t::THREADS, 0, stream>>>(g);
        else dense_f32_wide_kernel<64, false><<<grid, f32t::THREADS, 0, stream>>>(g);
    } else {
        if (vec) dense_f32_wide_kernel<128, true><<<grid, f32t::THREADS, 0, stream>>>(g);
        else dense_f32_wide_kernel<128, false><<<grid, f32t::THREADS, 0, stream>>>(g);
    }
    return finish_launch(what);
}

}  // namespace mi

extern "C" int mi_dense_f32(const float* A, const float* W, float* C, int T, int N, int K, cudaStream_t stream) {
    using namespace mi;
    if (T <= 0 || N <= 0) return kOk;
    if (K <= 0) { set_last_error("dense product (float32): inner size %d", K); return kBadShape; }
    const bool vec = (K % 4 == 0) && (((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0);
    return dense_f32_launch(DenseF32{A, W, C, T, N, K, K, N, 0, 0, 0}, 1, vec, stream, "dense_f32");
}

// `batch` products at once: C_b[T, N] = A_b[T, K] . W_b[N, K]^T with rows of A and C `lda` and `ldc` floats
// apart and the operands of product b at A + b * sA, W + b * sW (rows K apart), C + b * sC: the heads of a
// row of activations, each with a matrix of its own.  The same chain of additions per element as above.
extern "C" int mi_dense_f32_batched(const float* A, const float* W, float* C, int T, int N, int K, int lda, int ldc,
                                    int batch, int64_t sA, int64_t sW, int64_t sC, cudaStream_t stream) {
    using namespace mi;
    if (T <= 0 || N <= 0 || batch <= 0) return kOk;
    if (K <= 0 || lda < K || ldc < N || batch > 65535) {
        set_last_error("batched dense product (float32): inner size %d, rows %d and %d apart, %d products", K, lda, ldc, batch);
        return kBadShape;
    }
    const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (sA % 4 == 0) && (sW % 4 == 0) &&
                     (((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0);
    return dense_f32_launch(DenseF32{A, W, C, T, N, K, lda, ldc, sA, sW, sC}, batch, vec, stream, "dense_f32_batched");
}
