// Dense product of the true 32-bit path: C[T, N] = A[T, K] . W[N, K]^T, float in, float out.
//
// The additions of an output element and their order follow from the inner size K alone, whatever the number
// of rows and wherever a row lies in its tile, so a token's result does not depend on how many other
// tokens share its step: the float32 path gives the same bits for every way of cutting and batching the
// work.  (A library product picks other kernels, and other orders of summation, for other row counts.)
//   K < 512    one chain of fused multiply-adds over k in ascending order, on the CUDA cores (f32_tiles.cuh)
//   K >= 512   operands taken apart exactly, into three bfloat16 numbers each, on the tensor cores; sums of 32 terms added in
//              32 bits (f32_tc.cuh).
// Off the 64-bit result, relative to its norm, here and as a chain: normal numbers 7.3e-8 and 4.0e-7 at K = 512, 9.9e-8 and 8.0e-7
// at 2048, 1.4e-7 and 1.3e-6 at 5632; positive ones 6.1e-8 and 3.1e-7, 6.5e-8 and 6.1e-7, 7.8e-8 and 1.2e-6; rows of one number 2.5e-8 both
// (a row of a single 1.0 gives the weight's bits), of 2 2.5e-8 and 3.1e-8, of 8 2.8e-8 and 5.5e-8, of 64 4.8e-8 and 1.4e-7; numbers
// of 1e-41 1.8e-6 and 4.1e-5.
// Times in us with a cold L2, tensor cores and chain.  Against [6144, 2048]: 1 row 24 and 30, 32 rows 26 and 58, 64 rows 42 and 95,
// 512 rows 114 and 295 (113 TFLOP/s), 2,048 rows 372 and 1,011; against [2048, 5632]: 26 and 60, 30 and 73, 40 and 265, 95 and 336, 337 and 1,033.
// The line at 512: there the two meet (against [2048, 512]: 1 row 11 and 11, 48 rows 21 and 30, 256 rows 30 and 28, 512 rows 28 and 38, 2,048
// rows 71 and 105), and the tensor cores' four parts of the inner dimension need four chunks of 32 each.
// The reference runs every dense product in FP16 through cuBLAS (src/layers/mlp.cpp:120-130).

#include "f32_tc.cuh"
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

// Which form: up to DF_NARROW_ROWS rows a product is bound by reading W, and the narrow tiles keep more of it in flight; above,
// wide tiles of 128 columns, or of 64 where those of 128 would leave SMs without one.  Narrow and wide in us: 32 rows against
// [6144, 256] 14 and 18, [2048, 480] 12 and 27, [512, 384] 10 and 23; 64 rows 21 and 18, 16 and 29, 10 and 23; 256 rows 53 and 33, 39 and 27,
// 14 and 23: at 32 rows the narrow tiles are faster for any number of columns, further on only for few.
constexpr int DF_NARROW_ROWS = 32;

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
    const bool half = wide < sm_count();
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

// ---- inner sizes from f32tc::TC_MIN_K on: the tensor cores (f32_tc.cuh) ----

// Rows of activations per tile and blocks per tile (1: no cluster), -1: chosen here.
struct TcForm { int nt, split; };
struct TcLaunch {
    CUtensorMap map_w;
    dim3 grid;
    int split;
    cudaStream_t stream;
    const char* what;
};

template <bool PAIRED, int NT, bool SPLIT, bool VEC>
static int f32_tc_launch_one(const f32tc::Problem& g, const TcLaunch& l) {
    auto kern = f32tc::f32_tc_kernel<PAIRED, NT, SPLIT, VEC>;
    const size_t smem = f32tc::smem_bytes(NT, l.split);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaLaunchConfig_t lc = {};
    lc.gridDim = l.grid;
    lc.blockDim = dim3(f32tc::threads(NT));
    lc.dynamicSmemBytes = smem;
    lc.stream = l.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)l.split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = SPLIT ? 1 : 0;
    cudaLaunchKernelEx(&lc, kern, l.map_w, g);
    return finish_launch(l.what);
}
template <bool PAIRED, int NT>
static int f32_tc_launch_nt(const f32tc::Problem& g, const TcLaunch& l) {
    return l.split > 1 ? f32_tc_launch_one<PAIRED, NT, true, true>(g, l) : f32_tc_launch_one<PAIRED, NT, false, true>(g, l);
}

// Rows whose parts are made ahead of a product, at most so many bytes of them at a time: a product of more rows goes in bands
// (its rows do not touch each other).
constexpr int64_t TC_SCRATCH_BYTES = 128ll << 20;
static int64_t f32_tc_row_bytes(int K) { return 6ll * ((K + f32tc::FK - 1) / f32tc::FK * f32tc::FK); }
// tiles of up to nt rows that n rows make at most
static int64_t f32_tc_tiles(int64_t n, int groups, int nt) { return groups ? (n < n / nt + groups ? n : n / nt + groups) : (n + nt - 1) / nt; }
// Rows of a tile at most.  Of 60 experts' rows, tiles of 16, 32 and 64 against [2 x 1408, 2048]: 8 rows each 268, 274 and 312 us, 13 rows 311,
// 281 and 314, 17 rows 383, 285 and 319, 34 rows 610, 424 and 337.  Chains: 1 row each (16 tokens of 4 experts) 241 us, 183 here;
// 3 rows 337 and 263; 8 rows 429 and 269; 34 rows 800 and 337; against [2048, 1408] 113 and 116, 163 and 151, 230 and 155, 431 and 198.
static int f32_tc_tile(int64_t rows, int groups, int wanted) {
    if (wanted > 0) return wanted < 64 ? wanted : 64;
    const int64_t few = groups ? 9ll * groups : 16, more = groups ? 20ll * groups : 32;
    return rows <= few ? 16 : rows <= more ? 32 : 64;
}
// floats that the parts of `rows` rows of `batch` products each, or of `groups` experts together, take
static int64_t f32_tc_scratch(int64_t rows, int K, int groups, int batch, int wanted) {
    if (!f32tc::split_before(f32_tc_tile(rows, groups, wanted))) return 0;
    const int64_t own = f32_tc_row_bytes(K), most = TC_SCRATCH_BYTES / own / batch;
    int64_t all = rows + 16 * f32_tc_tiles(rows, groups, 64);
    if (all > most) all = most > 80 ? most : 80;
    return all * batch * (own / 4);
}

// `rows`: rows in all; `groups`: experts (0: a dense product).  `scratch`: f32_tc_scratch(rows, K, groups, batch, form.nt) floats.
template <bool PAIRED>
static int f32_tc_launch(f32tc::Problem g, float* scratch, int rows, int groups, int batch, TcForm form, cudaStream_t stream,
                         const char* what) {
    // all rows of W in one map: those of the experts, or of products that lie whole rows apart
    const int64_t own_rows = (PAIRED ? 2 : 1) * (int64_t)g.N;
    const int64_t w_rows = groups ? groups * own_rows : (int64_t)(batch - 1) * (g.sW / g.K) + own_rows;
    const bool vec = g.K % 4 == 0 && g.lda % 4 == 0 && g.sA % 4 == 0 && (batch == 1 || (g.sW > 0 && g.sW % g.K == 0)) &&
                     w_rows < (1ll << 31) - 128 &&
                     ((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.W)) & 15) == 0;
    const int sms = sm_count();
    const int64_t tiles_m = PAIRED ? (g.N + 63) / 64 : (g.N + 127) / 128;
    if (batch > 65535) { set_last_error("%s: %d products exceed the grid limit", what, batch); return kBadShape; }
    int nt = f32_tc_tile(rows, groups, form.nt);
    if (!vec && nt < 32) nt = 32;
    // rows of a launch: what the scratch holds (16 rows more for a tile), or the grid
    int64_t band = 65535ll * nt;
    if (f32tc::split_before(nt)) {
        const int64_t room = f32_tc_scratch(rows, g.K, groups, batch, form.nt) / (f32_tc_row_bytes(g.K) / 4) / batch;
        band = rows;
        while (band > 0 && band + 16 * f32_tc_tiles(band, groups, nt) > room) band = band / 2 / 64 * 64;
        if (band == 0) nt = 32, band = 65535ll * nt;   // (rows that are too long, or too many experts or products)
    }
    if (f32tc::split_before(nt) && (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 15))) { set_last_error("%s: no room for the rows' parts", what); return kBadShape; }
    TcLaunch l = {};
    l.stream = stream;
    l.what = what;
    if (vec && !tc::make_map_f32(&l.map_w, g.W, (uint64_t)w_rows, (uint64_t)g.K, PAIRED ? 64 : 128)) {
        set_last_error("%s: cuTensorMapEncodeTiled failed", what);
        return kLaunchFailed;
    }
    for (int64_t r0 = 0; r0 < rows; r0 += band) {
        const int n = (int)(rows - r0 < band ? rows - r0 : band);
        const int64_t tiles_y = f32_tc_tiles(n, groups, nt);
        if (tiles_y > 65535) {
            set_last_error("%s: %d rows of %d experts exceed the grid limit", what, rows, groups);
            return kBadShape;
        }
        g.row_begin = (int)r0;
        g.row_end = (int)r0 + n;
        l.split = form.split;
        if (l.split < 0) {
            // Up to four blocks share a tile where tiles alone leave SMs without work.  By one, two and four blocks, us: one row against
            // [6144, 2048] 31, 23, 29; [2048, 2048] 29, 21, 16; [2048, 5632] 62, 37, 25; 32 rows 35, 27, 33; 35, 25, 19; 76, 45, 29.
            l.split = 1;
            while (l.split < f32tc::PARTS && 2 * l.split * tiles_m * tiles_y * batch <= sms) l.split *= 2;
        }
        if (!vec) l.split = 1;
        while (l.split > 1 && l.split < f32tc::PARTS && (f32tc::PARTS / l.split) * 2 * nt * 512u > f32tc::SLOT_LIMIT) l.split *= 2;
        l.grid = dim3((unsigned)(tiles_m * l.split), (unsigned)tiles_y, (unsigned)batch);
        if (f32tc::split_before(nt)) {
            g.parts = (uint8_t*)scratch;
            auto split_rows = vec ? f32tc::f32_split_rows_kernel<true> : f32tc::f32_split_rows_kernel<false>;
            split_rows<<<dim3((unsigned)tiles_y, (g.K + f32tc::SPLIT_K - 1) / f32tc::SPLIT_K, batch), 256, 0, stream>>>(g, nt);
            const int rc = finish_launch(what);
            if (rc != kOk) return rc;
        }
        const int rc = !vec && nt == 64 ? f32_tc_launch_one<PAIRED, 64, false, false>(g, l)
                     : !vec ? f32_tc_launch_one<PAIRED, 32, false, false>(g, l)
                     : nt == 16 ? f32_tc_launch_nt<PAIRED, 16>(g, l)
                     : nt == 32 ? f32_tc_launch_nt<PAIRED, 32>(g, l) : f32_tc_launch_nt<PAIRED, 64>(g, l);
        if (rc != kOk) return rc;
    }
    return kOk;
}

}  // namespace mi

extern "C" int mi_f32_tc_min_inner() { return mi::f32tc::TC_MIN_K; }

// Floats of scratch (16-byte aligned) that a product of `rows` rows, of `groups` experts or (0) in each of `batch` products, takes;
// nt: rows per tile, or -1 (mi_f32_tc_form).
extern "C" int64_t mi_f32_tc_scratch(int64_t rows, int K, int groups, int batch, int nt) {
    return K >= mi::f32tc::TC_MIN_K && rows > 0 && batch > 0 ? mi::f32_tc_scratch(rows, K, groups, batch, nt) : 0;
}

// `batch` products at once: C_b[T, N] = A_b[T, K] . W_b[N, K]^T with rows of A and C `lda` and `ldc` floats
// apart and the operands of product b at A + b * sA, W + b * sW (rows K apart), C + b * sC: the heads of a
// row of activations, each with a matrix of its own.  The same additions in the same order per element as above.
extern "C" int mi_dense_f32_batched(const float* A, const float* W, float* C, int T, int N, int K, int lda, int ldc,
                                    int batch, int64_t sA, int64_t sW, int64_t sC, float* scratch, int* status, cudaStream_t stream) {
    using namespace mi;
    if (T <= 0 || N <= 0 || batch <= 0) return kOk;
    if (K <= 0 || lda < K || ldc < N || batch > 65535) {
        set_last_error("dense product (float32): inner size %d, rows %d and %d apart, %d products", K, lda, ldc, batch);
        return kBadShape;
    }
    if (K >= f32tc::TC_MIN_K)
        return f32_tc_launch<false>(f32tc::Problem{A, W, C, nullptr, nullptr, N, K, lda, ldc, 0, sA, sW, sC, 0, 0, nullptr, GluForm{}, status}, scratch, T, 0,
                                    batch, TcForm{-1, -1}, stream, "dense_f32");
    const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (sA % 4 == 0) && (sW % 4 == 0) &&
                     (((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0);
    return dense_f32_launch(DenseF32{A, W, C, T, N, K, lda, ldc, sA, sW, sC}, batch, vec, stream, "dense_f32");
}

// C[T, N] = A[T, K] . W[N, K]^T.  `status` (device int, zero before the first call) receives a non-zero code if a wait inside
// the kernel ran out.
extern "C" int mi_dense_f32(const float* A, const float* W, float* C, int T, int N, int K, float* scratch, int* status,
                            cudaStream_t stream) {
    return mi_dense_f32_batched(A, W, C, T, N, K, K, N, 1, 0, 0, 0, scratch, status, stream);
}
// Grouped product of float operands (contract of mi_grouped_gemm_plain) for K >= mi_f32_tc_min_inner(); nt, split: rows of
// activations per tile and blocks per tile, or -1.  E 0 and no offsets: one dense product.
extern "C" int mi_f32_tc_form(const float* A, const int* gather, const float* W, const int* offsets, float* C, int n_rows, int E,
                              int Nout, int K, int mode, int nt, int split, int glu_kind, float glu_limit, float glu_slope,
                              const float* row_scale, float* scratch, int* status, cudaStream_t stream) {
    using namespace mi;
    if (n_rows <= 0 || Nout <= 0) return kOk;
    const bool nts = nt == -1 || nt == 16 || nt == 32 || nt == 64 || nt == 128;
    const bool splits = split == -1 || split == 1 || ((split == 2 || split == 4) && nt > 0);
    if (K < f32tc::TC_MIN_K || !nts || !splits || (E > 0) != (offsets != nullptr)) {
        set_last_error("float32 product on tensor cores: inner size %d, %d experts, tiles of %d rows by %d blocks", K, E, nt, split);
        return kBadShape;
    }
    const GluForm glu{glu_kind, glu_limit, glu_slope, mode == 1 ? row_scale : nullptr};
    const f32tc::Problem g{A, W, C, gather, offsets, Nout, K, K, Nout, E, 0, 0, 0, 0, 0, nullptr, glu, status};
    const TcForm form{nt, split};
    return mode == 1 ? f32_tc_launch<true>(g, scratch, n_rows, E, 1, form, stream, "grouped_gemm_plain")
                     : f32_tc_launch<false>(g, scratch, n_rows, E, 1, form, stream, E ? "grouped_gemm_plain" : "dense_f32");
}
