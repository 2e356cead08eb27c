// y[M, N] = x[M, K] . W[N, K]^T (+ bias), float32 accumulation on the CUDA cores.
//
// This is the matrix product of the true 32-bit path (no tensor cores, hence no
// reduced-precision mode) and the fallback of the bfloat16 path for shapes the
// tensor-core kernel refuses.  It plays the part of the reference's `linear` /
// `linear_logits` (apps/qwen_serve.cu:27-39): weights are [out, in] row-major, the
// output is the storage type or float32 (logits).
//
// Every output is one chain of multiply-adds over k = 0 .. K - 1, whatever M and the tile: a row's result does not
// depend on the rows beside it, and the shapes below differ in speed only.
//
// A warp's lanes are 4 (rows of x) x 8 (rows of W); a thread owns TM x TN outputs, rows lane + 4 i of x against rows
// lane + 8 j of W, and reads both operands four numbers along k at a time (16 bytes; rows start 4 numbers off a multiple of 32,
// so that the eight rows of W a warp reads lie in different banks).  Tiles come in by `cp.async`, STAGES - 1 of them ahead, as
// they lie in memory: nothing is transposed.  Four numbers of k cost TM + TN loads and 4 TM TN multiply-adds, so the
// large patches are bound by the FMA pipe's operands and the small ones by loads and by the length of the chain.
#include "common.cuh"

#define SIMT_PAD 16     // bytes after a row of a tile

namespace simt {

__device__ __forceinline__ void copy16(void* smem, const void* global, bool there) {
    const int bytes = there ? 16 : 0;        // nothing is read where the source is not there: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(global), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copy4(void* smem, const void* global, bool there) {
    const int bytes = there ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(global), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ float4 four(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 four(const bf16* p) {
    const uint2 v = *(const uint2*)p;
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}

// Brings rows row0 .. row0 + ROWS - 1 of src[rows, K], BK numbers at a time, to shared memory; zeros outside.  A thread copies
// the same places of every tile.  VEC: 16 bytes at a time (K a multiple of that many numbers, rows 16-byte aligned).
template <typename T, int ROWS, int BK, int THREADS, bool VEC>
struct Loader {
    static constexpr int STRIDE = BK + SIMT_PAD / (int)sizeof(T), PER = VEC ? 16 / (int)sizeof(T) : 1, CHUNKS = BK / PER;
    static constexpr int STEP = THREADS / CHUNKS, COUNT = (ROWS + STEP - 1) / STEP;
    static_assert(THREADS % CHUNKS == 0 && (ROWS % STEP == 0 || ROWS < STEP), "a thread keeps its column from row to row");
    const T* from;
    int r, k, left, K;

    __device__ __forceinline__ Loader(const T* __restrict__ src, int row0, int rows, int K_) : K(K_) {
        r = threadIdx.x / CHUNKS;
        k = (threadIdx.x % CHUNKS) * PER;
        left = min(rows - row0, ROWS) - r;              // rows of the matrix at and after this thread's first
        from = src + (size_t)(left > 0 ? row0 + r : 0) * K;
    }
    __device__ __forceinline__ void operator()(T* tile, int k0) const {
        T* dst = tile + r * STRIDE + k;
        const bool inside = k0 + k < K;
        if (ROWS < STEP && r >= ROWS) return;
#pragma unroll
        for (int i = 0; i < COUNT; ++i) {
            const bool there = inside && i * STEP < left;
            const T* at = there ? from + (size_t)i * STEP * K + k0 + k : from;
            if (VEC) copy16(dst + i * STEP * STRIDE, at, there);
            else if (sizeof(T) == 4) copy4(dst + i * STEP * STRIDE, at, there);
            else dst[i * STEP * STRIDE] = there ? *at : from_f32<T>(0.f);
        }
    }
};

template <typename TIn, typename TOut, int WARPS_M, int WARPS_N, int TM, int TN, int BK, int STAGES, bool VEC>
__global__ void __launch_bounds__(WARPS_M* WARPS_N * 32, 1)
    gemm_simt_kernel(const TIn* __restrict__ x, const TIn* __restrict__ w, const float* __restrict__ bias, TOut* __restrict__ y, int M,
                     int N, int K) {
    constexpr int THREADS = WARPS_M * WARPS_N * 32, BM = WARPS_M * TM * 4, BN = WARPS_N * TN * 8;
    constexpr int STRIDE = BK + SIMT_PAD / (int)sizeof(TIn);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TIn* xs = (TIn*)smem_raw;                         // [STAGES][BM][STRIDE]
    TIn* ws = xs + STAGES * BM * STRIDE;              // [STAGES][BN][STRIDE]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int mt = (warp / WARPS_N) * TM * 4 + lane / 8, nt = (warp % WARPS_N) * TN * 8 + lane % 8;
    const int tiles = (K + BK - 1) / BK;

    const Loader<TIn, BM, BK, THREADS, VEC> load_x(x, m0, M, K);
    const Loader<TIn, BN, BK, THREADS, VEC> load_w(w, n0, N, K);
    pdl_wait();                                       // `linear` takes any W: the launch before this one may have made it
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < tiles) {
            load_w(ws + s * BN * STRIDE, s * BK);
            load_x(xs + s * BM * STRIDE, s * BK);
        }
        copy_commit();
    }

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int t = 0; t < tiles; ++t) {
        copy_wait<STAGES - 2>();
        __syncthreads();                              // tile t is there for all, and all are done with tile t - 1
        const int next = t + STAGES - 1;
        if (next < tiles) {
            load_w(ws + (next % STAGES) * BN * STRIDE, next * BK);
            load_x(xs + (next % STAGES) * BM * STRIDE, next * BK);
        }
        copy_commit();
        const TIn* xt = xs + (t % STAGES) * BM * STRIDE + mt * STRIDE;
        const TIn* wt = ws + (t % STAGES) * BN * STRIDE + nt * STRIDE;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = four(xt + 4 * i * STRIDE + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float4 b = four(wt + 8 * j * STRIDE + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + mt + 4 * i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + nt + 8 * j;
            if (gn >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[gn];
            y[(size_t)gm * N + gn] = from_f32<TOut>(v);
        }
    }
}

template <typename TIn, typename TOut, int WARPS_M, int WARPS_N, int TM, int TN, int BK, int STAGES, bool VEC>
static int launch(const void* x, const void* w, const float* bias, void* y, int M, int N, int K, cudaStream_t stream) {
    constexpr int BM = WARPS_M * TM * 4, BN = WARPS_N * TN * 8;
    constexpr int smem = STAGES * (BM + BN) * (BK * (int)sizeof(TIn) + SIMT_PAD);
    auto kernel = gemm_simt_kernel<TIn, TOut, WARPS_M, WARPS_N, TM, TN, BK, STAGES, VEC>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
    }
    kvb_launch(kernel, dim3((N + BN - 1) / BN, (M + BM - 1) / BM), dim3(WARPS_M * WARPS_N * 32), smem, stream, (const TIn*)x,
               (const TIn*)w, bias, (TOut*)y, M, N, K);
    return kvb_launch_status();
}

// Which tile.  K is never split, so only more tiles put more SMs to work, and a block alone on an SM waits for every load: small
// tiles while there are few, larger ones (fewer loads per multiply-add) once they fill the GPU several times over.  The lines lie
// where the measured times cross (float32, L2 cold, us; 4 x 8 | 16 x 16 | 16 x 32 | 32 x 64 | 64 x 64):
//   4 x 9,728 x 896: 23 | 27 | 25 | 37 | 63         16 x 896 x 4,864: 29 | 41 | 55 | 101 | 189   16 x 9,728 x 896: 47 | 29 | 25 | 37 | 64
//   64 x 896 x 4,864: 76 | 49 | 57 | 100 | 186      128 x 896 x 4,864: 131 | 78 | 64 | 100 | 189  250 x 9,728 x 896: 496 | 215 | 155 | 127 | 134
//   1,000 x 896 x 4,864: 879 | 410 | 301 | 287 | 328   1,000 x 9,728 x 896: 1,882 | 807 | 569 | 432 | 410
// K that is no multiple of four numbers comes in 4 bytes at a time, also by cp.async (1,000 x 896 x 4,863: 340 us; with plain loads in the same
// pipeline 470, before it 427), of eight in bfloat16 by plain loads (1,000 x 896 x 4,863: 428, before 458).
// One tile of 64 x 64, transposed in registers and not fetched ahead, took 95 / 356 / 95 / 363 / 350 / 220 / 499 / 711 us; the
// library's product takes 716 us at 2,048 x 9,728 x 896, this one 940.
template <typename TIn, typename TOut, bool VEC>
static int choose(const void* x, const void* w, const float* bias, void* y, int M, int N, int K, cudaStream_t stream) {
    const long long sms = kvb_sm_count();
    auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    if (tiles(4, 8) <= 9 * sms) return launch<TIn, TOut, 1, 1, 1, 1, 32, 8, VEC>(x, w, bias, y, M, N, K, stream);
    if (tiles(16, 16) <= 2 * sms) return launch<TIn, TOut, 1, 2, 4, 1, 32, 6, VEC>(x, w, bias, y, M, N, K, stream);
    if (tiles(16, 32) <= 4 * sms || M <= 48) return launch<TIn, TOut, 1, 2, 4, 2, 32, 6, VEC>(x, w, bias, y, M, N, K, stream);
    if (tiles(64, 64) < 8 * sms) return launch<TIn, TOut, 2, 2, 4, 4, 32, 3, VEC>(x, w, bias, y, M, N, K, stream);
    return launch<TIn, TOut, 2, 2, 8, 4, 16, 4, VEC>(x, w, bias, y, M, N, K, stream);
}

template <typename TIn, typename TOut>
static int run(const void* x, const void* w, const float* bias, void* y, int M, int N, int K, cudaStream_t stream) {
    const bool vec = K % (16 / (int)sizeof(TIn)) == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0;
    return vec ? choose<TIn, TOut, true>(x, w, bias, y, M, N, K, stream) : choose<TIn, TOut, false>(x, w, bias, y, M, N, K, stream);
}

}  // namespace simt

// in_dtype / out_dtype: 0 = float32, 1 = bfloat16.
KVB_API int kvb_gemm_simt(int in_dtype, int out_dtype, const void* x, const void* w, const float* bias, void* y,
                          int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return KVB_OK;
    if (K <= 0) return KVB_ERR_SHAPE;
    if ((M + 63) / 64 > 65535) return KVB_ERR_LIMIT;
    if (in_dtype == KVB_F32 && out_dtype == KVB_F32) return simt::run<float, float>(x, w, bias, y, M, N, K, stream);
    if (in_dtype == KVB_BF16 && out_dtype == KVB_BF16) return simt::run<bf16, bf16>(x, w, bias, y, M, N, K, stream);
    if (in_dtype == KVB_BF16 && out_dtype == KVB_F32) return simt::run<bf16, float>(x, w, bias, y, M, N, K, stream);
    return KVB_ERR_DTYPE;
}
