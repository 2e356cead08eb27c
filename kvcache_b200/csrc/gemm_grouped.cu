// The routed feed-forward's products for steps of many rows, on the fifth-generation tensor cores: for every row tile
// of the plan, out[rows of the tile] = act(A[rows] . W[expert of the tile]^T), with tcgen05.mma, the accumulator in
// tensor memory and operands brought into 128-byte-swizzled shared memory by TMA - the warp roles, the stage ring, the
// two accumulators and the bounded waits of the engine's plain product (gemm_tcgen05.cu), with the tiles taken from a
// list that a kernel wrote instead of from M and N.
//
// Rows are (token, choice) pairs sorted by expert; every expert's run is padded to whole tiles of 128 rows, so a tile
// never holds rows of two experts and the padding rows (whatever they contain) are computed and never stored.
// A is [row capacity, K]; W is the experts' matrices stacked, [experts * N, K]; tile i of the plan is
// (expert, first row, rows in use); plan[0] is the number of tiles.  Columns beyond N, up to the next multiple of 64, run
// into the next expert's rows in shared memory and are masked at the store.  K % 8 == 0 (the 16-byte stride rule of TMA).
//
// With many tiles a block is bound by what it brings from L2 (48 KB for 512 clocks of tensor work); with few rows an
// expert by reading the experts' matrices.  Storing a tile must stay below that: eight warps store (four before), a row's
// 16 results by one 32-byte store, and the gated activation takes one reciprocal instruction instead of an IEEE division,
// which alone held 16 divisions for every 32 columns of a row; the reciprocal is within 1 ulp and the result is rounded to
// 8 bits (28 layers against 64 bits: errors the same to 1e-5 of themselves, either way).  2,048 rows to 2 of 16 experts (L2 flushed, launch included): up 2432 x 896 52.2 -> 37.6 us, down 896 x 1216
// 31.3 -> 25.6 us; to 4 of 32 experts, up 2752 x 2048 113.6 -> 105.3 us, down 2048 x 1376 71.7 -> 69.6 us.
#include "tc_common.cuh"

namespace tc {

constexpr int BM = 128, BK = 64, BN = 256, BOX = 64;     // BN: columns of a tile at most; BOX: rows of W a copy brings
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES, BOX_BYTES = BOX * BK * 2;
constexpr int STAGES = 4, STORE_WARPS = 8, THREADS = 64 + 32 * STORE_WARPS;

struct Shared {
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
    uint64_t accum_full[2];
    uint64_t accum_empty[2];
    uint32_t tmem_base;
    int failed;
};

__device__ __forceinline__ float over_one_plus_exp(float num, float z) {       // num / (1 + e^z)
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(1.f + __expf(z)));
    return num * r;
}

// 16 results of one row to memory.  32 bytes at once where `wide` (the address is a multiple of 32), 16 where `vector`.
__device__ __forceinline__ void store16(const float* v, bf16* __restrict__ out, int left, bool vector, bool wide) {
    uint32_t p[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        __nv_bfloat162 v2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        p[i] = *reinterpret_cast<uint32_t*>(&v2);
    }
    if (wide && left >= 16) {
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(out), "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]),
                     "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]) : "memory");
    } else if (vector && left >= 16) {
        reinterpret_cast<uint4*>(out)[0] = make_uint4(p[0], p[1], p[2], p[3]);
        reinterpret_cast<uint4*>(out)[1] = make_uint4(p[4], p[5], p[6], p[7]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (i < left) out[i] = __float2bfloat16_rn(v[i]);
    }
}

// 32 consecutive accumulator columns of one row on their way to memory (`cols` of them are real); ACT 1: relu(v)^2.
// ACT 2: the columns are (gate, up) pairs and `out` points at the 16 results: g' sigmoid(1.702 g') (u' + 1), g' = min(g, limit),
// u' = clamp(u, +-limit); limit <= 0: silu(g) u.
template <int ACT>
__device__ __forceinline__ void store_chunk(const uint32_t* r, bf16* __restrict__ out, int cols, bool vector, bool wide, float limit) {
    float v[16];
    if constexpr (ACT == 2) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float g = __uint_as_float(r[2 * i]), u = __uint_as_float(r[2 * i + 1]);
            if (limit <= 0.f) {
                v[i] = over_one_plus_exp(g, -g) * u;
            } else {
                const float gc = fminf(g, limit), uc = fminf(fmaxf(u, -limit), limit);
                v[i] = over_one_plus_exp(gc, -1.702f * gc) * (uc + 1.f);
            }
        }
        store16(v, out, cols >> 1, vector, wide);
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                v[i] = __uint_as_float(r[16 * h + i]);
                if (ACT == 1) {
                    v[i] = fmaxf(v[i], 0.f);
                    v[i] *= v[i];
                }
            }
            store16(v, out + 16 * h, cols - 16 * h, vector, wide);
        }
    }
}

// The columns of a tile, 256, 192 or 128: whichever gives the block with the most tiles the fewest rows of A and W to bring
// in, the wider one where they are level.  Measured, 256 / 192 / 128 columns: 39 row tiles of 896 columns 27.6 / 26.7 / 24.7 us
// (128 taken), 23 of 896 21.3 / 20.5 / 24.6 (192), 39 of 2432 37.7 / 39.7 / 43.0 (256), 79 of 2752 105.4 / 115.6 / 139.4 (256).
__device__ __forceinline__ int tile_columns(int row_tiles, int N, int blocks) {
    int best = 0, best_rows = 0x7fffffff;
#pragma unroll
    for (int bn = BN; bn >= 128; bn -= 64) {
        const int rows = (row_tiles * ((N + bn - 1) / bn) + blocks - 1) / blocks * (BM + bn);
        if (rows < best_rows) { best_rows = rows; best = bn; }
    }
    return best;
}

template <int ACT>
__global__ void __launch_bounds__(THREADS, 1)
grouped_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, bf16* __restrict__ out,
                       const int* __restrict__ plan, const int* __restrict__ tile_list, int N, int K, float limit,
                       int* __restrict__ err) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ Shared sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kblocks = (K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&sh.full[s], 1); mbar_init(&sh.empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&sh.accum_full[b], 1); mbar_init(&sh.accum_empty[b], STORE_WARPS); }
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sh.tmem_base)), "r"(2 * BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = sh.tmem_base;
    pdl_wait();                                          // the plan and the rows are there from here on
    pdl_launch_dependents();
    const int row_tiles = plan[0], bn = tile_columns(row_tiles, N, gridDim.x);
    const int n_blocks = (N + bn - 1) / bn;
    const int num_tiles = row_tiles * n_blocks;

    // Tile t: row tile t / n_blocks of the plan, column block t % n_blocks (the column blocks of a row tile run side by side).
    if (warp == 0) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_w) : "memory");
            uint32_t it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                const int* t = tile_list + 3 * (tile / n_blocks);
                const int row0 = t[1], n0 = (tile % n_blocks) * bn, w_row = t[0] * N + n0;
                const int boxes = (min(bn, N - n0) + BOX - 1) / BOX;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t round = it / STAGES;
                    if (round > 0 && !mbar_wait(&sh.empty[s], (round - 1) & 1)) { atomicOr(err, KVB_DEV_TIMEOUT); sh.failed = 1; ok = false; break; }
                    mbar_expect_tx(&sh.full[s], A_BYTES + boxes * BOX_BYTES);
                    tma_load_2d(tiles + s * STAGE_BYTES, &map_a, kb * BK, row0, &sh.full[s]);
                    for (int j = 0; j < boxes; ++j)
                        tma_load_2d(tiles + s * STAGE_BYTES + A_BYTES + j * BOX_BYTES, &map_w, kb * BK, w_row + j * BOX, &sh.full[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t it = 0, local = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++local) {
                const int b = local & 1;
                const uint32_t use = local >> 1;
                const uint32_t idesc = instr_desc(BM, (min(bn, N - (tile % n_blocks) * bn) + BOX - 1) / BOX * BOX);
                if (use > 0 && !mbar_wait(&sh.accum_empty[b], (use - 1) & 1)) { atomicOr(err, KVB_DEV_TIMEOUT); sh.failed = 1; ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t acc = tmem + b * BN;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(&sh.full[s], (it / STAGES) & 1)) { atomicOr(err, KVB_DEV_TIMEOUT); sh.failed = 1; ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t a_addr = smem_u32(tiles + s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
                    const uint64_t adesc = smem_desc(a_addr), bdesc = smem_desc(b_addr);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma(acc, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                    umma_commit(&sh.empty[s]);
                }
                umma_commit(&sh.accum_full[b]);
            }
        }
    } else {
        // Two warps for each quarter of the accumulator's rows; they take its chunks of 32 columns in turn.
        const int quarter = warp & 3, first = (warp - 2) >> 2;
        const int out_cols = ACT == 2 ? N >> 1 : N;
        const bool vector = out_cols % 8 == 0, wide = out_cols % 16 == 0 && ((uintptr_t)out & 31) == 0;
        uint32_t local = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++local) {
            const int* t = tile_list + 3 * (tile / n_blocks);
            const int row0 = t[1], rows = t[2], n0 = (tile % n_blocks) * bn;
            const int b = local & 1;
            const int m = quarter * 32 + lane;
            ok = mbar_wait(&sh.accum_full[b], (local >> 1) & 1);
            if (!ok) { if (lane == 0) { atomicOr(err, KVB_DEV_TIMEOUT); sh.failed = 1; } break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
            for (int c = first; c * 32 < min(bn, N - n0); c += STORE_WARPS / 4) {
                uint32_t r[32];
                tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + b * BN + c * 32, r);
                const int n = n0 + c * 32;
                if (m >= rows) continue;
                store_chunk<ACT>(r, out + (size_t)(row0 + m) * out_cols + (ACT == 2 ? n >> 1 : n), N - n, vector, wide, limit);
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.accum_empty[b]);
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (sh.failed && threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) mbar_wait(&sh.full[s], 0);
    }
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(2 * BN) : "memory");
    }
}

// xs[place[p], :] = x[p / top, :] for every (row, choice) pair p: the step's rows in the order of the plan.
__global__ void gather_rows_kernel(const bf16* __restrict__ x, const int* __restrict__ place, bf16* __restrict__ xs, int top, int K) {
    pdl_wait();
    pdl_launch_dependents();
    const int p = blockIdx.x;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(p / top) * K);
    uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)place[p] * K);
    for (int i = threadIdx.x; i < K / 8; i += blockDim.x) dst[i] = src[i];
}

static int sm_count() {
    static int count = 0;
    if (!count) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    }
    return count;
}

}  // namespace tc

KVB_API int kvb_gather_rows(const void* x, const int* place, void* xs, int pairs, int top, int K, cudaStream_t stream) {
    if (pairs <= 0) return KVB_OK;
    if (K % 8 != 0 || top < 1) return KVB_ERR_SHAPE;
    kvb_launch(tc::gather_rows_kernel, dim3(pairs), dim3(128), 0, stream, (const bf16*)x, place, (bf16*)xs, top, K);
    return kvb_launch_status();
}

// a [row_capacity, K] in the plan's order (runs padded to 128 rows), w [experts * N, K], out [row_capacity, N] (act 2:
// [row_capacity, N / 2]); `max_tiles` bounds the plan's row tiles.
static int grouped_tcgen05(const void* a, const void* w, void* out, const int* plan, const int* tile_list, int max_tiles,
                           int row_capacity, int experts, int N, int K, int act, float limit, int* err, cudaStream_t stream) {
    using namespace tc;
    if (max_tiles <= 0) return KVB_OK;
    if (K % 8 != 0 || N < 1 || act < 0 || act > 2 || (act == 2 && N % 2 != 0)) return KVB_ERR_SHAPE;
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)out) % 16 != 0) return KVB_ERR_ALIGN;
    CUtensorMap ma, mw;
    int rc = make_bf16_map(&ma, a, row_capacity, K, K, BM);
    if (rc != KVB_OK) return rc;
    rc = make_bf16_map(&mw, w, (long long)experts * N, K, K, BOX);
    if (rc != KVB_OK) return rc;
    const size_t smem = (size_t)STAGES * STAGE_BYTES + 1024;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(grouped_tcgen05_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(grouped_tcgen05_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(grouped_tcgen05_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const long long tiles = (long long)max_tiles * ((N + 127) / 128);
    const int blocks = tiles < sm_count() ? (int)tiles : sm_count();
    auto kernel = act == 2 ? grouped_tcgen05_kernel<2> : act == 1 ? grouped_tcgen05_kernel<1> : grouped_tcgen05_kernel<0>;
    kvb_launch(kernel, dim3(blocks), dim3(THREADS), smem, stream, ma, mw, (bf16*)out, plan, tile_list, N, K, limit, err);
    return kvb_launch_status();
}

KVB_API int kvb_grouped_gemm_tcgen05(const void* a, const void* w, void* out, const int* plan, const int* tile_list, int max_tiles,
                                     int row_capacity, int experts, int N, int K, int act, int* err, cudaStream_t stream) {
    if (act > 1) return KVB_ERR_SHAPE;
    return grouped_tcgen05(a, w, out, plan, tile_list, max_tiles, row_capacity, experts, N, K, act, 0.f, err, stream);
}

// The same with the activation's constant: act 2 is the clamped gated activation of (gate, up) column pairs with `limit`.
KVB_API int kvb_grouped_gemm_tcgen05_act(const void* a, const void* w, void* out, const int* plan, const int* tile_list,
                                         int max_tiles, int row_capacity, int experts, int N, int K, int act, float limit, int* err,
                                         cudaStream_t stream) {
    return grouped_tcgen05(a, w, out, plan, tile_list, max_tiles, row_capacity, experts, N, K, act, limit, err, stream);
}
