// Causal attention over cache pages for any mix of rows, any head size and either storage
// type: the kernels of the float32 path and the fallback of the bfloat16 one.
//
// The first: one block per (row, query head).  The row's keys lo..pos (lo = 0, pos - window + 1 for a
// windowed layer, the first of the row's chunk for a negative `window`: first_seen_key) are visited in chunks of the block's width: each thread scores
// one key, the block takes the chunk's maximum and sum, and threads then own output
// dimensions for the weighted sum of values.  The running (max, sum, acc) update is the
// reference's online softmax (src/qwen_kernels.cu:159-176: m' = max(m, s), c = e^{m-m'},
// p = e^{s-m'}, l = l c + p, acc = acc c + p v; out = acc / l), the chunked form of it
// is the reference's two-pass block softmax (src/batched.cu:97-130).  kv_head = h / (Hq / Hkv)
// and scale applied after the dot product (src/qwen_kernels.cu:148-167).
// Chunk boundaries are counted from `lo`, so a row's summation order is the same however
// the step was cut.  `keep_first` (with a window): the request's first keys stay visible - the row then visits keys
// 0 .. min(keep_first, lo) - 1 and lo .. pos as one list.  `sink` (one logit per query head, or null): the softmax's
// denominator also holds exp(sink[h]), a key without a value; the running maximum and sum start from it.
// `cap` > 0: a score s (after the scale) becomes cap * tanh(s / cap).  `slopes` (one number per query head, or null): a
// key (pos - j) tokens back then loses slopes[h] * (pos - j).
#include "common.cuh"

#define ATTN_THREADS 128
#define ATTN_MAX_D 2048

template <typename T>
__global__ void paged_attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pages,
                                               const T* __restrict__ v_pages, const int* __restrict__ block_table,
                                               int table_stride, const int* __restrict__ positions,
                                               const int* __restrict__ row_segment, T* __restrict__ out, int Hq,
                                               int Hkv, int D, int Dv, int page_size, int window, int keep_first,
                                               const float* __restrict__ sink, float scale, float cap,
                                               const float* __restrict__ slopes, int* __restrict__ err) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ float smem[];
    float* q_s = smem;                    // [D]
    float* p_s = smem + D;                // [ATTN_THREADS]
    int* page_s = (int*)(p_s + ATTN_THREADS);  // [ATTN_THREADS] page offset of each key of the chunk
    float* scratch = (float*)(page_s + ATTN_THREADS);  // [33]

    const int r = blockIdx.x, h = blockIdx.y;
    const int hk = h / (Hq / Hkv);
    const int pos = positions[r];
    const int seg = row_segment[r];
    const int* table = block_table + (size_t)seg * table_stride;
    const int lo = first_seen_key(pos, window);
    const int kept = min(keep_first, lo);          // keys before the window that stay visible
    const int visible = kept + pos - lo + 1;
    // Values as wide as the keys lie in a pool of their own; narrower ones (Dv < D) are the first Dv numbers of the key
    // rows themselves (a latent that serves as key and as value), and `v_pages` is then the key pool.
    const int v_stride = v_pages == k_pages ? D : Dv;

    const T* qr = q + ((size_t)r * Hq + h) * D;
    for (int d = threadIdx.x; d < D; d += blockDim.x) q_s[d] = to_f32<T>(qr[d]);
    __syncthreads();

    constexpr int DPT = ATTN_MAX_D / ATTN_THREADS;  // output dims per thread
    float acc[DPT];
#pragma unroll
    for (int i = 0; i < DPT; ++i) acc[i] = 0.f;
    float m = -FLT_MAX, l = 0.f;
    const float slope = slopes ? slopes[h] : 0.f;
    if (sink) {
        m = sink[h];
        l = 1.f;
    }

    for (int base = 0; base < visible; base += ATTN_THREADS) {
        const int i = base + threadIdx.x;
        const int j = i < kept ? i : lo + (i - kept);
        float s = -FLT_MAX;
        int off = -1;
        if (i < visible) {
            const int page = table[j / page_size];
            if (page < 0) {
                atomicOr(err, KVB_DEV_BAD_PAGE);
            } else {
                off = ((page * Hkv + hk) * page_size + (j % page_size));
                const T* kr = k_pages + (size_t)off * D;
                float dot = 0.f;
                for (int d = 0; d < D; ++d) dot += q_s[d] * to_f32<T>(kr[d]);
                s = dot * scale;
                if (cap > 0.f) s = cap * tanhf(s / cap);
                if (slopes) s -= slope * (float)(pos - j);
            }
        }
        const float cmax = block_max(s, scratch);
        const float m_new = fmaxf(m, cmax);
        const float corr = expf(m - m_new);
        const float p = (off >= 0) ? expf(s - m_new) : 0.f;
        p_s[threadIdx.x] = p;
        page_s[threadIdx.x] = off;
        const float csum = block_sum(p, scratch);   // also orders the writes to p_s / page_s
        l = l * corr + csum;
        m = m_new;
        const int n = min(ATTN_THREADS, visible - base);
#pragma unroll
        for (int i = 0; i < DPT; ++i) {
            const int d = threadIdx.x + i * ATTN_THREADS;
            if (d < Dv) {
                float a = acc[i] * corr;
                for (int t = 0; t < n; ++t) {
                    const int o = page_s[t];
                    if (o >= 0) a += p_s[t] * to_f32<T>(v_pages[(size_t)o * v_stride + d]);
                }
                acc[i] = a;
            }
        }
        __syncthreads();
    }
    T* orow = out + ((size_t)r * Hq + h) * Dv;
#pragma unroll
    for (int i = 0; i < DPT; ++i) {
        const int d = threadIdx.x + i * ATTN_THREADS;
        if (d < Dv) orow[d] = from_f32<T>(l > 0.f ? acc[i] / l : 0.f);
    }
}

KVB_API int kvb_paged_attention_generic(int dtype, const void* q, const void* k_pages, const void* v_pages,
                                        const int* block_table, int table_stride, const int* positions,
                                        const int* row_segment, void* out, int T, int Hq, int Hkv, int D,
                                        int page_size, int window, float scale, int* err, cudaStream_t stream);

// The same where a row's value is the first `Dv` numbers of its key row (one pool): out is [T, Hq * Dv].
KVB_API int kvb_paged_attention_shared(int dtype, const void* q, const void* k_pages, const int* block_table, int table_stride,
                                       const int* positions, const int* row_segment, void* out, int T, int Hq, int Hkv, int D,
                                       int Dv, int page_size, int window, float scale, int* err, cudaStream_t stream);

static int launch_generic(int dtype, const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                          int table_stride, const int* positions, const int* row_segment, void* out, int T, int Hq, int Hkv,
                          int D, int Dv, int page_size, int window, float scale, int* err, cudaStream_t stream,
                          int keep_first = 0, const float* sink = nullptr, float cap = 0.f, const float* slopes = nullptr) {
    if (T <= 0) return KVB_OK;
    if (keep_first < 0) return KVB_ERR_SHAPE;
    if (window <= 0) keep_first = 0;
    if (D > ATTN_MAX_D || D < 1 || Dv < 1 || Dv > ATTN_MAX_D || (Dv > D && v_pages == k_pages) || Hkv < 1 || Hq % Hkv != 0)
        return KVB_ERR_SHAPE;
    const size_t smem = (size_t)(D + 2 * ATTN_THREADS + 33) * sizeof(float);
    dim3 grid(T, Hq);
    if (dtype == KVB_F32)
        kvb_launch(paged_attention_generic_kernel<float>, dim3(grid), dim3(ATTN_THREADS), smem, stream, 
            (const float*)q, (const float*)k_pages, (const float*)v_pages, block_table, table_stride, positions,
            row_segment, (float*)out, Hq, Hkv, D, Dv, page_size, window, keep_first, sink, scale, cap, slopes, err);
    else if (dtype == KVB_BF16)
        kvb_launch(paged_attention_generic_kernel<bf16>, dim3(grid), dim3(ATTN_THREADS), smem, stream, 
            (const bf16*)q, (const bf16*)k_pages, (const bf16*)v_pages, block_table, table_stride, positions,
            row_segment, (bf16*)out, Hq, Hkv, D, Dv, page_size, window, keep_first, sink, scale, cap, slopes, err);
    else
        return KVB_ERR_DTYPE;
    return kvb_launch_status();
}

KVB_API int kvb_paged_attention_generic(int dtype, const void* q, const void* k_pages, const void* v_pages,
                                        const int* block_table, int table_stride, const int* positions,
                                        const int* row_segment, void* out, int T, int Hq, int Hkv, int D,
                                        int page_size, int window, float scale, int* err, cudaStream_t stream) {
    if (v_pages == k_pages) return KVB_ERR_SHAPE;      // one pool for both is the other entry point's case
    return launch_generic(dtype, q, k_pages, v_pages, block_table, table_stride, positions, row_segment, out, T, Hq, Hkv, D, D,
                          page_size, window, scale, err, stream);
}

KVB_API int kvb_paged_attention_shared(int dtype, const void* q, const void* k_pages, const int* block_table, int table_stride,
                                       const int* positions, const int* row_segment, void* out, int T, int Hq, int Hkv, int D,
                                       int Dv, int page_size, int window, float scale, int* err, cudaStream_t stream) {
    return launch_generic(dtype, q, k_pages, k_pages, block_table, table_stride, positions, row_segment, out, T, Hq, Hkv, D, Dv,
                          page_size, window, scale, err, stream);
}

// Keys of D numbers and values of Dv numbers in pools of their own: out is [T, Hq * Dv].
KVB_API int kvb_paged_attention_kv(int dtype, const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                   int table_stride, const int* positions, const int* row_segment, void* out, int T, int Hq,
                                   int Hkv, int D, int Dv, int page_size, int window, float scale, int* err, cudaStream_t stream) {
    if (v_pages == k_pages) return KVB_ERR_SHAPE;
    return launch_generic(dtype, q, k_pages, v_pages, block_table, table_stride, positions, row_segment, out, T, Hq, Hkv, D, Dv,
                          page_size, window, scale, err, stream);
}

// Keys of D numbers and values of Dv numbers (pools of their own), a window that keeps the request's first `keep_first`
// keys visible, and a sink logit per query head in the softmax's denominator (`sink` null: none).
KVB_API int kvb_paged_attention_sink(int dtype, const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                     int table_stride, const int* positions, const int* row_segment, void* out, int T, int Hq,
                                     int Hkv, int D, int Dv, int page_size, int window, int keep_first, const float* sink,
                                     float scale, int* err, cudaStream_t stream) {
    if (v_pages == k_pages) return KVB_ERR_SHAPE;
    return launch_generic(dtype, q, k_pages, v_pages, block_table, table_stride, positions, row_segment, out, T, Hq, Hkv, D, Dv,
                          page_size, window, scale, err, stream, keep_first, sink);
}

// Every option at once.  `v_pages` null: a row's value is the first Dv numbers of its key row (one pool).  `window` is the
// caller's own (a layer may read a cache entry that keeps more than it sees).
KVB_API int kvb_paged_attention_ext(int dtype, const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                    int table_stride, const int* positions, const int* row_segment, void* out, int T, int Hq,
                                    int Hkv, int D, int Dv, int page_size, int window, int keep_first, const float* sink,
                                    float scale, float cap, const float* slopes, int* err, cudaStream_t stream) {
    if (cap < 0.f) return KVB_ERR_SHAPE;
    return launch_generic(dtype, q, k_pages, v_pages ? v_pages : k_pages, block_table, table_stride, positions, row_segment, out, T,
                          Hq, Hkv, D, Dv, page_size, window, scale, err, stream, keep_first, sink, cap, slopes);
}

// ---- float32, head sizes up to 128: tiles of query rows against tiles of keys ---------------------------------------------
// A block takes 16 TM rows (token, query head) of one segment and key/value head - all of them read the same keys - and walks
// the keys in tiles of 64 counted from position 0, so that a row meets the same tiles in the same order however the step was
// cut and whatever TM is: a tile of which a row sees nothing leaves its sums as they are.  Thread (ty, tx) of 16 x 16 scores
// rows ty + 16 i against keys tx + 16 j, four numbers along the head at a time, and then owns output columns 4 tx + 64 c.
// K and V tiles come in by `cp.async`, the next pair while this one is worked on (rows of K start 4 numbers off a multiple of
// 32: eight keys lie in different banks).  A row's maximum and sum run over the 16 lanes that share it.
// Bound by the shared-memory loads beside the multiply-adds in prompts, by the latency of a tile of keys in single tokens.  Measured
// against a block per (row, head), which reads every key from L2 for each of them: 1,000 rows of 14 heads of 64: 2,008 -> 117 us; 512 rows of
// 16 heads of 128 behind 2,048 keys: 9,935 -> 541 us; one token with 1,000 keys, 14 heads of 64 (two of keys): 105 -> 53 us; 64 tokens with
// 1,000 keys: 365 -> 69; eight rows of a new prompt: 5.2 -> 4.7.  The line in `CudaKernels.paged_attention`: heads of 48 and 32 numbers with
// keys of their own are ahead in prompts (160 rows of 8: 29 -> 14 and 31 -> 13 us) but behind in 64 single tokens with 30 keys (16 heads of 48: 11 -> 14 us;
// 8 of 32 level); 20 numbers: 160 rows of 3 heads in chunks of 48 tokens 7.0 -> 8.2.
namespace rows32 {

__device__ __forceinline__ void copy16(float* smem, const float* global, bool there) {
    const int bytes = there ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(global), "r"(bytes)
                 : "memory");
}

struct Params {
    const float* q;
    const float* k_pages;
    const float* v_pages;
    float* out;
    const int* block_table;
    const int* seg_q_start;
    const int* seg_q_len;
    const int* seg_kv_len;
    const float* sink;
    const float* slopes;
    int* err;
    int table_stride, segments, Hq, Hkv, D, Dv, page_size, reach, keep_first;
    float scale, cap;
};

constexpr int BN = 64, PS = BN + 4;

// acc += weights of keys k0 .. k1 - 1 (multiples of 4) of a tile . their values.  PARTIAL: a weight below zero marks a key that the row
// does not see, whose value is left out whatever it holds (a later token's may be infinite).
template <int TM, int CD, bool PARTIAL>
__device__ __forceinline__ void weigh(const float* ps, const float* vt, float4 (&acc)[TM][CD], int k0, int k1) {
    constexpr int VS = CD * 64;
#pragma unroll 2
    for (int k = k0; k < k1; k += 4) {
        float4 w[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) w[i] = *(const float4*)(ps + 16 * i * PS + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int c = 0; c < CD; ++c) {
                const float4 v = *(const float4*)(vt + (k + kk) * VS + 64 * c);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float e = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
                    if (PARTIAL && e < 0.f) continue;
                    acc[i][c].x = fmaf(e, v.x, acc[i][c].x);
                    acc[i][c].y = fmaf(e, v.y, acc[i][c].y);
                    acc[i][c].z = fmaf(e, v.z, acc[i][c].z);
                    acc[i][c].w = fmaf(e, v.w, acc[i][c].w);
                }
            }
    }
}

// s[i][j] = q row i . key 16 j, for the first NJ of the four.
template <int TM, int NJ>
__device__ __forceinline__ void score(const float* qt, const float* kt, int D, int KS, float (&s)[TM][4]) {
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
        float4 a[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = *(const float4*)(qt + 16 * i * KS + d);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const float4 b = *(const float4*)(kt + 16 * j * KS + d);
#pragma unroll
            for (int i = 0; i < TM; ++i) s[i][j] = fmaf(a[i].x, b.x, s[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i) s[i][j] = fmaf(a[i].y, b.y, s[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i) s[i][j] = fmaf(a[i].z, b.z, s[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i) s[i][j] = fmaf(a[i].w, b.w, s[i][j]);
        }
    }
}

// CD: 64-column groups of a value row; STAGES: tiles of keys held at once; NY: rows side by side, 16 threads each (16, or 4 with TM = 1).
template <int TM, int CD, int STAGES, int NY>
__global__ void __launch_bounds__(16 * NY) attention_rows_kernel(const Params p) {
    constexpr int BM = NY * TM, VS = CD * 64, THREADS = 16 * NY;
    static_assert((NY == 16 || TM == 1) && THREADS >= BN, "a thread looks up one key of a tile");
    extern __shared__ __align__(16) float sm[];
    const int KS = p.D + 4;
    float* qs = sm;                        // [BM][KS]
    float* ps = qs + BM * KS;              // [BM][PS]
    float* ks = ps + BM * PS;              // [STAGES][BN][KS]
    float* vs = ks + STAGES * BN * KS;     // [STAGES][BN][VS]
    __shared__ int where[3 * BN];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int group = p.Hq / p.Hkv, hk = blockIdx.y;
    pdl_wait();
    pdl_launch_dependents();

    // Which segment and which of its tiles: segments take ceil(rows * group / BM) blocks each, the last tiles (most keys) first.  A
    // warp counts 32 segments at a time.
    int seg = -1, tile = (int)gridDim.x - 1 - (int)blockIdx.x;
    for (int base = 0; base < p.segments; base += 32) {
        const int lane = tid & 31, mine = base + lane < p.segments ? (p.seg_q_len[base + lane] * group + BM - 1) / BM : 0;
        int upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int before = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += before;
        }
        const unsigned found = __ballot_sync(0xffffffffu, tile < upto);
        if (found) {
            const int at = __ffs(found) - 1;
            seg = base + at;
            tile -= __shfl_sync(0xffffffffu, upto - mine, at);
            break;
        }
        tile -= __shfl_sync(0xffffffffu, upto, 31);
    }
    if (seg < 0) return;
    const int q_len = p.seg_q_len[seg], q_first = p.seg_q_start[seg], start = p.seg_kv_len[seg] - q_len;
    const int m0 = tile * BM, rows = min(BM, q_len * group - m0);
    const int* table = p.block_table + (size_t)seg * p.table_stride;
    const bool working = TM > 1 || (tid >> 5) * 2 < rows;      // (one row tile) a warp whose two rows are past the end only fetches

    auto q_at = [&](int m) { return (size_t)(q_first + (m0 + m) / group) * p.Hq + hk * group + (m0 + m) % group; };
    for (int c = tid; c < BM * (p.D / 4); c += THREADS) {
        const int m = c / (p.D / 4), d = (c % (p.D / 4)) * 4;
        *(float4*)(qs + m * KS + d) = m < rows ? *(const float4*)(p.q + q_at(m) * p.D + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    int pos[TM], lo[TM];
    float m_run[TM], l_run[TM], slope[TM];
    float4 acc[TM][CD];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = min(ty + 16 * i, rows - 1), h = hk * group + (m0 + m) % group;
        pos[i] = start + (m0 + m) / group;
        lo[i] = first_seen_key(pos[i], p.reach);
        slope[i] = p.slopes ? p.slopes[h] : 0.f;
        m_run[i] = p.sink ? p.sink[h] : -FLT_MAX;
        l_run[i] = p.sink ? 1.f : 0.f;
#pragma unroll
        for (int c = 0; c < CD; ++c) acc[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int end = start + (m0 + rows - 1) / group + 1;                       // keys any row of the tile sees end here ...
    const int lo_first = first_seen_key(start + m0 / group, p.reach), lo_last = first_seen_key(end - 1, p.reach);
    const int first = lo_first / BN;                                           // ... and start in this tile, kept ones apart
    const int kept_tiles = min((min(p.keep_first, first * BN) + BN - 1) / BN, first);
    const int tiles = kept_tiles + (end + BN - 1) / BN - first;

    auto key_of = [&](int t) { return (t < kept_tiles ? t : first + t - kept_tiles) * BN; };
    // Where the keys of tile t lie (a row of the pools, or -1), looked up two tiles ahead by one thread a key.
    auto look_up = [&](int t) {
        const int j = key_of(t) + tid;
        if (t >= tiles || j >= end) return -1;
        const int page = table[j / p.page_size];
        if (page >= 0) return (page * p.Hkv + hk) * p.page_size + j % p.page_size;
        // A page is wanted only if some row of the tile sees the key (a window's earlier pages have been given back).
        if (j >= lo_first || j < p.keep_first) atomicOr(p.err, KVB_DEV_BAD_PAGE);
        return -1;
    };
    // Steps of few rows (one row tile): of a tile's keys only those k0 .. k1 - 1 that some row sees, to the next four, are fetched (from
    // the tile's first on), scored and weighed.
    auto seen_from = [&](int t) { return TM > 1 || key_of(t) < p.keep_first ? 0 : max(lo_first - key_of(t), 0) & ~3; };
    auto seen_to = [&](int t) { return TM > 1 ? BN : min(BN, ((t < kept_tiles ? p.keep_first : end) - key_of(t) + 3) & ~3); };
    auto fetch = [&](int t) {                          // a key row: 16 threads
        float* kd = ks + t % STAGES * BN * KS;
        float* vd = vs + t % STAGES * BN * VS;
        const int rows_seen = seen_to(t);
#pragma unroll
        for (int r0 = 0; r0 < BN; r0 += NY) {
            const int r = r0 + ty;
            if (TM == 1 && r >= rows_seen) break;
            const int at = where[(t % 3) * BN + r];
            const size_t row = at >= 0 ? at : 0;
            for (int d = tx * 4; d < p.D; d += 64) copy16(kd + r * KS + d, p.k_pages + row * p.D + d, at >= 0);
#pragma unroll
            for (int c = 0; c < CD; ++c) {
                const int d = tx * 4 + 64 * c;
                if (d < p.Dv) copy16(vd + r * VS + d, p.v_pages + row * p.Dv + d, at >= 0);      // (columns past a value row are never stored)
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    if (tid < BN) {
        where[tid] = look_up(0);
        where[BN + tid] = look_up(1);
    }
    __syncthreads();
    if (STAGES == 2) fetch(0);
    for (int t = 0; t < tiles; ++t) {
        if (STAGES == 1) fetch(t);
        if (STAGES == 2 && t + 1 < tiles) {
            fetch(t + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        const int later = tid < BN ? look_up(t + 2) : -1;
        __syncthreads();
        const int j0 = key_of(t);
        const float* kt = ks + t % STAGES * BN * KS + tx * KS;
        const float* vt = vs + t % STAGES * BN * VS + tx * 4;
        const float* qt = qs + ty * KS;
        float s[TM][4];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
        const int k0 = seen_from(t), k1 = seen_to(t);
        if (working) {
            if (TM == 1 && k1 <= 16) score<TM, 1>(qt, kt, p.D, KS, s);
            else score<TM, 4>(qt, kt, p.D, KS, s);
        }
        unsigned there = 0;                            // keys whose page is missing (flagged above) are seen by nobody
#pragma unroll
        for (int j = 0; j < 4; ++j) there |= where[(t % 3) * BN + tx + 16 * j] >= 0 ? 1u << j : 0u;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            if (!working) break;
            float top = -FLT_MAX;
            unsigned seen = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = j0 + tx + 16 * j;
                if ((there >> j & 1) && key <= pos[i] && (key >= lo[i] || key < p.keep_first)) {
                    float v = __fmul_rn(s[i][j], p.scale);       // one rounding sequence in every instance of the kernel
                    if (p.cap > 0.f) v = __fmul_rn(p.cap, tanhf(v / p.cap));
                    if (p.slopes) v = fmaf(-slope[i], (float)(pos[i] - key), v);
                    s[i][j] = v;
                    seen |= 1u << j;
                    top = fmaxf(top, v);
                }
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_new = fmaxf(m_run[i], top), corr = expf(m_run[i] - m_new);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = (seen >> j & 1) ? expf(s[i][j] - m_new) : 0.f;
                ps[(ty + 16 * i) * PS + tx + 16 * j] = (seen >> j & 1) ? e : -1.f;
                sum += e;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l_run[i] = fmaf(l_run[i], corr, sum);
            m_run[i] = m_new;
#pragma unroll
            for (int c = 0; c < CD; ++c) {
                acc[i][c].x *= corr; acc[i][c].y *= corr; acc[i][c].z *= corr; acc[i][c].w *= corr;
            }
        }
        const bool whole = j0 + BN - 1 <= start + m0 / group && (j0 >= lo_last || j0 + BN <= p.keep_first);
        const bool held = __syncthreads_and(there == 15u);   // (rows past the segment's last carry its last row's position)
        if (working) {
            if (whole && held) weigh<TM, CD, false>(ps + ty * PS, vt, acc, 0, BN);
            else if (k1 - k0 == BN) weigh<TM, CD, true>(ps + ty * PS, vt, acc, 0, BN);
            else weigh<TM, CD, true>(ps + ty * PS, vt, acc, k0, k1);
        }
        if (tid < BN) where[((t + 2) % 3) * BN + tid] = later;
        __syncthreads();                               // the tile's stage is free for the one after next
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = ty + 16 * i;
        if (m >= rows) continue;
        const float l = l_run[i];
#pragma unroll
        for (int c = 0; c < CD; ++c) {
            const int d = tx * 4 + 64 * c;
            if (d >= p.Dv) continue;
            const float4 a = acc[i][c];
            *(float4*)(p.out + q_at(m) * p.Dv + d) = l > 0.f ? make_float4(a.x / l, a.y / l, a.z / l, a.w / l) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

template <int TM, int CD, int STAGES = 2, int NY = 16>
static int launch(const Params& p, int T, cudaStream_t stream) {
    const int smem = (int)sizeof(float) * (NY * TM * (p.D + 4) + NY * TM * PS + STAGES * BN * (p.D + 4) + STAGES * BN * CD * 64);
    if (smem > 44 * 1024) {                            // (the kernel has some shared memory of its own beside it)
        cudaError_t e = cudaFuncSetAttribute(attention_rows_kernel<TM, CD, STAGES, NY>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
    }
    const long long blocks = ((long long)T * (p.Hq / p.Hkv) + NY * TM - 1) / (NY * TM) + p.segments;
    if (blocks > 0x7fffffffLL || p.Hkv > 65535) return KVB_ERR_LIMIT;
    kvb_launch(attention_rows_kernel<TM, CD, STAGES, NY>, dim3((unsigned)blocks, p.Hkv), dim3(16 * NY), smem, stream, p);
    return kvb_launch_status();
}

}  // namespace rows32

// float32, D and Dv up to 128 in steps of 4, every option of `kvb_paged_attention_ext`; rows by segment: segment s is rows
// seg_q_start[s] .. + seg_q_len[s], the last of its seg_kv_len[s] positions.  `seg_rows`: the longest segment's rows.
KVB_API int kvb_paged_attention_rows32(const void* q, const void* k_pages, const void* v_pages, const int* block_table, int table_stride,
                                       const int* seg_q_start, const int* seg_q_len, const int* seg_kv_len, void* out, int T,
                                       int segments, int seg_rows, int Hq, int Hkv, int D, int Dv, int page_size, int reach,
                                       int keep_first, const float* sink, float scale, float cap, const float* slopes, int* err,
                                       cudaStream_t stream) {
    if (T <= 0 || segments <= 0) return KVB_OK;
    if (D < 4 || D > 128 || D % 4 || Dv < 4 || Dv > 128 || Dv % 4 || Hkv < 1 || Hq % Hkv != 0 || v_pages == k_pages || keep_first < 0 || cap < 0.f)
        return KVB_ERR_SHAPE;
    if (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) % 16 != 0) return KVB_ERR_ALIGN;
    rows32::Params p{(const float*)q, (const float*)k_pages, (const float*)v_pages, (float*)out, block_table, seg_q_start, seg_q_len,
                     seg_kv_len, sink, slopes, err, table_stride, segments, Hq, Hkv, D, Dv, page_size, reach,
                     reach > 0 ? keep_first : 0, scale, cap};
    // The most rows a block that one segment fills and that leave every SM a block: fewer reads of the keys, more rows per load.
    const long long all = (long long)T * (Hq / Hkv), one = (long long)seg_rows * (Hq / Hkv), sms = kvb_sm_count();
    const int tm = one > 32 && (all + 63) / 64 * Hkv >= sms ? 4 : one > 16 && (all + 31) / 32 * Hkv >= sms ? 2 : 1;
    // Many segments of few rows: one stage of keys a block, so that more blocks share an SM (and for values of up to 64 numbers eight rows
    // a block).  64 single tokens behind 100 keys, 8 heads of 64 | 128, each with keys of its own: 13 | 24 us, in blocks of sixteen rows with
    // two stages 23 | 50, a block per row and head 24 | 37.
    const long long blocks = (long long)segments * Hkv;
    if (Dv <= 64 && one <= 8 && blocks > 2 * sms) return rows32::launch<1, 1, 1, 8>(p, T, stream);
    if (Dv > 64 && one <= 16 && blocks > sms) return rows32::launch<1, 2, 1>(p, T, stream);
    if (Dv <= 64) return tm == 4 ? rows32::launch<4, 1>(p, T, stream) : tm == 2 ? rows32::launch<2, 1>(p, T, stream) : rows32::launch<1, 1>(p, T, stream);
    return tm == 4 ? rows32::launch<4, 2>(p, T, stream) : tm == 2 ? rows32::launch<2, 2>(p, T, stream) : rows32::launch<1, 2>(p, T, stream);
}
