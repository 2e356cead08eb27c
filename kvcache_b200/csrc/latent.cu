// Operators of the latent-attention mixer and of blocks that normalise a sublayer's result before adding it.
//
//   norm_add_rmsnorm          h += norm(delta [* sigmoid(gate)]; dw) (or delta as it is), out = norm(h; w) (or h as it is) [| tail]
//   latent_norm_rope_append   the two latents of a row normalised, the shared key part rotated, the cache row written
//   head_linear               one small matrix product per head: out[t, h, :N] = x[t, h, :K] . W[h]^T, with the rotation
//                             of the head's trailing columns or a sigmoid gate in its epilogue
//
// Everything between loads and stores is float32: sums of squares, norms, angles, the gate.  Reductions run in a
// fixed order per row (`block_sum`), so a row's result does not depend on the rows beside it.
#include "common.cuh"
#include "mma_tile.cuh"

// ---------------------------------------------------------------------------------------------------------------
// One block per output row.  d = delta[r] (times sigmoid(gate[r]), element by element, if gate);
// v = h[r] + (dw ? d * rsqrt(mean(d^2) + deps) * dw : d); rows == null: h[r] = v.
// out[o, :H] = w ? v * rsqrt(mean(v^2) + eps) * w : v;  out[o, H:2H] = tail[r] if tail.  The row lives in shared memory.
template <typename T>
__global__ void norm_add_rmsnorm_kernel(float* __restrict__ h, const T* __restrict__ delta, const T* __restrict__ gate,
                                        const float* __restrict__ dw, float deps, const float* __restrict__ w, float eps,
                                        T* __restrict__ out, const int* __restrict__ rows, const float* __restrict__ tail, int H) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ float row_s[];          // [H] then 33 of scratch, then [H] for the gated delta if there is a gate
    float* scratch = row_s + H;
    float* gated_s = scratch + 33;
    const int o = blockIdx.x;
    const int r = rows ? rows[o] : o;
    float* hr = h + (size_t)r * H;
    const T* dr = delta ? delta + (size_t)r * H : nullptr;
    const T* gr = (delta && gate) ? gate + (size_t)r * H : nullptr;
    float dinv = 1.f;
    if (gr) {
        for (int i = threadIdx.x; i < H; i += blockDim.x)     // each thread reads back what it wrote itself
            gated_s[i] = to_f32<T>(dr[i]) / (1.f + expf(-to_f32<T>(gr[i])));
    }
    auto d_at = [&](int i) { return gr ? gated_s[i] : to_f32<T>(dr[i]); };
    if (dr && dw) {
        float ss = 0.f;
        for (int i = threadIdx.x; i < H; i += blockDim.x) {
            const float d = d_at(i);
            ss += d * d;
        }
        dinv = 1.f / sqrtf(block_sum(ss, scratch) / (float)H + deps);
    }
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float v = hr[i];
        if (dr) v += dw ? d_at(i) * dinv * dw[i] : d_at(i);
        if (dr && !rows) hr[i] = v;
        row_s[i] = v;
        ss += v * v;
    }
    if (!out) return;
    float inv = 1.f;
    if (w) inv = 1.f / sqrtf(block_sum(ss, scratch) / (float)H + eps);
    const int stride = tail ? 2 * H : H;
    T* orow = out + (size_t)o * stride;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {     // each thread reads back what it wrote itself
        orow[i] = from_f32<T>(w ? row_s[i] * inv * w[i] : row_s[i]);
        if (tail) orow[H + i] = from_f32<T>(tail[(size_t)r * H + i]);
    }
}

KVB_API int kvb_norm_add_rmsnorm(int dtype, float* h, const void* delta, const void* gate, const float* dw, float deps,
                                 const float* w, float eps, void* out, const int* rows, const float* tail, int n_rows, int H,
                                 cudaStream_t stream) {
    if (n_rows <= 0) return KVB_OK;
    if (H < 1) return KVB_ERR_SHAPE;
    const size_t smem = (size_t)((gate ? 2 : 1) * H + 33) * sizeof(float);
    if (smem > 200 * 1024) return KVB_ERR_LIMIT;
    const int threads = H >= 2048 ? 512 : (H >= 512 ? 256 : 128);
    if (dtype == KVB_F32) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(norm_add_rmsnorm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kvb_launch(norm_add_rmsnorm_kernel<float>, dim3(n_rows), dim3(threads), smem, stream, h, (const float*)delta, (const float*)gate,
                   dw, deps, w, eps, (float*)out, rows, tail, H);
    } else if (dtype == KVB_BF16) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(norm_add_rmsnorm_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kvb_launch(norm_add_rmsnorm_kernel<bf16>, dim3(n_rows), dim3(threads), smem, stream, h, (const bf16*)delta, (const bf16*)gate,
                   dw, deps, w, eps, (bf16*)out, rows, tail, H);
    } else {
        return KVB_ERR_DTYPE;
    }
    return kvb_launch_status();
}

// ---------------------------------------------------------------------------------------------------------------
// One block per row of the fused projection `proj` [T, P]: columns [0, q_rank) are the query latent (q_rank 0: there is
// none, and cq is not written), [kv_col, kv_col + kv_rank) the key/value latent, the next rot_dim the key part that all
// heads share.
//   cq[r]                 = norm(query latent; qw)
//   cache row of (r's request, r's position) = [norm(key/value latent; kw) | R_pos(shared key part)]
// R rotates the first 2 * rot_half numbers (t pairs with t + rot_half); the rest pass unchanged.
template <typename T>
__global__ void latent_norm_rope_append_kernel(const T* __restrict__ proj, int P, int q_rank, int kv_col, int kv_rank, int rot_dim,
                                               const float* __restrict__ qw, const float* __restrict__ kw, float eps,
                                               const float* __restrict__ cos_t, const float* __restrict__ sin_t, int rot_half,
                                               int table_len, const int* __restrict__ positions,
                                               const int* __restrict__ row_segment, const int* __restrict__ block_table,
                                               int table_stride, T* __restrict__ k_pages, int page_size, int write_kv,
                                               T* __restrict__ cq, int* __restrict__ err) {
    __shared__ float scratch[33];
    const int r = blockIdx.x;
    const int pos = positions[r];
    const int key_dim = kv_rank + rot_dim;
    T* dst = nullptr;
    if (write_kv) {
        const int page = block_table[(size_t)row_segment[r] * table_stride + pos / page_size];
        if (page < 0) {
            if (threadIdx.x == 0) atomicOr(err, KVB_DEV_BAD_PAGE);
        } else {
            dst = k_pages + ((size_t)page * page_size + (pos % page_size)) * key_dim;
        }
    }
    const bool pos_ok = pos >= 0 && pos < table_len;
    if (!pos_ok && threadIdx.x == 0) atomicOr(err, KVB_DEV_BAD_POS);
    const float* cr = cos_t + (size_t)(pos_ok ? pos : 0) * rot_half;
    const float* sr = sin_t + (size_t)(pos_ok ? pos : 0) * rot_half;
    pdl_wait();
    pdl_launch_dependents();
    const T* src = proj + (size_t)r * P;
    float sq = 0.f, sk = 0.f;
    for (int i = threadIdx.x; i < q_rank; i += blockDim.x) {
        const float v = to_f32<T>(src[i]);
        sq += v * v;
    }
    for (int i = threadIdx.x; i < kv_rank; i += blockDim.x) {
        const float v = to_f32<T>(src[kv_col + i]);
        sk += v * v;
    }
    const float qinv = q_rank > 0 ? 1.f / sqrtf(block_sum(sq, scratch) / (float)q_rank + eps) : 0.f;
    const float kinv = 1.f / sqrtf(block_sum(sk, scratch) / (float)kv_rank + eps);
    for (int i = threadIdx.x; i < q_rank; i += blockDim.x)
        cq[(size_t)r * q_rank + i] = from_f32<T>(to_f32<T>(src[i]) * qinv * qw[i]);
    if (!dst) return;
    for (int i = threadIdx.x; i < kv_rank; i += blockDim.x) dst[i] = from_f32<T>(to_f32<T>(src[kv_col + i]) * kinv * kw[i]);
    const T* kr = src + kv_col + kv_rank;
    for (int i = threadIdx.x; i < rot_dim; i += blockDim.x) {
        float x = to_f32<T>(kr[i]);
        if (i < 2 * rot_half) {
            const bool low = i < rot_half;
            const int t = low ? i : i - rot_half;
            const float xp = to_f32<T>(kr[low ? i + rot_half : i - rot_half]);
            x = low ? (x * cr[t] - xp * sr[t]) : (x * cr[t] + xp * sr[t]);
        }
        dst[kv_rank + i] = from_f32<T>(x);
    }
}

KVB_API int kvb_latent_norm_rope_append(int dtype, const void* proj, int P, int q_rank, int kv_col, int kv_rank, int rot_dim, const float* qw,
                                        const float* kw, float eps, const float* cos_t, const float* sin_t, int rot_half,
                                        int table_len, const int* positions, const int* row_segment, const int* block_table,
                                        int table_stride, void* k_pages, int page_size, int write_kv, void* cq, int T,
                                        int* err, cudaStream_t stream) {
    if (T <= 0) return KVB_OK;
    if (q_rank < 0 || kv_col < q_rank || kv_rank < 1 || rot_dim < 0 || 2 * rot_half > rot_dim || kv_col + kv_rank + rot_dim > P ||
        (q_rank > 0 && (qw == nullptr || cq == nullptr)))
        return KVB_ERR_SHAPE;
    const int threads = 128;
    if (dtype == KVB_F32)
        kvb_launch(latent_norm_rope_append_kernel<float>, dim3(T), dim3(threads), 0, stream, (const float*)proj, P, q_rank, kv_col, kv_rank,
                   rot_dim, qw, kw, eps, cos_t, sin_t, rot_half, table_len, positions, row_segment, block_table, table_stride,
                   (float*)k_pages, page_size, write_kv, (float*)cq, err);
    else if (dtype == KVB_BF16)
        kvb_launch(latent_norm_rope_append_kernel<bf16>, dim3(T), dim3(threads), 0, stream, (const bf16*)proj, P, q_rank, kv_col, kv_rank,
                   rot_dim, qw, kw, eps, cos_t, sin_t, rot_half, table_len, positions, row_segment, block_table, table_stride,
                   (bf16*)k_pages, page_size, write_kv, (bf16*)cq, err);
    else
        return KVB_ERR_DTYPE;
    return kvb_launch_status();
}

// ---------------------------------------------------------------------------------------------------------------
// What attention over an expanded latent starts from, in one launch.  The first 32 * n_blocks blocks copy four cached rows each:
// the keys of a list of blocks of 128 (segment, first key) out of the pages, the latent into lat [128 n_blocks, C], the rotated part
// into rot [128 n_blocks, 64]; rows beyond the segment's keys, rows before the first key that a window of `window` keys leaves its first
// row (their pages may have been given back) and columns beyond the rotated part are zeros.  The others rotate
// the queries where they lie: the last `rot_dim` numbers of each head of q (rows of `q_ld`, heads of dim + rot_dim), by the row's position.
// Bound by launch and latency: 2,048 keys of 576 numbers and 16 heads of 64 rotated numbers are 13 MB, 2 us of them.  VEC pairs a
// thread: eight, 16 bytes a load, where the halves of the rotated part are steps of eight (2,048 rows of 16 heads: 10.8 us with one a thread, 4.4 with eight).
template <int VEC>
__global__ void __launch_bounds__(128) latent_expand_prepare_kernel(
    const bf16* __restrict__ k_pages, const int* __restrict__ block_table, int table_stride, int page_size, const int* __restrict__ blocks,
    int n_blocks, const int* __restrict__ seg_q_len, const int* __restrict__ seg_kv_len, int window, int C, int rot_dim, bf16* __restrict__ lat, bf16* __restrict__ rot, bf16* __restrict__ q,
    int q_ld, int H, int dim, const float* __restrict__ cos_t, const float* __restrict__ sin_t, int rot_half, int table_len,
    const int* __restrict__ positions, int T, int* __restrict__ err) {
    const int copies = 32 * n_blocks, tid = threadIdx.x;
    if ((int)blockIdx.x < copies) {
        const int row = 4 * blockIdx.x + (tid >> 5), lane = tid & 31;      // a warp a row
        const int seg = blocks[2 * (row >> 7)], key = blocks[2 * (row >> 7) + 1] + (row & 127);
        const bf16* src = nullptr;
        const int kv_len = seg_kv_len[seg];
        if (key < kv_len && key >= first_seen_key(kv_len - seg_q_len[seg], window)) {
            const int page = block_table[(size_t)seg * table_stride + key / page_size];
            if (page < 0) {
                if (lane == 0) atomicOr(err, KVB_DEV_BAD_PAGE);
            } else {
                src = k_pages + ((size_t)page * page_size + key % page_size) * (C + rot_dim);
            }
        }
        pdl_wait();
        pdl_launch_dependents();
        const uint4 zero = make_uint4(0, 0, 0, 0);
        for (int c = lane; c < C / 8; c += 32)
            reinterpret_cast<uint4*>(lat + (size_t)row * C)[c] = src ? reinterpret_cast<const uint4*>(src)[c] : zero;
        if (lane < 8) reinterpret_cast<uint4*>(rot + (size_t)row * 64)[lane] = src && lane < rot_dim / 8 ? reinterpret_cast<const uint4*>(src + C)[lane] : zero;
        return;
    }
    const int parts = rot_half / VEC, at = (blockIdx.x - copies) * 128 + tid;       // (row, head, VEC pairs)
    const int t = at / (H * parts);
    int pos = 0;
    if (t < T) {
        pos = positions[t];
        if (pos < 0 || pos >= table_len) { atomicOr(err, KVB_DEV_BAD_POS); pos = 0; }
    }
    pdl_wait();
    pdl_launch_dependents();
    if (t >= T) return;
    const int rest = at - t * H * parts, h = rest / parts, i = (rest - h * parts) * VEC;
    bf16* x = q + (size_t)t * q_ld + h * (dim + rot_dim) + dim + i;
    const float *c = cos_t + (size_t)pos * rot_half + i, *s = sin_t + (size_t)pos * rot_half + i;
    __align__(16) bf16 lo[VEC], hi[VEC];
    if constexpr (VEC == 8) {
        *reinterpret_cast<uint4*>(lo) = *reinterpret_cast<const uint4*>(x);
        *reinterpret_cast<uint4*>(hi) = *reinterpret_cast<const uint4*>(x + rot_half);
    } else {
        lo[0] = x[0]; hi[0] = x[rot_half];
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
        const float u = __bfloat162float(lo[e]), v = __bfloat162float(hi[e]);
        lo[e] = __float2bfloat16_rn(u * c[e] - v * s[e]);
        hi[e] = __float2bfloat16_rn(v * c[e] + u * s[e]);
    }
    if constexpr (VEC == 8) {
        *reinterpret_cast<uint4*>(x) = *reinterpret_cast<const uint4*>(lo);
        *reinterpret_cast<uint4*>(x + rot_half) = *reinterpret_cast<const uint4*>(hi);
    } else {
        x[0] = lo[0]; x[rot_half] = hi[0];
    }
}

// blocks: int32 [n_blocks, 2] (segment, first key of 128); window: keys that a row sees (0: all).  Latents and rotated parts in steps of eight numbers, rows on 16 bytes.
KVB_API int kvb_latent_expand_prepare(const void* k_pages, const int* block_table, int table_stride, int page_size, const int* blocks, int n_blocks,
                                      const int* seg_q_len, const int* seg_kv_len, int window, int C, int rot_dim, void* lat, void* rot, void* q, int q_ld, int H, int dim,
                                      const float* cos_t, const float* sin_t, int rot_half, int table_len, const int* positions, int T,
                                      int* err, cudaStream_t stream) {
    if (T <= 0 || n_blocks <= 0) return KVB_OK;
    if (C < 8 || C % 8 != 0 || rot_dim < 8 || rot_dim > 64 || rot_dim % 8 != 0 || rot_half < 0 || 2 * rot_half > rot_dim || page_size < 1 ||
        window < 0 || H < 1 || H * (dim + rot_dim) > q_ld || (long long)T * H * rot_half > 0x7fffff00LL)
        return KVB_ERR_SHAPE;
    if (((uintptr_t)k_pages | (uintptr_t)lat | (uintptr_t)rot) & 15) return KVB_ERR_ALIGN;
    const bool eights = rot_half % 8 == 0 && dim % 8 == 0 && q_ld % 8 == 0 && !((uintptr_t)q & 15);
    const int turns = (T * H * rot_half / (eights ? 8 : 1) + 127) / 128;
    kvb_launch(eights ? latent_expand_prepare_kernel<8> : latent_expand_prepare_kernel<1>, dim3(32 * n_blocks + turns), dim3(128), 0, stream, (const bf16*)k_pages, block_table, table_stride,
               page_size, blocks, n_blocks, seg_q_len, seg_kv_len, window, C, rot_dim, (bf16*)lat, (bf16*)rot, (bf16*)q, q_ld, H, dim, cos_t, sin_t, rot_half,
               table_len, positions, T, err);
    return kvb_launch_status();
}

// ---------------------------------------------------------------------------------------------------------------
// out[t, h * os + n] = sum_k x[t, h * xs + k] * w[h, n, k]   (n < N, k < K), float32 accumulation on the CUDA cores:
// the form of the true 32-bit path and of shapes the tensor-core form refuses.  Tiles of BM x 64 outputs of one head,
// 16 of K at a time, K walked in the same order whatever T is.
//   gate:    out *= sigmoid(gate[t * gs + gc + h * os + n]), or, with `gate_heads`, sigmoid(gate[t * gs + gc + h]) (one number a head)
//   x_ld:    elements between rows of x (the heads' inputs may be columns of wider rows)
//   rot > 0: the head's trailing columns x[t, h * xs + K + i], i < rot, are rotated by the row's position (first
//            2 * rot_half of them; pair (i, i + rot_half)) and stored at out[t, h * os + N + i].
template <typename T, int BM>
__global__ void __launch_bounds__(256) head_linear_simt_kernel(const T* __restrict__ x, int xs, int x_ld, const T* __restrict__ w,
                                                               T* __restrict__ out, int os, int M, int N, int K, int H,
                                                               const T* __restrict__ gate, int gs, int gc, int gate_heads, int rot, int rot_half,
                                                               const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                                               int table_len, const int* __restrict__ positions,
                                                               int* __restrict__ err) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int BN = 64, BK = 16, TM = BM / 16;
    __shared__ float xs_s[BK][BM + 4];
    __shared__ float ws_s[BK][BN + 4];
    const int tid = threadIdx.x;
    const int ty = tid / 16, tx = tid % 16;
    const int h = blockIdx.z;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const size_t xrow = (size_t)x_ld, orow = (size_t)H * os;
    const T* xh = x + (size_t)h * xs;
    const T* wh = w + (size_t)h * N * K;

    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        for (int e = tid; e < BM * BK; e += 256) {
            const int row = e / BK, kk = e % BK;
            const int gm = m0 + row;
            xs_s[kk][row] = (gm < M && k0 + kk < K) ? to_f32<T>(xh[(size_t)gm * xrow + k0 + kk]) : 0.f;
        }
        for (int e = tid; e < BN * BK; e += 256) {
            const int row = e / BK, kk = e % BK;
            const int gn = n0 + row;
            ws_s[kk][row] = (gn < N && k0 + kk < K) ? to_f32<T>(wh[(size_t)gn * K + k0 + kk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[4];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = xs_s[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws_s[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            float v = acc[i][j];
            if (gate) {
                const float g = to_f32<T>(gate[(size_t)gm * gs + gc + (gate_heads ? (size_t)h : (size_t)h * os + gn)]);
                v *= 1.f / (1.f + expf(-g));
            }
            out[(size_t)gm * orow + (size_t)h * os + gn] = from_f32<T>(v);
        }
    }
    if (rot > 0 && blockIdx.x == 0) {
        for (int e = tid; e < BM * rot; e += 256) {
            const int row = e / rot, i = e % rot;
            const int gm = m0 + row;
            if (gm >= M) continue;
            const int pos = positions[gm];
            const bool pos_ok = pos >= 0 && pos < table_len;
            if (!pos_ok) atomicOr(err, KVB_DEV_BAD_POS);
            const T* src = xh + (size_t)gm * xrow + K;
            float v = to_f32<T>(src[i]);
            if (i < 2 * rot_half && pos_ok) {
                const bool low = i < rot_half;
                const int t = low ? i : i - rot_half;
                const float vp = to_f32<T>(src[low ? i + rot_half : i - rot_half]);
                const float c = cos_t[(size_t)pos * rot_half + t], s = sin_t[(size_t)pos * rot_half + t];
                v = low ? (v * c - vp * s) : (v * c + vp * s);
            }
            out[(size_t)gm * orow + (size_t)h * os + N + i] = from_f32<T>(v);
        }
    }
}

// The same on the tensor cores (bfloat16; K, xs and the heads' offsets in steps of 8 elements, os even).
template <int MT>
__global__ void __launch_bounds__(mt::THREADS) head_linear_mma_kernel(const bf16* __restrict__ x, int xs, int x_ld, const bf16* __restrict__ w,
                                                                      bf16* __restrict__ out, int os, int M, int N, int K, int H,
                                                                      const bf16* __restrict__ gate, int gs, int gc, int gate_heads, int rot,
                                                                      int rot_half, const float* __restrict__ cos_t,
                                                                      const float* __restrict__ sin_t, int table_len,
                                                                      const int* __restrict__ positions, int* __restrict__ err) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int BM = 16 * MT;
    __shared__ __align__(16) mt::Smem<MT> sm;
    const int h = blockIdx.z, m0 = blockIdx.y * BM, n0 = blockIdx.x * mt::BN;
    const size_t xrow = (size_t)x_ld, orow = (size_t)H * os;
    const bf16* xh = x + (size_t)h * xs;
    auto a_row = [&](int r) -> const bf16* { return m0 + r < M ? xh + (size_t)(m0 + r) * xrow : nullptr; };
    auto store = [&](int r, int c, float v0, float v1) {
        const int gm = m0 + r, gn = n0 + c;
        if (gm >= M || gn >= N) return;
        bf16* dst = out + (size_t)gm * orow + (size_t)h * os + gn;
        if (gate && gate_heads) {
            const float s = 1.f / (1.f + expf(-__bfloat162float(gate[(size_t)gm * gs + gc + h])));
            v0 *= s;
            v1 *= s;
        } else if (gate) {
            const bf16* gp = gate + (size_t)gm * gs + gc + (size_t)h * os + gn;
            v0 *= 1.f / (1.f + expf(-__bfloat162float(gp[0])));
            if (gn + 1 < N) v1 *= 1.f / (1.f + expf(-__bfloat162float(gp[1])));
        }
        if (gn + 1 < N) *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(v0, v1);
        else dst[0] = __float2bfloat16_rn(v0);
    };
    mt::tile_product<MT>(sm, a_row, w + ((size_t)h * N + n0) * K, min(mt::BN, N - n0), K, store);
    if (rot > 0 && blockIdx.x == 0) {
        for (int e = threadIdx.x; e < BM * rot; e += mt::THREADS) {
            const int row = e / rot, i = e % rot;
            const int gm = m0 + row;
            if (gm >= M) continue;
            const int pos = positions[gm];
            const bool pos_ok = pos >= 0 && pos < table_len;
            if (!pos_ok) atomicOr(err, KVB_DEV_BAD_POS);
            const bf16* src = xh + (size_t)gm * xrow + K;
            float v = __bfloat162float(src[i]);
            if (i < 2 * rot_half && pos_ok) {
                const bool low = i < rot_half;
                const int t = low ? i : i - rot_half;
                const float vp = __bfloat162float(src[low ? i + rot_half : i - rot_half]);
                const float c = cos_t[(size_t)pos * rot_half + t], s = sin_t[(size_t)pos * rot_half + t];
                v = low ? (v * c - vp * s) : (v * c + vp * s);
            }
            out[(size_t)gm * orow + (size_t)h * os + N + i] = __float2bfloat16_rn(v);
        }
    }
}

// The same for more than 16 rows: tiles of BM x 128 outputs, 64 of K at a time in a ring of stages, the rotated columns made while
// the first are on their way, the gates asked for before the product, the result through shared memory to rows of 16 bytes.  K is
// walked in the same order as above: the same bits.  WM x WN warps.  Bound by the writes (prompts) and by the latency of W and x.
// Tiles of 64 x 64 with 32 of K in two stages, 4-byte stores and one of eight blocks on all of a tile's rotated columns took, for 16 heads
// of 128 -> 512 (+ 64 rotated) and 512 -> 128 with gates: 28 and 25 us at 32 rows (now 9 and 15), 43 and 29 at 200 (12 and 16), 72 and 43 at 2,048 (40 and 43).
namespace hl {
constexpr int BN = 128, BK = 64, STRIDE = BK + 8, OUT_STRIDE = BN + 8;
template <int BM, int STAGES> __host__ __device__ constexpr int smem_bytes() { return STAGES * (BM + BN) * STRIDE * 2; }     // the result fits in what the stages leave
}
template <int BM, int WM, int WN, int STAGES, bool CHANNEL_GATE>      // a gate for every number, or one a head (or none)
__global__ void __launch_bounds__(32 * WM * WN) head_linear_wide_kernel(const bf16* __restrict__ x, int xs, int x_ld, const bf16* __restrict__ w,
                                                                        bf16* __restrict__ out, int os, int M, int N, int K, int H,
                                                                        const bf16* __restrict__ gate, int gs, int gc, int rot,
                                                                        int rot_half, const float* __restrict__ cos_t,
                                                                        const float* __restrict__ sin_t, int table_len,
                                                                        const int* __restrict__ positions, int* __restrict__ err) {
    constexpr int BN = hl::BN, BK = hl::BK, STRIDE = hl::STRIDE, THREADS = 32 * WM * WN, CH = BK / 8;
    constexpr int MT = BM / WM / 16, NT = BN / WN / 8;
    static_assert(NT % 2 == 0 && BM * hl::OUT_STRIDE * 2 <= hl::smem_bytes<BM, STAGES>(), "");
    extern __shared__ __align__(16) unsigned char hl_smem[];
    bf16* as = reinterpret_cast<bf16*>(hl_smem);                   // [STAGES][BM][STRIDE]
    bf16* ws = as + STAGES * BM * STRIDE;                          // [STAGES][BN][STRIDE]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp / WN, wn = warp % WN;
    const int h = blockIdx.z, m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const bf16* xh = x + (size_t)h * xs;
    const bf16* wh = w + ((size_t)h * N + n0) * K;
    const int steps = (K + BK - 1) / BK, n_valid = min(BN, N - n0);
    auto load_w = [&](int step) {
        bf16* dst = ws + (step % STAGES) * BN * STRIDE;
        for (int e = tid; e < BN * CH; e += THREADS) {
            const int r = e / CH, c = (e % CH) * 8, k = step * BK + c;
            const bool valid = r < n_valid && k < K;
            mt::cp_async16(dst + r * STRIDE + c, valid ? wh + (size_t)r * K + k : w, valid);
        }
    };
    auto load_x = [&](int step) {
        bf16* dst = as + (step % STAGES) * BM * STRIDE;
        for (int e = tid; e < BM * CH; e += THREADS) {
            const int r = e / CH, c = (e % CH) * 8, k = step * BK + c;
            const bool valid = m0 + r < M && k < K;
            mt::cp_async16(dst + r * STRIDE + c, valid ? xh + (size_t)(m0 + r) * x_ld + k : w, valid);
        }
    };
    pdl_wait();                                                    // the launch before this one may have made x, W or the gates
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) {
            load_w(s);
            load_x(s);
        }
        mt::cp_async_commit();
    }
    // The rotated columns, while the first steps are on their way: the blocks of a row tile share its rows, a thread takes both
    // numbers of a pair (or one that is not rotated).
    if (rot > 0) {
        const int items = rot - rot_half, per = (BM + (int)gridDim.x - 1) / (int)gridDim.x, first = blockIdx.x * per;
        const int rows = min(min(per, BM - first), M - m0 - first);
        for (int e = tid; e < rows * items; e += THREADS) {
            const int row = e / items, i = e - row * items, gm = m0 + first + row;
            const int pos = positions[gm];
            const bool pos_ok = pos >= 0 && pos < table_len;
            if (!pos_ok) atomicOr(err, KVB_DEV_BAD_POS);
            const bf16* src = xh + (size_t)gm * x_ld + K;
            bf16* dst = out + (size_t)gm * H * os + (size_t)h * os + N;
            if (i < rot_half) {
                float v = __bfloat162float(src[i]), vp = __bfloat162float(src[i + rot_half]);
                if (pos_ok) {
                    const float c = cos_t[(size_t)pos * rot_half + i], s = sin_t[(size_t)pos * rot_half + i];
                    const float low = v * c - vp * s;
                    vp = vp * c + v * s;
                    v = low;
                }
                dst[i] = __float2bfloat16_rn(v);
                dst[i + rot_half] = __float2bfloat16_rn(vp);
            } else {
                dst[i + rot_half] = src[i + rot_half];
            }
        }
    }
    // The gates of this thread's results are asked for before the product.
    const int g = lane >> 2, t4 = lane & 3;
    float2 gates[MT][2][NT];
    if (CHANNEL_GATE) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int hi = 0; hi < 2; ++hi)
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const int gm = m0 + wm * MT * 16 + i * 16 + g + 8 * hi, gn = n0 + wn * NT * 8 + j * 8 + 2 * t4;
                    const bool there = gm < M && gn < N;           // N is even
                    const bf16* gp = gate + (there ? (size_t)gm * gs + gc + (size_t)h * os + gn : 0);
                    gates[i][hi][j] = there ? make_float2(__bfloat162float(gp[0]), __bfloat162float(gp[1])) : make_float2(0.f, 0.f);
                }
    }
    float acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
    for (int s = 0; s < steps; ++s) {
        mt::cp_async_wait<STAGES - 2>();
        __syncthreads();                                           // step s is there, and all are done with the stage refilled now
        if (s + STAGES - 1 < steps) {
            load_w(s + STAGES - 1);
            load_x(s + STAGES - 1);
        }
        mt::cp_async_commit();
        const bf16* at = as + (s % STAGES) * BM * STRIDE + (wm * MT * 16 + (lane & 15)) * STRIDE + (lane >> 4) * 8;
        const bf16* wt = ws + (s % STAGES) * BN * STRIDE + (wn * NT * 8 + (lane & 7) + (lane >> 4) * 8) * STRIDE + ((lane >> 3) & 1) * 8;
#pragma unroll
        for (int ks = 0; ks < BK / 16; ++ks) {
            uint32_t a[MT][4];
#pragma unroll
            for (int i = 0; i < MT; ++i) mt::ldmatrix_x4(a[i][0], a[i][1], a[i][2], a[i][3], at + i * 16 * STRIDE + ks * 16);
#pragma unroll
            for (int j = 0; j < NT; j += 2) {
                uint32_t b[4];
                mt::ldmatrix_x4(b[0], b[1], b[2], b[3], wt + j * 8 * STRIDE + ks * 16);
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    mt::mma_bf16(acc[i][j], a[i], b[0], b[1]);
                    mt::mma_bf16(acc[i][j + 1], a[i], b[2], b[3]);
                }
            }
        }
    }
    mt::cp_async_wait<0>();
    __syncthreads();                                               // the stages become the result's tile
    bf16* tile = as;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int hi = 0; hi < 2; ++hi) {
            const int r = wm * MT * 16 + i * 16 + g + 8 * hi, gm = m0 + r;
            float head_gate = 1.f;
            if (!CHANNEL_GATE && gate && gm < M) head_gate = 1.f / (1.f + expf(-__bfloat162float(gate[(size_t)gm * gs + gc + h])));
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const int c = wn * NT * 8 + j * 8 + 2 * t4;
                float v0 = acc[i][j][2 * hi], v1 = acc[i][j][2 * hi + 1];
                if (!CHANNEL_GATE) {
                    v0 *= head_gate;
                    v1 *= head_gate;
                } else {
                    v0 *= 1.f / (1.f + expf(-gates[i][hi][j].x));
                    v1 *= 1.f / (1.f + expf(-gates[i][hi][j].y));
                }
                *reinterpret_cast<__nv_bfloat162*>(tile + r * hl::OUT_STRIDE + c) = __floats2bfloat162_rn(v0, v1);
            }
        }
    __syncthreads();
    for (int e = tid; e < BM * (BN / 8); e += THREADS) {
        const int r = e / (BN / 8), c = (e % (BN / 8)) * 8;
        if (m0 + r < M && n0 + c < N)
            *reinterpret_cast<uint4*>(out + (size_t)(m0 + r) * H * os + (size_t)h * os + n0 + c) =
                *reinterpret_cast<const uint4*>(tile + r * hl::OUT_STRIDE + c);
    }
}

template <int BM, int WM, int WN, int STAGES>
static int launch_head_linear_wide(const bf16* x, int xs, int x_ld, const bf16* w, bf16* out, int os, int M, int N, int K, int H,
                                   const bf16* gate, int gs, int gc, int gate_heads, int rot, int rot_half, const float* cos_t,
                                   const float* sin_t, int table_len, const int* positions, int* err, cudaStream_t stream) {
    auto kernel = gate && !gate_heads ? head_linear_wide_kernel<BM, WM, WN, STAGES, true> : head_linear_wide_kernel<BM, WM, WN, STAGES, false>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, hl::smem_bytes<BM, STAGES>());
    if (e != cudaSuccess) return (int)e;
    kvb_launch(kernel, dim3((N + hl::BN - 1) / hl::BN, (M + BM - 1) / BM, H), dim3(32 * WM * WN), hl::smem_bytes<BM, STAGES>(), stream, x, xs, x_ld, w,
               out, os, M, N, K, H, gate, gs, gc, rot, rot_half, cos_t, sin_t, table_len, positions, err);
    return kvb_launch_status();
}

template <typename T, int BM>
static void launch_head_linear(const T* x, int xs, int x_ld, const T* w, T* out, int os, int M, int N, int K, int H, const T* gate, int gs,
                               int gc, int gate_heads, int rot, int rot_half, const float* cos_t, const float* sin_t, int table_len,
                               const int* positions, int* err, cudaStream_t stream) {
    dim3 grid((N + 63) / 64, (M + BM - 1) / BM, H);
    kvb_launch(head_linear_simt_kernel<T, BM>, grid, dim3(256), 0, stream, x, xs, x_ld, w, out, os, M, N, K, H, gate, gs, gc, gate_heads, rot, rot_half,
               cos_t, sin_t, table_len, positions, err);
}

KVB_API int kvb_head_linear(int dtype, const void* x, int xs, int x_ld, const void* w, void* out, int os, int M, int N, int K, int H,
                            const void* gate, int gs, int gc, int gate_heads, int rot, int rot_half, const float* cos_t, const float* sin_t,
                            int table_len, const int* positions, int* err, cudaStream_t stream) {
    if (M <= 0 || H <= 0) return KVB_OK;
    if (N < 1 || K < 1 || xs < K + rot || os < N + rot || 2 * rot_half > rot || x_ld < H * xs) return KVB_ERR_SHAPE;
    if ((M + 15) / 16 > 65535 || H > 65535) return KVB_ERR_LIMIT;
#define KVB_HEAD_LINEAR(T, BM)                                                                                             \
    launch_head_linear<T, BM>((const T*)x, xs, x_ld, (const T*)w, (T*)out, os, M, N, K, H, (const T*)gate, gs, gc, gate_heads, rot, rot_half, cos_t, \
                              sin_t, table_len, positions, err, stream)
    if (dtype == KVB_F32) {
        if (M <= 16) KVB_HEAD_LINEAR(float, 16); else KVB_HEAD_LINEAR(float, 64);
    } else if (dtype == KVB_BF16) {
        const bool aligned = K % 8 == 0 && xs % 8 == 0 && x_ld % 8 == 0 && os % 2 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0 &&
                             (uintptr_t)out % 4 == 0;
        if (aligned && getenv("KVB_HEAD_LINEAR_SIMT") == nullptr) {
            const bf16 *xb = (const bf16*)x, *wb = (const bf16*)w, *gb = (const bf16*)gate;
            // Rows of the result that start on 16 bytes; tiles of 32 rows with four stages while few of them fill the GPU, then of 64 rows with
            // two, so that more blocks share an SM (2,048 rows of 16 heads, 128 -> 512: 41 us, 82 with tiles of 32, 49 with 128).
            if (M > 16 && N % 8 == 0 && os % 8 == 0 && (uintptr_t)out % 16 == 0) {
                const long long small = (long long)((N + hl::BN - 1) / hl::BN) * ((M + 31) / 32) * H;
                return small <= 2 * kvb_sm_count()
                           ? launch_head_linear_wide<32, 1, 4, 4>(xb, xs, x_ld, wb, (bf16*)out, os, M, N, K, H, gb, gs, gc, gate_heads, rot,
                                                                  rot_half, cos_t, sin_t, table_len, positions, err, stream)
                           : launch_head_linear_wide<64, 2, 4, 2>(xb, xs, x_ld, wb, (bf16*)out, os, M, N, K, H, gb, gs, gc, gate_heads, rot,
                                                                  rot_half, cos_t, sin_t, table_len, positions, err, stream);
            }
            if (M <= 16)
                kvb_launch(head_linear_mma_kernel<1>, dim3((N + 63) / 64, (M + 15) / 16, H), dim3(mt::THREADS), 0, stream, xb, xs, x_ld, wb,
                           (bf16*)out, os, M, N, K, H, gb, gs, gc, gate_heads, rot, rot_half, cos_t, sin_t, table_len, positions, err);
            else
                kvb_launch(head_linear_mma_kernel<4>, dim3((N + 63) / 64, (M + 63) / 64, H), dim3(mt::THREADS), 0, stream, xb, xs, x_ld, wb,
                           (bf16*)out, os, M, N, K, H, gb, gs, gc, gate_heads, rot, rot_half, cos_t, sin_t, table_len, positions, err);
        } else if (M <= 16) {
            KVB_HEAD_LINEAR(bf16, 16);
        } else {
            KVB_HEAD_LINEAR(bf16, 64);
        }
    } else {
        return KVB_ERR_DTYPE;
    }
#undef KVB_HEAD_LINEAR
    return kvb_launch_status();
}
