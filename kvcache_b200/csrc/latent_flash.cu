// Attention over a cache of shared key rows (bfloat16, tensor cores): every head of a token scores the same row of
// Dk numbers per cached token, and the row's first Dv numbers are its value.  q [T, H * Dk], out [T, H * Dv].
//
// Because all heads read the same keys, the rows of a tile are (token, head) pairs: row m of a request's portion is
// token m / H, head m % H, and q and out are contiguous in m.  A decoded token with H heads fills a tile of 16 rows
// as well as 16 tokens of one head would; a key tile is read once for all heads.
//
// A block of 8 warps owns BM = 16 * MT rows and a run of keys [kb, ke) (a work item made on the host, see
// kernels/latent_plan.py).  Per tile of 64 keys, brought by cp.async into rows padded by 16 bytes:
//   scores   a warp takes one of the MT row tiles and an MT-th of the keys (mma.sync m16n8k16 over Dk), scaled to base 2,
//            masked (causal by the row's own position, window) and written to shared memory as float32 (with a warp on eight
//            keys of every row tile, Q was read from shared memory eight times a tile and bound it: 2,048 rows of 16 heads, keys
//            of 576, 448 -> 404 us; 1,024 rows behind 1,024 of 14 heads, keys of 288, 200 -> 177; tiles of 48 keys in two stages: the same);
//   softmax  float32: running maximum and sum per row, p = 2^(s - m) rounded to bfloat16 for the second product,
//            the sum taken from the unrounded p;
//   values   warp w owns output columns [8 NV w, 8 NV (w + 1)) for all row tiles: O = O * 2^(m_old - m_new) + P . V,
//            V read from the same shared rows as the keys (ldmatrix.trans).
// With `nsplit` > 1 the items of a tile leave (O, m, l) in scratch and `latent_flash_merge_kernel` adds them in the
// order of the splits; the split depends on the step's tiles, not on which block runs first.
// Two key stages where shared memory allows (the next tile is requested before this one is used), else one.
// `window` > 0: a row at position p sees keys p - window + 1 .. p; the work list starts a tile's keys at the 64-key tile
// that holds the first key its first row sees, and keys before that key are not fetched (a windowed cache entry may have
// given their pages back) but zero-filled and masked.  `sink` (one logit per head, or null): the softmax's denominator
// also holds exp(sink[h]); the rows of a tile's first split start from (m, l) = (sink, 1) instead of (-inf, 0).
#include "tc_common.cuh"

namespace lf {

constexpr int BN = 64;            // keys in a tile
constexpr int THREADS = 256;
constexpr float MASKED = -1e30f;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
    const int bytes = valid ? 16 : 0;   // 0 source bytes: the 16 destination bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(smem)), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;\n" ::); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t& r0, uint32_t& r1, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct Layout {
    int dk_pad, qs, rs, ss, ps;          // padded Dk; strides (elements) of the Q, key, score and P rows
    size_t q_off, k_off, s_off, p_off, st_off, total;
};

__host__ __device__ inline Layout make_layout(int MT, int NV, int Dk, int nstage) {
    Layout L;
    const int BM = 16 * MT;
    L.dk_pad = (Dk + 31) / 32 * 32;
    const int dv_pad = 64 * NV;
    L.qs = L.dk_pad + 8;
    L.rs = (L.dk_pad > dv_pad ? L.dk_pad : dv_pad) + 8;
    L.ss = BN + 8;
    L.ps = BN + 8;
    size_t at = 0;
    L.q_off = at;  at += (size_t)BM * L.qs * 2;
    L.k_off = at;  at += (size_t)nstage * BN * L.rs * 2;
    L.s_off = at;  at += (size_t)BM * L.ss * 4;
    L.p_off = at;  at += (size_t)BM * L.ps * 2;
    L.st_off = at; at += (size_t)BM * 4 * 4;          // m, l, corr, position of every row
    L.total = at;
    return L;
}

// Tiles of 64 rows with values of up to 256 numbers are held to 128 registers, so that two blocks share an SM and one's copies
// and softmax overlap the other's products.
template <int MT, int NV>
__global__ void __launch_bounds__(THREADS, (MT == 4 && NV <= 4) ? 2 : 1) latent_flash_kernel(
    const bf16* __restrict__ q, bf16* __restrict__ out, const bf16* __restrict__ k_pages, const int* __restrict__ block_table,
    int table_stride, const int* __restrict__ items, const int* __restrict__ seg_q_start, const int* __restrict__ seg_q_len,
    const int* __restrict__ seg_kv_len, float* __restrict__ part_o, float* __restrict__ part_ml, int H, int Dk, int Dv,
    int page_size, int window, float scale_log2, int nsplit, int nstage, const float* __restrict__ sink, int* __restrict__ err) {
    constexpr int BM = 16 * MT;
    constexpr int SN = 8 / MT, NT = BN / (8 * SN);          // scores: warps along the keys, and tiles of eight keys a warp
    extern __shared__ __align__(16) unsigned char smem[];
    const Layout L = make_layout(MT, NV, Dk, nstage);
    bf16* Qs = reinterpret_cast<bf16*>(smem + L.q_off);
    bf16* Ks = reinterpret_cast<bf16*>(smem + L.k_off);
    float* Ss = reinterpret_cast<float*>(smem + L.s_off);
    bf16* Ps = reinterpret_cast<bf16*>(smem + L.p_off);
    float* m_run = reinterpret_cast<float*>(smem + L.st_off);
    float* l_run = m_run + BM;
    float* corr = l_run + BM;
    int* rowpos = reinterpret_cast<int*>(corr + BM);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int* item = items + 4 * blockIdx.x;
    const int seg = item[0], m0 = item[1], kb = item[2], ke = item[3];
    const int q_len = seg_q_len[seg], kv_len = seg_kv_len[seg];
    const int start = kv_len - q_len;                       // tokens cached before this step
    const int M_total = q_len * H;
    const size_t row_base = (size_t)seg_q_start[seg] * H + m0;   // q and out are contiguous in (token, head)
    const int* table = block_table + (size_t)seg * table_stride;
    const int key_lo = window > 0 ? max(0, start + m0 / H - window + 1) : 0;     // the first key any row of the tile sees
    const bool first_split = blockIdx.x % nsplit == 0;
    pdl_wait();
    pdl_launch_dependents();

    // ---- the rows: positions, running state, Q into shared memory -----------------------------------------------
    for (int r = tid; r < BM; r += THREADS) {
        const int m = m0 + r;
        rowpos[r] = m < M_total ? start + m / H : -1;
        const bool from_sink = sink != nullptr && first_split && m < M_total;
        m_run[r] = from_sink ? sink[m % H] * 1.4426950408889634f : MASKED;
        l_run[r] = from_sink ? 1.f : 0.f;
    }
    const int q_chunks = L.dk_pad / 8;
    for (int e = tid; e < BM * q_chunks; e += THREADS) {
        const int r = e / q_chunks, c = e - r * q_chunks;
        const bool valid = m0 + r < M_total && c * 8 < Dk;
        cp_async16(Qs + (size_t)r * L.qs + c * 8, q + (row_base + (valid ? r : 0)) * Dk + (valid ? c * 8 : 0), valid);
    }
    cp_async_commit();

    const int row_chunks = (L.rs - 8) / 8;                  // chunks of a key row in shared memory, padding columns included
    auto load_keys = [&](int tile, int stage) {
        bf16* dst = Ks + (size_t)stage * BN * L.rs;
        const int r = tid >> 2;                             // four threads share a key row
        const int j = kb + tile * BN + r;
        const bool there = j < ke && j >= key_lo;
        size_t off = 0;
        if (there) {
            const int page = __ldg(table + j / page_size);
            if (page < 0) atomicOr(err, KVB_DEV_BAD_PAGE);
            off = ((size_t)(page < 0 ? 0 : page) * page_size + (j % page_size)) * Dk;
        }
        for (int c = tid & 3; c < row_chunks; c += 4) {
            const bool valid = there && c * 8 < Dk;
            cp_async16(dst + (size_t)r * L.rs + c * 8, k_pages + off + (valid ? c * 8 : 0), valid);
        }
        cp_async_commit();
    };

    float o[MT][NV][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nv = 0; nv < NV; ++nv) o[mt][nv][0] = o[mt][nv][1] = o[mt][nv][2] = o[mt][nv][3] = 0.f;

    const int ntiles = (ke - kb + BN - 1) / BN;
    if (ntiles > 0) load_keys(0, 0);
    const int KS2 = L.dk_pad / 32;
    for (int tile = 0; tile < ntiles; ++tile) {
        const int stage = nstage == 2 ? (tile & 1) : 0;
        const bool ahead = nstage == 2 && tile + 1 < ntiles;
        if (ahead) load_keys(tile + 1, stage ^ 1);
        if (ahead) cp_async_wait_one(); else cp_async_wait_all();
        __syncthreads();
        const bf16* Kt = Ks + (size_t)stage * BN * L.rs;
        const int key0 = kb + tile * BN;

        // ---- scores: a warp takes one row tile and NT tiles of eight keys, so that Q and the keys are read SN and MT times ----
        const int mt = warp / SN, key_first = (warp % SN) * 8 * NT;
        float s[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
        constexpr int AHEAD = MT == 4 ? 2 : 3;
#pragma unroll AHEAD
        for (int k2 = 0; k2 < KS2; ++k2) {
            uint32_t a[2][4];
#pragma unroll
            for (int half = 0; half < 2; ++half)
                ldmatrix_x4(a[half][0], a[half][1], a[half][2], a[half][3],
                            Qs + (size_t)(mt * 16 + (lane & 15)) * L.qs + k2 * 32 + half * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                uint32_t b[4];
                ldmatrix_x4(b[0], b[1], b[2], b[3], Kt + (size_t)(key_first + 8 * nt + (lane & 7)) * L.rs + k2 * 32 + (lane >> 3) * 8);
                mma_bf16(s[nt], a[0], b[0], b[1]);
                mma_bf16(s[nt], a[1], b[2], b[3]);
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
            for (int hi = 0; hi < 2; ++hi) {             // rows g and g + 8: two columns each, stored as one 8-byte word
                const int r = mt * 16 + g + hi * 8;
                const int c = key_first + 8 * nt + 2 * t4;
                const int pos = rowpos[r];
                float2 v;
                {
                    const int j = key0 + c;
                    const bool seen = j < ke && j <= pos && (window <= 0 || j > pos - window);
                    v.x = seen ? s[nt][2 * hi] * scale_log2 : MASKED;
                }
                {
                    const int j = key0 + c + 1;
                    const bool seen = j < ke && j <= pos && (window <= 0 || j > pos - window);
                    v.y = seen ? s[nt][2 * hi + 1] * scale_log2 : MASKED;
                }
                *reinterpret_cast<float2*>(Ss + r * L.ss + c) = v;
            }
        }
        __syncthreads();

        // ---- softmax of the tile: TPR threads share a row -------------------------------------------------------------
        {
            constexpr int TPR = THREADS / BM, CPT = BN / TPR;
            const int r = tid / TPR, c0 = (tid % TPR) * CPT;
            float v[CPT];
            float mx = MASKED;
#pragma unroll
            for (int i = 0; i < CPT; i += 4) {
                const float4 f = *reinterpret_cast<const float4*>(Ss + r * L.ss + c0 + i);
                v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
            }
#pragma unroll
            for (int i = 0; i < CPT; ++i) mx = fmaxf(mx, v[i]);
#pragma unroll
            for (int d = TPR / 2; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
            const float m_old = m_run[r];
            const float m_new = fmaxf(m_old, mx);
            float sum = 0.f;
            uint32_t packed[CPT / 2];
#pragma unroll
            for (int i = 0; i < CPT; i += 2) {
                const float p0 = v[i] > 0.5f * MASKED ? exp2f(v[i] - m_new) : 0.f;
                const float p1 = v[i + 1] > 0.5f * MASKED ? exp2f(v[i + 1] - m_new) : 0.f;
                sum += p0;
                sum += p1;
                __nv_bfloat162 pp = __floats2bfloat162_rn(p0, p1);
                packed[i / 2] = *reinterpret_cast<uint32_t*>(&pp);
            }
            if constexpr (CPT == 4) {
                *reinterpret_cast<uint2*>(Ps + r * L.ps + c0) = make_uint2(packed[0], packed[1]);
            } else {
#pragma unroll
                for (int i = 0; i < CPT / 8; ++i)
                    *reinterpret_cast<uint4*>(Ps + r * L.ps + c0 + 8 * i) = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
            }
#pragma unroll
            for (int d = TPR / 2; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            if (tid % TPR == 0) {
                const float cf = exp2f(m_old - m_new);
                corr[r] = cf;
                l_run[r] = l_run[r] * cf + sum;
                m_run[r] = m_new;
            }
        }
        __syncthreads();

        // ---- O = O * corr + P . V for this warp's columns --------------------------------------------------------------
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const float c0 = corr[mt * 16 + g], c1 = corr[mt * 16 + g + 8];
#pragma unroll
            for (int nv = 0; nv < NV; ++nv) {
                o[mt][nv][0] *= c0; o[mt][nv][1] *= c0; o[mt][nv][2] *= c1; o[mt][nv][3] *= c1;
            }
        }
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
            uint32_t b[NV][2];
            const int krow = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
            if constexpr (NV == 1) {
                ldmatrix_x2_trans(b[0][0], b[0][1], Kt + (size_t)krow * L.rs + warp * 8);
            } else {
#pragma unroll
                for (int n2 = 0; n2 < NV / 2; ++n2)
                    ldmatrix_x4_trans(b[2 * n2][0], b[2 * n2][1], b[2 * n2 + 1][0], b[2 * n2 + 1][1],
                                      Kt + (size_t)krow * L.rs + warp * 8 * NV + n2 * 16 + (lane >> 4) * 8);
            }
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                uint32_t a[4];
                ldmatrix_x4(a[0], a[1], a[2], a[3], Ps + (size_t)(mt * 16 + (lane & 15)) * L.ps + kk * 16 + (lane >> 4) * 8);
#pragma unroll
                for (int nv = 0; nv < NV; ++nv) mma_bf16(o[mt][nv], a, b[nv][0], b[nv][1]);
            }
        }
        __syncthreads();                    // the stage and P may be overwritten now
        if (nstage == 1 && tile + 1 < ntiles) load_keys(tile + 1, 0);
    }
    cp_async_wait_all();                    // Q's group, if there was no tile at all

    // ---- the rows' results ---------------------------------------------------------------------------------------------
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int hi = 0; hi < 2; ++hi) {
            const int r = mt * 16 + g + hi * 8;
            if (m0 + r >= M_total) continue;
            if (nsplit == 1) {
                const float l = l_run[r];
                const float inv = l > 0.f ? 1.f / l : 0.f;
                bf16* orow = out + (row_base + r) * Dv;
#pragma unroll
                for (int nv = 0; nv < NV; ++nv) {
                    const int d = warp * 8 * NV + nv * 8 + 2 * t4;
                    if (d + 1 < Dv) {
                        *reinterpret_cast<__nv_bfloat162*>(orow + d) = __floats2bfloat162_rn(o[mt][nv][2 * hi] * inv, o[mt][nv][2 * hi + 1] * inv);
                    } else if (d < Dv) {
                        orow[d] = __float2bfloat16_rn(o[mt][nv][2 * hi] * inv);
                    }
                }
            } else {
                float* prow = part_o + ((size_t)blockIdx.x * BM + r) * Dv;
#pragma unroll
                for (int nv = 0; nv < NV; ++nv) {
                    const int d = warp * 8 * NV + nv * 8 + 2 * t4;
                    if (d < Dv) prow[d] = o[mt][nv][2 * hi];
                    if (d + 1 < Dv) prow[d + 1] = o[mt][nv][2 * hi + 1];
                }
            }
        }
    }
    if (nsplit > 1)
        for (int r = tid; r < BM; r += THREADS) {
            part_ml[((size_t)blockIdx.x * BM + r) * 2] = m_run[r];
            part_ml[((size_t)blockIdx.x * BM + r) * 2 + 1] = l_run[r];
        }
}

// ---- tiles of 16 rows: decoded tokens ------------------------------------------------------------------------------------
// The same sums for one tile of rows, with what bounded it there taken out: the rows' Q is held in registers (every warp read it from
// shared memory for every tile of keys), a warp's scores run in four chains of products, they stay in registers (row maxima meet in
// shared memory, P alone is written), and keys come as one bulk copy a row, STAGES - 1 tiles ahead, their pages looked up a tile before.  Two
// barriers a tile instead of four.  KS: sixteens of Q a thread holds.
// What bounds it: the stream of keys, 3.4 TB/s of it (32 tokens of 16 heads with 4,096 keys of 576: 66 us with tiles of 16 rows of the kernel
// above, 44 here; a layer of 64 of them 173 -> 128 us, of 14 heads with keys of 288 93 -> 82, of one 31 -> 29).  With pages looked up
// where they are wanted, by one warp for all rows, it took 72: everything waited for that warp at the next barrier.
template <int NV, int KS, int STAGES, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS) latent_rows16_kernel(
    const bf16* __restrict__ q, bf16* __restrict__ out, const bf16* __restrict__ k_pages, const int* __restrict__ block_table,
    int table_stride, const int* __restrict__ items, const int* __restrict__ seg_q_start, const int* __restrict__ seg_q_len,
    const int* __restrict__ seg_kv_len, float* __restrict__ part_o, float* __restrict__ part_ml, int H, int Dk, int Dv, int rs,
    int page_size, int window, float scale_log2, int nsplit, const float* __restrict__ sink, int* __restrict__ err) {
    constexpr int BM = 16, WARPS = THREADS / 32;
    constexpr bool OWN_Q = KS <= 20;                        // Q has a place of its own, else it is read by way of the last stage
    constexpr int LEAD = OWN_Q ? STAGES : STAGES - 1;       // tiles asked for at once
    extern __shared__ __align__(128) unsigned char smem[];
    bf16* Ks = reinterpret_cast<bf16*>(smem);               // stage s at s * BN * rs; rows of rs numbers, 16 bytes beyond a multiple of 128
    __shared__ __align__(16) bf16 Ps[2][BM][BN + 8];
    __shared__ __align__(16) float tops[2][BM][WARPS];
    __shared__ __align__(8) uint64_t full[STAGES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int* item = items + 4 * blockIdx.x;
    const int seg = item[0], m0 = item[1], kb = item[2], ke = item[3];
    const int q_len = seg_q_len[seg], kv_len = seg_kv_len[seg], start = kv_len - q_len, M_total = q_len * H;
    const size_t row_base = (size_t)seg_q_start[seg] * H + m0;
    const int* table = block_table + (size_t)seg * table_stride;
    const int key_lo = window > 0 ? max(0, start + m0 / H - window + 1) : 0;
    const bool first_split = blockIdx.x % nsplit == 0;
    const int ntiles = (ke - kb + BN - 1) / BN, row_bytes = Dk * 2;
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) tc::mbar_init(&full[i], WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // Columns beyond Dk, up to what products read, are zeros for good.
    const int pad = (max(KS * 16, 64 * NV) - Dk) / 8;
    for (int i = tid; i < STAGES * BN * pad; i += THREADS)
        *reinterpret_cast<uint4*>(Ks + (size_t)(i / pad) * rs + Dk + i % pad * 8) = make_uint4(0, 0, 0, 0);
    __syncthreads();

    // Every warp brings in eight rows of a tile, its first lanes one each; rows that no query sees, or beyond the run, are zeros.  The
    // page a lane wants is looked up a tile before it is wanted: the way to it is what all would wait for at the next barrier.
    const int my_row = 8 * warp + (lane & 7);
    auto lookup = [&](int tile) -> int {
        const int j = kb + tile * BN + my_row;
        if (lane >= 8 || j >= ke || j < key_lo) return -1;
        const int page = table[j / page_size];
        if (page < 0) atomicOr(err, KVB_DEV_BAD_PAGE);
        return max(page, 0);
    };
    auto fetch = [&](int tile, int page) {
        bf16* dst = Ks + ((size_t)(tile % STAGES) * BN + my_row) * rs;
        uint64_t* bar = &full[tile % STAGES];
        const int there = __popc(__ballot_sync(0xffffffffu, page >= 0));
        if (lane < 8 && page < 0)
            for (int c = 0; c < Dk / 8; ++c) *reinterpret_cast<uint4*>(dst + c * 8) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");       // copies may come to the same place later
        __syncwarp();                                       // the zeros before the barrier's word
        if (lane == 0) tc::mbar_expect_tx(bar, there * row_bytes);
        __syncwarp();
        if (page >= 0)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                         ::"r"(smem_addr(dst)), "l"(k_pages + ((size_t)page * page_size + (kb + tile * BN + my_row) % page_size) * Dk), "r"(row_bytes),
                           "r"(smem_addr(bar)) : "memory");
    };
    // Keys of earlier steps are asked for while the kernel before is still running; its own are among a request's last.
    int asked = 0;
    for (; asked < LEAD && asked < ntiles && min(ke, kb + (asked + 1) * BN) <= start; ++asked) fetch(asked, lookup(asked));
    int page_next = lookup(asked);
    pdl_wait();
    pdl_launch_dependents();
    for (; asked < LEAD && asked < ntiles; ++asked) {
        fetch(asked, page_next);
        page_next = lookup(asked + 1);
    }

    // Rows g and g + 8 of Q, by way of shared memory (straight from memory, four bytes a load and all of it for every
    // warp, they cost a step of short histories 3 us).
    uint32_t a[KS][4];
    {
        bf16* Qs = Ks + (size_t)(OWN_Q ? STAGES : STAGES - 1) * BN * rs;
        for (int e = tid; e < BM * KS * 2; e += THREADS) {
            const int r = e / (KS * 2), c = e % (KS * 2) * 8;
            *reinterpret_cast<uint4*>(Qs + (size_t)r * rs + c) =
                m0 + r < M_total && c < Dk ? *reinterpret_cast<const uint4*>(q + (row_base + r) * Dk + c) : make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int k = 0; k < KS; ++k) ldmatrix_x4(a[k][0], a[k][1], a[k][2], a[k][3], Qs + (size_t)(lane & 15) * rs + k * 16 + (lane >> 4) * 8);
        if (!OWN_Q) __syncthreads();
        for (int e = tid; !OWN_Q && e < BM * pad; e += THREADS) *reinterpret_cast<uint4*>(Qs + (size_t)(e / pad) * rs + Dk + e % pad * 8) = make_uint4(0, 0, 0, 0);
    }
    float m[2], l[2];
    int pos[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = m0 + g + 8 * i;
        pos[i] = row < M_total ? start + row / H : -1;
        const bool from_sink = sink != nullptr && first_split && row < M_total;
        m[i] = from_sink ? sink[row % H] * 1.4426950408889634f : MASKED;
        l[i] = from_sink && warp == 0 && t4 == 0 ? 1.f : 0.f;
    }
    float o[NV][4];
#pragma unroll
    for (int nv = 0; nv < NV; ++nv) o[nv][0] = o[nv][1] = o[nv][2] = o[nv][3] = 0.f;

    for (int tile = 0; tile < ntiles; ++tile) {
        const int par = tile & 1;
        const bf16* Kt = Ks + (size_t)(tile % STAGES) * BN * rs;
        const bool ok = tc::mbar_wait(&full[tile % STAGES], (tile / STAGES) & 1);
        float s[4][4];
#pragma unroll
        for (int c = 0; c < 4; ++c) s[c][0] = s[c][1] = s[c][2] = s[c][3] = 0.f;
        const bf16* at = Kt + (size_t)(8 * warp + (lane & 7)) * rs + (lane >> 3) * 8;
#pragma unroll
        for (int k2 = 0; k2 < KS / 2; ++k2) {
            uint32_t b[4];
            ldmatrix_x4(b[0], b[1], b[2], b[3], at + k2 * 32);
            mma_bf16(s[(2 * k2) & 3], a[2 * k2], b[0], b[1]);
            mma_bf16(s[(2 * k2 + 1) & 3], a[2 * k2 + 1], b[2], b[3]);
        }
        float v[2][2], top[2];
        const int j0 = kb + tile * BN + 8 * warp + 2 * t4;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int j = j0 + e, x = 2 * i + e;
                const bool seen = j < ke && j <= pos[i] && (window <= 0 || j > pos[i] - window);
                v[i][e] = seen ? ((s[0][x] + s[1][x]) + (s[2][x] + s[3][x])) * scale_log2 : MASKED;
            }
            top[i] = fmaxf(v[i][0], v[i][1]);
            top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], 1));
            top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], 2));
            if (t4 == 0) tops[par][g + 8 * i][warp] = top[i];
        }
        // ... and all are done with the tile before: its stage may be filled.  If anyone's wait has run out nothing more is asked for, and the
        // copies that are still on their way are waited for, as long again.
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicOr(err, tc::KVB_DEV_TIMEOUT);
                for (int c = tile; c < ntiles && c < max(LEAD, tile + STAGES - 1); ++c) tc::mbar_wait(&full[c % STAGES], (c / STAGES) & 1);
            }
            __syncthreads();
            break;
        }
        const int next = tile + STAGES - 1;
        if (next >= LEAD && next < ntiles) {
            fetch(next, page_next);
            page_next = lookup(next + 1);
        }
        float corr[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float4* f = reinterpret_cast<const float4*>(tops[par][g + 8 * i]);
            const float4 x = f[0], y = f[1];
            const float m_new = fmaxf(m[i], fmaxf(fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)), fmaxf(fmaxf(y.x, y.y), fmaxf(y.z, y.w))));
            corr[i] = exp2f(m[i] - m_new);
            m[i] = m_new;
            const float p0 = v[i][0] > 0.5f * MASKED ? exp2f(v[i][0] - m_new) : 0.f, p1 = v[i][1] > 0.5f * MASKED ? exp2f(v[i][1] - m_new) : 0.f;
            l[i] = l[i] * corr[i] + (p0 + p1);
            *reinterpret_cast<__nv_bfloat162*>(&Ps[par][g + 8 * i][8 * warp + 2 * t4]) = __floats2bfloat162_rn(p0, p1);
        }
        __syncthreads();
#pragma unroll
        for (int nv = 0; nv < NV; ++nv) { o[nv][0] *= corr[0]; o[nv][1] *= corr[0]; o[nv][2] *= corr[1]; o[nv][3] *= corr[1]; }
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
            uint32_t p[4], b[NV][2];
            ldmatrix_x4(p[0], p[1], p[2], p[3], &Ps[par][lane & 15][kk * 16 + (lane >> 4) * 8]);
            const int krow = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
            if constexpr (NV == 1) {
                ldmatrix_x2_trans(b[0][0], b[0][1], Kt + (size_t)krow * rs + warp * 8);
            } else {
#pragma unroll
                for (int n2 = 0; n2 < NV / 2; ++n2)
                    ldmatrix_x4_trans(b[2 * n2][0], b[2 * n2][1], b[2 * n2 + 1][0], b[2 * n2 + 1][1],
                                      Kt + (size_t)krow * rs + warp * 8 * NV + n2 * 16 + (lane >> 4) * 8);
            }
#pragma unroll
            for (int nv = 0; nv < NV; ++nv) mma_bf16(o[nv], p, b[nv][0], b[nv][1]);
        }
    }
    // The rows' sums: over the four lanes of a row, then over the warps in their order.
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
        if (t4 == 0) tops[0][g + 8 * i][warp] = l[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = g + 8 * i;
        if (m0 + r >= M_total) continue;
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) sum += tops[0][r][w];
        const float inv = sum > 0.f ? 1.f / sum : 0.f;
        bf16* orow = out + (row_base + r) * Dv;
        float* prow = nsplit > 1 ? part_o + ((size_t)blockIdx.x * BM + r) * Dv : nullptr;
#pragma unroll
        for (int nv = 0; nv < NV; ++nv) {
            const int d = warp * 8 * NV + nv * 8 + 2 * t4;   // Dv is a multiple of four
            if (d >= Dv) continue;
            if (nsplit == 1) *reinterpret_cast<__nv_bfloat162*>(orow + d) = __floats2bfloat162_rn(o[nv][2 * i] * inv, o[nv][2 * i + 1] * inv);
            else *reinterpret_cast<float2*>(prow + d) = make_float2(o[nv][2 * i], o[nv][2 * i + 1]);
        }
        if (nsplit > 1 && warp == 0 && t4 == 0) {
            part_ml[((size_t)blockIdx.x * BM + r) * 2] = m[i];
            part_ml[((size_t)blockIdx.x * BM + r) * 2 + 1] = sum;
        }
    }
}

// out[row] = sum_s 2^(m_s - M) O_s[row] / sum_s 2^(m_s - M) l_s over the `nsplit` items of the row's tile.
// Grid (tiles, BM); the items of tile i are i * nsplit .. (i + 1) * nsplit - 1.  A block is MERGE_GROUPS x Dv / 4 threads:
// thread (g, c) adds four columns of the splits g, g + MERGE_GROUPS, ... (independent loads, all in flight at once), and the
// groups' sums are added in the order of the groups - a fixed order, whichever block runs first.  At least a warp of threads, which
// the splits' weights take, however few the columns are.
constexpr int MAX_SPLITS = 32, MERGE_GROUPS = 8;
__global__ void latent_flash_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                          const int* __restrict__ items, const int* __restrict__ seg_q_start,
                                          const int* __restrict__ seg_q_len, bf16* __restrict__ out, int H, int Dv, int BM,
                                          int nsplit) {
    __shared__ float weight[MAX_SPLITS];
    __shared__ float inv_s;
    extern __shared__ float4 sums[];                     // [MERGE_GROUPS][Dv / 4]
    const int first = blockIdx.x * nsplit, r = blockIdx.y;
    const int seg = items[4 * first], m0 = items[4 * first + 1];
    const int cols = Dv >> 2;
    const int g = threadIdx.x / cols, c = threadIdx.x - g * cols;
    pdl_wait();
    pdl_launch_dependents();
    if (m0 + r >= seg_q_len[seg] * H) return;
    const float4* base = reinterpret_cast<const float4*>(part_o + ((size_t)first * BM + r) * Dv) + c;
    const size_t step = (size_t)BM * cols;
    float4 v[MAX_SPLITS / MERGE_GROUPS];
#pragma unroll
    for (int i = 0; i < MAX_SPLITS / MERGE_GROUPS; ++i) {
        const int s = g + i * MERGE_GROUPS;
        v[i] = g < MERGE_GROUPS && s < nsplit ? base[(size_t)s * step] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (threadIdx.x < 32) {
        const int s = threadIdx.x;
        const float* ml = part_ml + ((size_t)(first + (s < nsplit ? s : 0)) * BM + r) * 2;
        const float m = s < nsplit ? ml[0] : MASKED, l = s < nsplit ? ml[1] : 0.f;
        const float M = warp_max(m);
        const float w = exp2f(m - M);
        weight[s] = w;
        float total = 0.f;                               // summed in the order of the splits
        for (int i = 0; i < nsplit; ++i) total += __shfl_sync(0xffffffffu, w * l, i);
        if (s == 0) inv_s = total > 0.f ? 1.f / total : 0.f;
    }
    __syncthreads();
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < MAX_SPLITS / MERGE_GROUPS; ++i) {
        const int s = g + i * MERGE_GROUPS;
        const float w = g < MERGE_GROUPS && s < nsplit ? weight[s] : 0.f;
        acc.x += w * v[i].x; acc.y += w * v[i].y; acc.z += w * v[i].z; acc.w += w * v[i].w;
    }
    if (g < MERGE_GROUPS) sums[g * cols + c] = acc;
    __syncthreads();
    if (g == 0) {
        float4 t = sums[c];
        for (int k = 1; k < MERGE_GROUPS; ++k) {
            const float4 u = sums[k * cols + c];
            t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
        }
        const float inv = inv_s;
        bf16* orow = out + ((size_t)seg_q_start[seg] * H + m0 + r) * Dv + 4 * c;
        *reinterpret_cast<__nv_bfloat162*>(orow) = __floats2bfloat162_rn(t.x * inv, t.y * inv);
        *reinterpret_cast<__nv_bfloat162*>(orow + 2) = __floats2bfloat162_rn(t.z * inv, t.w * inv);
    }
}

template <int MT, int NV>
static int launch(const bf16* q, bf16* out, const bf16* k_pages, const int* block_table, int table_stride, const int* items,
                  int n_items, const int* seg_q_start, const int* seg_q_len, const int* seg_kv_len, float* part_o, float* part_ml,
                  int H, int Dk, int Dv, int page_size, int window, float scale, int nsplit, const float* sink, int* err,
                  cudaStream_t stream) {
    int nstage = 2;
    Layout L = make_layout(MT, NV, Dk, nstage);
    // One stage where two stages would keep a second block off the SM (two blocks hide more than a second stage), or do not fit.
    const Layout one = make_layout(MT, NV, Dk, 1);
    const bool two_blocks = MT == 4 && NV <= 4;
    if (L.total > 220 * 1024 || (two_blocks && 2 * L.total > 220 * 1024 && 2 * one.total <= 220 * 1024)) {
        nstage = 1;
        L = one;
        if (L.total > 220 * 1024) return KVB_ERR_LIMIT;
    }
    static size_t configured = 0;                       // per instantiation
    if (L.total > configured) {
        if (cudaFuncSetAttribute(latent_flash_kernel<MT, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.total) != cudaSuccess)
            return (int)cudaGetLastError();
        configured = L.total;
    }
    kvb_launch(latent_flash_kernel<MT, NV>, dim3(n_items), dim3(THREADS), L.total, stream, q, out, k_pages, block_table, table_stride,
               items, seg_q_start, seg_q_len, seg_kv_len, part_o, part_ml, H, Dk, Dv, page_size, window,
               scale * 1.4426950408889634f, nsplit, nstage, sink, err);
    return kvb_launch_status();
}

// Whether an instance of the kernel for tiles of 16 rows takes these sizes: every row on 16 bytes, Q's sixteens in registers, and as many
// value columns as the instance of that key size has accumulators for.  Other sizes go to the kernel above, and so do those that it is
// ahead at, since an instance multiplies as many columns whatever the key size and the largest one fills an SM.  Layers of 16 heads in a graph, in us, the kernel
// above and this one, one token with 300 keys / 8 with 600 / 32 with 4,096: keys of 40 numbers (not taken) 20.3 and 21.1 / 22.6 and 24.6 / 41.7 and 44.9;
// 96 (not taken) 21.5 and 21.7 / 23.8 and 24.8 / 44.0 and 44.1; 112 22.4 and 22.1 / 24.6 and 24.8 / 47.9 and 45.0; 336 with values of 256 (not taken)
// 25.9 and 26.7 / 31.9 and 36.5 / 67.4 and 72.0; 336 with 272 26.1 and 27.3 / 29.3 and 31.8 / 87.9 and 71.8; 576 29.6 and 29.6 / 33.5 and 33.4 / 106 and 81.
static bool rows16_fits(int Dk, int Dv, const void* k_pages) {
    const int most = Dk <= 160 ? 128 : Dk <= 320 ? 256 : 512;
    const bool two_blocks_above = Dk > 320 && Dk <= 352 && Dv <= 256;       // two blocks an SM of the kernel above, one of the largest instance
    return Dk >= 104 && Dk <= 576 && Dv <= Dk && Dv <= most && !two_blocks_above && !((uintptr_t)k_pages & 15);
}

template <int NV, int KS, int STAGES, int BLOCKS>
static int launch_rows16(const bf16* q, bf16* out, const bf16* k_pages, const int* block_table, int table_stride, const int* items,
                         int n_items, const int* seg_q_start, const int* seg_q_len, const int* seg_kv_len, float* part_o, float* part_ml,
                         int H, int Dk, int Dv, int page_size, int window, float scale, int nsplit, const float* sink, int* err,
                         cudaStream_t stream) {
    constexpr int columns = KS * 16 > 64 * NV ? KS * 16 : 64 * NV;
    const int rs = (columns + 63) / 64 * 64 + 8;
    constexpr int bytes = (STAGES * BN + (KS <= 20 ? 16 : 0)) * ((columns + 63) / 64 * 64 + 8) * 2;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(latent_rows16_kernel<NV, KS, STAGES, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
            return (int)cudaGetLastError();
        configured = true;
    }
    kvb_launch(latent_rows16_kernel<NV, KS, STAGES, BLOCKS>, dim3(n_items), dim3(THREADS), (size_t)bytes, stream, q, out, k_pages, block_table,
               table_stride, items, seg_q_start, seg_q_len, seg_kv_len, part_o, part_ml, H, Dk, Dv, rs, page_size, window,
               scale * 1.4426950408889634f, nsplit, sink, err);
    return kvb_launch_status();
}

}  // namespace lf

// Whether the kernel takes these sizes (else the caller uses the generic kernel): 0 yes, negative no.
KVB_API int kvb_latent_flash_supports(int Dk, int Dv, int BM) {
    if (Dk % 8 != 0 || Dk < 8 || Dv < 4 || Dv % 4 != 0 || Dv > Dk || Dv > 512 || (BM != 16 && BM != 32 && BM != 64)) return KVB_ERR_SHAPE;
    const int NV = Dv <= 64 ? 1 : (Dv <= 128 ? 2 : (Dv <= 256 ? 4 : 8));
    return lf::make_layout(BM / 16, NV, Dk, 1).total <= 220 * 1024 ? KVB_OK : KVB_ERR_LIMIT;
}

// items: n_items x (segment, first row of the tile, first key, end of keys); the items of a tile are consecutive and
// every tile has `nsplit` of them.  part_o [n_items, BM, Dv] and part_ml [n_items, BM, 2] float32 are needed if nsplit > 1.
KVB_API int kvb_latent_flash(const void* q, void* out, const void* k_pages, const int* block_table, int table_stride,
                             const int* items, int n_items, int n_tiles, const int* seg_q_start, const int* seg_q_len,
                             const int* seg_kv_len, float* part_o, float* part_ml, int H, int Dk, int Dv, int BM, int page_size,
                             int window, float scale, int nsplit, const float* sink, int* err, cudaStream_t stream) {
    if (n_items <= 0) return KVB_OK;
    const int ok = kvb_latent_flash_supports(Dk, Dv, BM);
    if (ok != KVB_OK) return ok;
    if (nsplit < 1 || nsplit > lf::MAX_SPLITS || n_tiles * nsplit != n_items || (nsplit > 1 && (!part_o || !part_ml))) return KVB_ERR_SHAPE;
    const int NV = Dv <= 64 ? 1 : (Dv <= 128 ? 2 : (Dv <= 256 ? 4 : 8));
    int code = KVB_ERR_SHAPE;
#define KVB_LF(MT, NV_)                                                                                                      \
    code = lf::launch<MT, NV_>((const bf16*)q, (bf16*)out, (const bf16*)k_pages, block_table, table_stride, items, n_items,  \
                               seg_q_start, seg_q_len, seg_kv_len, part_o, part_ml, H, Dk, Dv, page_size, window, scale,    \
                               nsplit, sink, err, stream)
#define KVB_ROWS16(NV_, KS, STAGES, BLOCKS)                                                                                    \
    code = lf::launch_rows16<NV_, KS, STAGES, BLOCKS>((const bf16*)q, (bf16*)out, (const bf16*)k_pages, block_table, table_stride, items,  \
                                                      n_items, seg_q_start, seg_q_len, seg_kv_len, part_o, part_ml, H, Dk, Dv, page_size,  \
                                                      window, scale, nsplit, sink, err, stream)
    if (BM == 16 && lf::rows16_fits(Dk, Dv, k_pages)) {
        if (Dk <= 160) { if (NV == 1) KVB_ROWS16(1, 10, 2, 2); else KVB_ROWS16(2, 10, 2, 2); }
        else if (Dk <= 320) { if (NV == 1) KVB_ROWS16(1, 20, 2, 2); else if (NV == 2) KVB_ROWS16(2, 20, 2, 2); else KVB_ROWS16(4, 20, 2, 2); }
        else if (NV == 1) KVB_ROWS16(1, 36, 3, 1); else if (NV == 2) KVB_ROWS16(2, 36, 3, 1); else if (NV == 4) KVB_ROWS16(4, 36, 3, 1);
        else KVB_ROWS16(8, 36, 3, 1);
    } else if (BM == 16) {
        if (NV == 1) KVB_LF(1, 1); else if (NV == 2) KVB_LF(1, 2); else if (NV == 4) KVB_LF(1, 4); else KVB_LF(1, 8);
    } else if (BM == 32) {
        if (NV == 1) KVB_LF(2, 1); else if (NV == 2) KVB_LF(2, 2); else if (NV == 4) KVB_LF(2, 4); else KVB_LF(2, 8);
    } else {
        if (NV == 1) KVB_LF(4, 1); else if (NV == 2) KVB_LF(4, 2); else if (NV == 4) KVB_LF(4, 4); else KVB_LF(4, 8);
    }
#undef KVB_LF
#undef KVB_ROWS16
    if (code != KVB_OK || nsplit == 1) return code;
    kvb_launch(lf::latent_flash_merge_kernel, dim3(n_tiles, BM), dim3(lf::MERGE_GROUPS * (Dv / 4) < 32 ? 32 : lf::MERGE_GROUPS * (Dv / 4)), (size_t)lf::MERGE_GROUPS * Dv * 4, stream, (const float*)part_o, (const float*)part_ml,
               items, seg_q_start, seg_q_len, (bf16*)out, H, Dv, BM, nsplit);
    return kvb_launch_status();
}
