// Scans of mixers that carry a matrix S [D, Dv] per request and head from token to token, sixteen tokens at a time on the tensor
// cores: the form for portions of many tokens (single tokens and short portions: recurrent.cu).
//
//   CHUNK_GATED_DELTA     S~ = diag(a) S, S' = S~ + k (b (v - S~^T k))^T, o = S'^T q     (a: a decay per key channel, b: a number)
//   CHUNK_DELTA_RULE      S' = diag(a) S - c (u^T S) + k v^T, o = S'^T q                 (both terms read the old state)
//   CHUNK_CHANNEL_DECAY   S' = diag(a) S + k v^T, o = S'^T q
//   CHUNK_HEAD_DECAY      S' = a S + d k v^T, o = S'^T q                                 (a, d: numbers per head)
//
// Written out over a chunk of C = 16 tokens that starts from S_0, with L_t the product of the decays up to token t (per channel)
// and r(t, s) that of the decays after token s up to t, all of it is products of small matrices:
//
//   Z = W V + Y S_0               what the tokens read, or write: delta rules only, the solution of a triangular system
//   O = Q S_0 + A1 V + A2 Z       Q_t = L_t q_t; A_ts = sum_d q_t r(t, s) key_s, for s <= t
//   S_C = L_C S_0 + K1^T V + K2^T Z       K_s = r(C, s) key_s
//
// Launches (1), a block per (chunk, head) and all of them at once, make the matrices that do not know S_0 (the "record" of the
// chunk) on the CUDA cores: the decays between two tokens are multiplied up one after the other and never divided by, so that
// any decay down to zero is exact.  Launch (2) walks a segment's chunks in order, a block per 16 value channels of a head:
// S^T lives in the accumulators of its warps, each with 8 KT key channels, and is at the same time the A operand of Y S_0 and
// Q S_0 - the two fragments of `mma.sync` hold the same numbers if neighbouring channels are taken as the halves of a step of
// eight.  The warps' partial sums meet once a chunk through shared memory, added in one order by all of them.  A record lies in
// scratch as it will lie in shared memory and comes in by one bulk copy, a chunk ahead.
//
// A number x is split into h = tf32(x) and l = x - h, and a product is h h + h l + l h (what is left out is 2^-22 of it); sums that
// run on from step to step are added on the CUDA cores, because the tensor cores' own accumulation truncates.  Against 64 bits a
// scan alone is off by 1.3e-7 to 1.6e-7 of its results and 1.1e-7 to 1.6e-7 of its state, the scans over tokens by 1.0e-7 and 0.6e-7;
// a layer's state, whose inputs come from products with float32 sums of their own, by 7e-6 to 3e-5 either way.
//
// What bounds it: the chain of a chunk - its products, one exchange, one wait: 0.8 us with 64 key channels, 1.2 to 1.4 with 128 -
// times the chunks of the longest segment; the tensor pipe is idle for most of it.  Measured beside the form each replaces (us;
// records and walk): gated delta 777 x 14 x 64 x 64: 117 -> 64, 1,500 x 16 x 128 x 128: 326 -> 154; delta rule 543 + 905 + 363 x 16 x
// 128: 662 -> 179 (records 45, systems 11, walk 123), 1,000 x 14 x 64: 199 -> 90; channel decays 600 + 400 x 8 x 128 x 256: 154 -> 56; head decays 2,048 x 64 x
// 128 x 64: 279 -> 189.
// A segment's result does not depend on what else the step holds.  An infinite or undefined value spreads within its chunk of
// sixteen tokens, in its own value channel, also to tokens before it.
// State layout: [slot, head, key channel, value channel].
#include "common.cuh"
#include "tc_common.cuh"

namespace sc {

enum { CHUNK_GATED_DELTA = 0, CHUNK_DELTA_RULE = 1, CHUNK_CHANNEL_DECAY = 2, CHUNK_HEAD_DECAY = 3 };
constexpr int C = 16;

__host__ __device__ constexpr bool has_z(int mode) { return mode <= CHUNK_DELTA_RULE; }
__host__ __device__ constexpr bool has_v(int mode) { return mode != CHUNK_GATED_DELTA; }      // V enters O and S_C by itself
__host__ __device__ constexpr int padded(int D) { return (D + 63) / 64 * 64; }

// The record of a (chunk, head), in floats, as it lies in scratch and, copied as it is, in shared memory: rows [Y | Q] of DP + 8
// floats, rows [K1 | K2] of DP + 4, the chunk's decay, 16 x 16 matrices [W | A1 | A2] in rows of 24; the parts a mode does not
// have are not there.  The strides are those whose reads as operands meet no bank twice.  Head decay: [Q | K1] once for all heads
// that share them, then per head [L_t | d r(C, t) | L_C, 15 unused | A1].
struct Record { int y, q, k1, k2, decay, w, a1, a2, total, shared; };     // `shared`: the floats that heads share (at the start)
__host__ __device__ constexpr Record record_of(int mode, int DP) {
    Record r = {};
    int at = 0;
    r.y = at;  at += has_z(mode) ? C * (DP + 8) : 0;
    r.q = at;  at += C * (DP + 8);
    r.k1 = at; at += has_v(mode) ? C * (DP + 4) : 0;
    r.k2 = at; at += has_z(mode) ? C * (DP + 4) : 0;
    r.shared = mode == CHUNK_HEAD_DECAY ? at : 0;
    r.decay = at; at += mode == CHUNK_HEAD_DECAY ? 3 * C : DP;
    r.w = at;  at += has_z(mode) ? C * 24 : 0;
    r.a1 = at; at += has_v(mode) ? C * 24 : 0;
    r.a2 = at; at += has_z(mode) ? C * 24 : 0;
    r.total = at;
    return r;
}

// Where a step's rows lie (float32).  q, k, v: columns of `rows` [T, stride]; a head reads number h / qk_div of q and k.
struct Rows {
    const float* rows;
    const float* gates;          // gated delta: [a: H D | b: H]; delta rule: [a: H D | u: H D | c: H D]; channel decay: [a: H D];
                                 // head decay: [a: H | d: H]
    int stride, gate_stride, q_col, k_col, v_col, qk_div;
};
struct Segments {
    const int* q_start;
    const int* q_len;
    const int* slot;
    int count;
};

// Which rows the step's chunk `id` covers; false beyond the last.
__device__ __forceinline__ bool find_chunk(int id, const Segments& seg, int& r0, int& count) {
    for (int s = 0; s < seg.count; ++s) {
        const int n = seg.q_len[s], mine = (n + C - 1) / C;
        if (id < mine) {
            r0 = seg.q_start[s] + id * C;
            count = min(C, n - id * C);
            return true;
        }
        id -= mine;
    }
    return false;
}

// v[i]: this lane's share of 16 sums over 16 neighbouring lanes; lane `part` returns the sum of number `part`.
__device__ __forceinline__ float sum16(float (&v)[16], int part) {
#pragma unroll
    for (int offset = 8; offset >= 1; offset >>= 1) {
        const bool upper = part & offset;
#pragma unroll
        for (int i = 0; i < offset; ++i) {
            const float mine = upper ? v[i + offset] : v[i], other = upper ? v[i] : v[i + offset];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, other, offset);
        }
    }
    return v[0];
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float c) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c))));
}
__device__ __forceinline__ void scale4(float4& a, const float4& b) { a.x *= b.x; a.y *= b.y; a.z *= b.z; a.w *= b.w; }

// ---- launches (1): the records ---------------------------------------------------------------------------------------------
// grid (chunks, heads), 256 threads.  Thread (s, part): token s as a key, channels 4 part .. + 3 of every 64.
template <int MODE, int NI>          // NI: 64-channel groups of a row
__global__ void __launch_bounds__(256, MODE == CHUNK_DELTA_RULE && NI == 2 ? 3 : 4) chunk_records_kernel(const Rows in, const Segments seg,
                                                                                                       float* __restrict__ records, int H,
                                                                                                       int D, int wide) {
    constexpr int DP = 64 * NI, PARTS = MODE == CHUNK_DELTA_RULE ? 5 : 3;
    __shared__ __align__(16) float rows_s[PARTS][C][DP];       // q, k, a (, u, c)
    __shared__ float low_s[C][C + 1], mat_s[C][C + 1], b_s[C];
    const int tid = threadIdx.x, s = tid >> 4, part = tid & 15, h = blockIdx.y;
    pdl_wait();
    pdl_launch_dependents();
    int r0, count;
    if (!find_chunk(blockIdx.x, seg, r0, count)) return;
    constexpr Record R = record_of(MODE, DP);
    float* rec = records + ((size_t)blockIdx.x * H + h) * R.total;

    // Tokens beyond the segment's end change nothing: a = 1, everything else 0.  So do channels beyond D.
    {
        const bool row_there = s < count;
        const float* row = in.rows + (size_t)(r0 + (row_there ? s : 0)) * in.stride + h / in.qk_div * D;
        const float* gate = in.gates + (size_t)(r0 + (row_there ? s : 0)) * in.gate_stride + (size_t)h * D;
        const float* from[5] = {row + in.q_col, row + in.k_col, gate, gate + (size_t)H * D, gate + (size_t)2 * H * D};
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int d = 64 * i + 4 * part;
#pragma unroll
            for (int x = 0; x < PARTS; ++x) {
                const float none = x == 2 ? 1.f : 0.f;
                float4 v = make_float4(none, none, none, none);
                if (row_there) {
                    if (wide) {                                    // rows start on 16 bytes and D is a multiple of 4
                        if (d < D) v = *(const float4*)(from[x] + d);
                    } else {
                        if (d < D) v.x = from[x][d];
                        if (d + 1 < D) v.y = from[x][d + 1];
                        if (d + 2 < D) v.z = from[x][d + 2];
                        if (d + 3 < D) v.w = from[x][d + 3];
                    }
                }
                *(float4*)&rows_s[x][s][d] = v;
            }
        }
    }
    if (MODE == CHUNK_GATED_DELTA && tid < C) b_s[tid] = tid < count ? in.gates[(size_t)(r0 + tid) * in.gate_stride + (size_t)H * D + h] : 0.f;
    __syncthreads();

    auto at = [&](int which, int t, int i) { return *(const float4*)&rows_s[which][t][64 * i + 4 * part]; };
    {
        // Sums over the channels between token s and every later one, the key decayed on the way.
        float4 key[NI], rem[NI];
        float qs[C], us[C], qc[C], uc[C];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            key[i] = at(1, s, i);
            if (MODE == CHUNK_DELTA_RULE) rem[i] = at(4, s, i);
        }
#pragma unroll
        for (int t = 0; t < C; ++t) {
            qs[t] = us[t] = qc[t] = uc[t] = 0.f;
            if (t >= s) {
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    const float4 q = at(0, t, i);
                    if (t > s) {
                        const float4 a = at(2, t, i);
                        if (MODE == CHUNK_DELTA_RULE) {            // reads the state before the token's own decay
                            const float4 u = at(3, t, i);
                            us[t] = dot4(u, key[i], us[t]);
                            uc[t] = dot4(u, rem[i], uc[t]);
                            scale4(rem[i], a);
                        }
                        scale4(key[i], a);
                        if (MODE == CHUNK_GATED_DELTA) us[t] = dot4(at(1, t, i), key[i], us[t]);
                    }
                    qs[t] = dot4(q, key[i], qs[t]);
                    if (MODE == CHUNK_DELTA_RULE) qc[t] = dot4(q, rem[i], qc[t]);
                }
            }
        }
        // Token `part` reads key s (zero before it).
        rec[(MODE == CHUNK_GATED_DELTA ? R.a2 : R.a1) + part * 24 + s] = sum16(qs, part);
        if (MODE == CHUNK_GATED_DELTA) low_s[part][s] = sum16(us, part);
        if (MODE == CHUNK_DELTA_RULE) {                            // for the next launch: u . c below the diagonal, u . k mirrored above
            rec[R.a2 + part * 24 + s] = -sum16(qc, part);
            const float uk = sum16(us, part), ur = sum16(uc, part);
            if (part > s) {
                rec[R.w + part * 24 + s] = ur;
                rec[R.w + s * 24 + part] = uk;
            }
        }
    }
    if (MODE == CHUNK_GATED_DELTA) {
        __syncthreads();
        if (tid < C) {                                             // the triangular system, a thread per column
            float x[C];
#pragma unroll
            for (int t = 0; t < C; ++t) {
                float v = t == tid ? 1.f : 0.f;
#pragma unroll
                for (int j = 0; j < C; ++j)
                    if (j < t) v = fmaf(-low_s[t][j], x[j], v);
                x[t] = b_s[t] * v;
                mat_s[t][tid] = x[t];
            }
        }
    }
    // Rows decayed from the chunk's start (the lower threads) and to its end (the upper), a thread per channel.
    if (MODE != CHUNK_GATED_DELTA) __syncthreads();                // all have read q
    const int d = tid % DP;
    if (tid < DP) {
        float run = 1.f;
#pragma unroll
        for (int t = 0; t < C; ++t) {
            const float before = run;
            run *= rows_s[2][t][d];
            rec[R.q + t * (DP + 8) + d] = rows_s[0][t][d] * run;
            if (MODE == CHUNK_GATED_DELTA) rows_s[0][t][d] = rows_s[1][t][d] * run;                    // the key as it meets S_0
            if (MODE == CHUNK_DELTA_RULE) rec[R.y + t * (DP + 8) + d] = rows_s[3][t][d] * before;
        }
        rec[R.decay + d] = run;
    } else if (tid < 2 * DP) {
        float run = 1.f;
#pragma unroll
        for (int t = C - 1; t >= 0; --t) {
            rec[(has_v(MODE) ? R.k1 : R.k2) + t * (DP + 4) + d] = rows_s[1][t][d] * run;
            if (MODE == CHUNK_DELTA_RULE) rec[R.k2 + t * (DP + 4) + d] = -rows_s[4][t][d] * run;
            run *= rows_s[2][t][d];
        }
    }
    if (MODE != CHUNK_GATED_DELTA) return;
    __syncthreads();
    // Y = -W . (the keys that meet S_0): thread (t = s, part).
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < C; ++j) {
            if (j <= s) {
                const float m = -mat_s[s][j];
                const float4 v = at(0, j, i);
                sum.x = fmaf(m, v.x, sum.x); sum.y = fmaf(m, v.y, sum.y); sum.z = fmaf(m, v.z, sum.z); sum.w = fmaf(m, v.w, sum.w);
            }
        }
        *(float4*)(rec + R.y + s * (DP + 8) + 64 * i + 4 * part) = sum;
    }
    rec[R.w + s * 24 + part] = part <= s ? mat_s[s][part] : 0.f;
}

// Delta rule: T = (1 + u . c)^-1, Y = T . (the reads that meet S_0, where Y will lie), W = T (u . k).  grid (chunks, heads), a thread
// per channel.  By itself, because half a block would wait for the system's sixteen threads in the launch before it.
template <int NI>
__global__ void __launch_bounds__(64 * NI) chunk_solve_kernel(const Segments seg, float* __restrict__ records, int H) {
    constexpr int DP = 64 * NI;
    constexpr Record R = record_of(CHUNK_DELTA_RULE, DP);
    __shared__ float low_s[C][C + 1], mat_s[C][C + 1];
    const int d = threadIdx.x;
    pdl_wait();
    pdl_launch_dependents();
    int r0, count;
    if (!find_chunk(blockIdx.x, seg, r0, count)) return;
    float* rec = records + ((size_t)blockIdx.x * H + blockIdx.y) * R.total;
    for (int i = d; i < C * C; i += DP) low_s[i / C][i % C] = i / C == i % C ? 0.f : rec[R.w + i / C * 24 + i % C];
    float x[C];
#pragma unroll
    for (int t = 0; t < C; ++t) x[t] = rec[R.y + t * (DP + 8) + d];
    __syncthreads();
    if (d < C) {
        float v[C];
#pragma unroll
        for (int t = 0; t < C; ++t) {
            v[t] = t == d ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < C; ++j)
                if (j < t) v[t] = fmaf(-low_s[t][j], v[j], v[t]);
            mat_s[t][d] = v[t];
        }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < C; ++t) {
        float y = 0.f;
#pragma unroll
        for (int j = 0; j < C; ++j)
            if (j <= t) y = fmaf(mat_s[t][j], x[j], y);
        rec[R.y + t * (DP + 8) + d] = y;
    }
    for (int i = d; i < C * C; i += DP) {
        const int t = i / C, s = i % C;
        float w = 0.f;
        for (int j = s + 1; j <= t; ++j) w = fmaf(mat_s[t][j], low_s[s][j], w);       // u . k of (j, s) lies at (s, j)
        rec[R.w + t * 24 + s] = w;
    }
}

// Head decay: grid (chunks, groups of heads with one q and k).
template <int NI>
__global__ void __launch_bounds__(256) head_records_kernel(const Rows in, const Segments seg, float* __restrict__ records, int H, int D) {
    constexpr int DP = 64 * NI, HEADS = 16;
    __shared__ __align__(16) float q_s[C][DP], k_s[C][DP];
    __shared__ float qk_s[C][C + 1], a_s[HEADS][C], d_s[HEADS][C];
    const int tid = threadIdx.x, s = tid >> 4, part = tid & 15, g = blockIdx.y;
    pdl_wait();
    pdl_launch_dependents();
    int r0, count;
    if (!find_chunk(blockIdx.x, seg, r0, count)) return;
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = 64 * i + 4 * part + e;
            const bool there = s < count && d < D;
            const float* row = in.rows + (size_t)(r0 + (there ? s : 0)) * in.stride + (size_t)g * D + (there ? d : 0);
            q_s[s][d] = there ? row[in.q_col] : 0.f;
            k_s[s][d] = there ? row[in.k_col] : 0.f;
        }
    __syncthreads();
    float sums[C];
#pragma unroll
    for (int t = 0; t < C; ++t) {
        sums[t] = 0.f;
#pragma unroll
        for (int i = 0; i < NI; ++i)
            sums[t] = dot4(*(const float4*)&q_s[t][64 * i + 4 * part], *(const float4*)&k_s[s][64 * i + 4 * part], sums[t]);
    }
    qk_s[part][s] = sum16(sums, part);
    constexpr Record R = record_of(CHUNK_HEAD_DECAY, DP);
    const int groups = H / in.qk_div, first = g * in.qk_div, last = first + in.qk_div;
    {
        float* rec = records + ((size_t)blockIdx.x * groups + g) * R.shared;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int d = 64 * i + 4 * part;
            *(float4*)(rec + R.q + s * (DP + 8) + d) = *(const float4*)&q_s[s][d];
            *(float4*)(rec + R.k1 + s * (DP + 4) + d) = *(const float4*)&k_s[s][d];
        }
        records += (size_t)gridDim.x * groups * R.shared;
    }
    for (int h0 = first; h0 < last; h0 += HEADS) {
        __syncthreads();
        {                                                          // head h0 + part, token s
            const bool there = h0 + part < last && s < count;
            const float* gate = in.gates + (size_t)(r0 + (there ? s : 0)) * in.gate_stride + (there ? h0 + part : 0);
            a_s[part][s] = there ? gate[0] : 1.f;
            d_s[part][s] = there ? gate[H] : 0.f;
        }
        __syncthreads();
        // Thread (head h0 + s, token `part` as a key).
        const int h = h0 + s;
        if (h < last) {
            float* rec = records + ((size_t)blockIdx.x * H + h) * (R.total - R.shared);
            const float gain = d_s[s][part];
            float run = 1.f, all = 1.f;
#pragma unroll
            for (int t = 0; t < C; ++t) {
                const float a = a_s[s][t];
                if (t > part) run *= a;
                all *= t <= part ? a : 1.f;
                rec[R.a1 - R.shared + t * 24 + part] = t >= part ? qk_s[t][part] * (gain * run) : 0.f;
            }
            rec[part] = all;                                       // L_t, t = part
            rec[C + part] = gain * run;
            if (part == C - 1) rec[2 * C] = all;                   // L_C
        }
    }
}

// ---- launch (2): the walk -------------------------------------------------------------------------------------------------
struct Split { uint32_t h[4], l[4]; };
__device__ __forceinline__ void split1(float x, uint32_t& h, uint32_t& l) {
    h = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;         // ten bits of fraction, rounded to the nearest
    l = __float_as_uint(x - __uint_as_float(h));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// An accumulator fragment (columns 2 t, 2 t + 1) as the A operand of a step of eight along those columns.
__device__ __forceinline__ Split as_operand(const float (&c)[4]) {
    Split s;
    split1(c[0], s.h[0], s.l[0]);
    split1(c[2], s.h[1], s.l[1]);
    split1(c[1], s.h[2], s.l[2]);
    split1(c[3], s.h[3], s.l[3]);
    return s;
}
// p[i] = a(i) b[i], N of them side by side: a product waits about 70 clocks for the one before it on the same accumulator, so that
// one after the other they would bound the walk.  The cross products come first: the large one is rounded last.
template <int N, typename A>
__device__ __forceinline__ void products(float (&p)[N][4], A a, const float (&b)[N][2]) {
    uint32_t h[N][2], l[N][2];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        split1(b[i][0], h[i][0], l[i][0]);
        split1(b[i][1], h[i][1], l[i][1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) p[i][e] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) mma_tf32(p[i], a(i).h, l[i][0], l[i][1]);
#pragma unroll
    for (int i = 0; i < N; ++i) mma_tf32(p[i], a(i).l, h[i][0], h[i][1]);
#pragma unroll
    for (int i = 0; i < N; ++i) mma_tf32(p[i], a(i).h, h[i][0], h[i][1]);
}
__device__ __forceinline__ void pair(float (&b)[2], const float* at) {
    const float2 v = *(const float2*)at;
    b[0] = v.x;
    b[1] = v.y;
}
__device__ __forceinline__ void add4(float (&sum)[4], const float (&p)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[e] += p[e];
}

__device__ __forceinline__ void copy_bulk(float* smem, const float* gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(tc::smem_u32(smem)), "l"(gmem), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
}

// grid (16 value channels, heads, segments), WD warps of 8 KT key channels.
template <int MODE, int NI, int KT, int STAGES>
__global__ void __launch_bounds__(64 * NI / (8 * KT) * 32) chunk_walk_kernel(const Rows in, const Segments seg, const float* __restrict__ records,
                                                                             int max_chunks, float q_scale, float* __restrict__ memory,
                                                                             float* __restrict__ out, int H, int D, int Dv, int* __restrict__ err) {
    constexpr bool Z = has_z(MODE), V = has_v(MODE);
    constexpr int DP = 64 * NI, WD = DP / (8 * KT);
    constexpr int NX = Z ? 4 : 2;                              // accumulator fragments a warp hands over: Q S_0 (, Y S_0)
    constexpr Record R = record_of(MODE, DP);
    static_assert(WD >= 2, "the first two warps write the results of eight tokens each");
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(16) float4 meet[2][WD][NX][32];
    __shared__ __align__(8) uint64_t full[STAGES];
    const int tid = threadIdx.x, lane = tid & 31, wd = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int h = blockIdx.y, sg = blockIdx.z;
    const int n = seg.q_len[sg], r0 = seg.q_start[sg], slot = seg.slot[sg];
    if (n <= 0) return;
    int chunk0 = 0;
    for (int i = 0; i < sg; ++i) chunk0 += (seg.q_len[i] + C - 1) / C;
    const int chunks = (n + C - 1) / C, ch0 = 8 * KT * wd;

    float* mem = memory + ((size_t)slot * H + h) * D * Dv;
    const int col = 16 * blockIdx.x + g;
    const bool col0 = col < Dv, col1 = col + 8 < Dv;
    float S[KT][4];                                            // S^T: rows are value channels col, col + 8; columns key channels
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = ch0 + 8 * kt + 2 * t4 + (e & 1);
            S[kt][e] = d < D && (e < 2 ? col0 : col1) ? mem[(size_t)d * Dv + col + 8 * (e >> 1)] : 0.f;
        }
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) tc::mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    pdl_launch_dependents();

    const int groups = H / in.qk_div;
    auto fetch = [&](int ci) {                                 // one thread: the chunk's record, as it lies
        float* b = sm + (ci % STAGES) * R.total;
        uint64_t* bar = &full[ci % STAGES];
        const size_t id = chunk0 + ci;
        tc::mbar_expect_tx(bar, R.total * 4);
        if (R.shared) {
            copy_bulk(b, records + (id * groups + h / in.qk_div) * R.shared, R.shared * 4, bar);
            copy_bulk(b + R.shared, records + (size_t)max_chunks * groups * R.shared + (id * H + h) * (R.total - R.shared), (R.total - R.shared) * 4, bar);
        } else {
            copy_bulk(b, records + (id * H + h) * R.total, R.total * 4, bar);
        }
    };
    // V^T as an operand: steps of eight tokens, tokens 2 t and 2 t + 1 its halves.
    const float* v_at = in.rows + (size_t)(r0 + 2 * t4) * in.stride + in.v_col + (size_t)h * Dv + col;     // of the chunk asked for next
    const size_t v_chunk = (size_t)C * in.stride;
    auto values = [&](int left, float (&raw)[2][4]) {          // `left`: tokens from the chunk's first on
        if (left >= C && 16 * (int)blockIdx.x + C <= Dv) {
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const float* at = v_at + (size_t)(8 * ks) * in.stride;
                raw[ks][0] = at[0]; raw[ks][2] = at[8];
                at += in.stride;
                raw[ks][1] = at[0]; raw[ks][3] = at[8];
            }
        } else {
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = 8 * ks + (e & 1);
                    raw[ks][e] = 2 * t4 + t < left && (e < 2 ? col0 : col1) ? v_at[(size_t)t * in.stride + 8 * (e >> 1)] : 0.f;
                }
        }
        v_at += v_chunk;
    };
    __syncthreads();
    if (tid == 0)
        for (int i = 0; i < STAGES - 1 && i < chunks; ++i) fetch(i);
    float raw[2][4], next[2][4];
    values(n, next);

    // The results of a chunk: warps 0 and 1, eight tokens each.
    float held[4], level[2];                                   // A V (+ A Z), and what Q S_0 is multiplied by (head decay)
    const size_t o_row = (size_t)H * Dv;
    float* o_at = out + (size_t)(r0 + 8 * wd + 2 * t4) * o_row + (size_t)h * Dv + col;
    auto store = [&](int ci) {                                 // called for the chunks in order
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < WD; ++w) {
            const float4 part = meet[ci & 1][w][wd][lane];
            o[0] += part.x; o[1] += part.y; o[2] += part.z; o[3] += part.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (MODE == CHUNK_HEAD_DECAY) o[e] *= level[e & 1];
            o[e] = (o[e] + held[e]) * q_scale;
        }
        const int left = n - ci * C - 8 * wd - 2 * t4;
        if (left > 0) {
            if (col0) o_at[0] = o[0];
            if (col1) o_at[8] = o[2];
        }
        if (left > 1) {
            if (col0) o_at[o_row] = o[1];
            if (col1) o_at[o_row + 8] = o[3];
        }
        o_at += C * o_row;
    };

    bool bad = false;
    int ci = 0;
    for (; ci < chunks; ++ci) {
        if (__syncthreads_or(bad)) break;                      // all are done with chunk ci - 1 (a wait that ran out ends the walk)
        if (tid == 0 && ci + STAGES - 1 < chunks) fetch(ci + STAGES - 1);
        if (!Z && ci > 0 && wd < 2) store(ci - 1);
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
#pragma unroll
            for (int e = 0; e < 4; ++e) raw[ks][e] = next[ks][e];
        if (ci + 1 < chunks) values(n - (ci + 1) * C, next);
        if (!tc::mbar_wait(&full[ci % STAGES], (ci / STAGES) & 1)) {
            bad = true;
            atomicOr(err, tc::KVB_DEV_TIMEOUT);
        }
        const float* b = sm + (ci % STAGES) * R.total;

        // This warp's channels' share of Q S_0 and Y S_0.
        float sum[NX][4];
#pragma unroll
        for (int x = 0; x < NX; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[x][e] = 0.f;
        constexpr int KP = KT < 8 / NX ? KT : 8 / NX;          // steps of eight channels taken together
#pragma unroll
        for (int k0 = 0; k0 < KT; k0 += KP) {
            Split a[KP];
            float bb[KP * NX][2], p[KP * NX][4];
#pragma unroll
            for (int k = 0; k < KP; ++k) {
                a[k] = as_operand(S[k0 + k]);
#pragma unroll
                for (int x = 0; x < NX; ++x)
                    pair(bb[k * NX + x], b + (x < 2 ? R.q : R.y) + (8 * (x & 1) + g) * (DP + 8) + ch0 + 8 * (k0 + k) + 2 * t4);
            }
            products<KP * NX>(p, [&](int i) -> const Split& { return a[i / NX]; }, bb);
#pragma unroll
            for (int i = 0; i < KP * NX; ++i) add4(sum[i % NX], p[i]);
        }
#pragma unroll
        for (int x = 0; x < NX; ++x) meet[ci & 1][wd][x][lane] = make_float4(sum[x][0], sum[x][1], sum[x][2], sum[x][3]);

        Split v[2], z[2];
        v[0] = as_operand(raw[0]);
        v[1] = as_operand(raw[1]);
        float wv[2][4];
        if (Z) {
            float bb[3][2], p[3][4];                           // W is zero above its diagonal
            pair(bb[0], b + R.w + g * 24 + 2 * t4);
            pair(bb[1], b + R.w + (8 + g) * 24 + 2 * t4);
            pair(bb[2], b + R.w + (8 + g) * 24 + 8 + 2 * t4);
            products<3>(p, [&](int i) -> const Split& { return v[i / 2]; }, bb);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                wv[0][e] = p[0][e];
                wv[1][e] = p[1][e] + p[2][e];
            }
            __syncthreads();
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float total[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int w = 0; w < WD; ++w) {
                    const float4 part = meet[ci & 1][w][2 + nt][lane];
                    total[0] += part.x; total[1] += part.y; total[2] += part.z; total[3] += part.w;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) total[e] += wv[nt][e];
                z[nt] = as_operand(total);
            }
        }
        if (wd < 2) {
            constexpr int NA = (V ? 2 : 0) + (Z ? 2 : 0);      // (for the first eight tokens the second half of A is zero)
            float bb[NA][2], p[NA][4];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                if (V) pair(bb[ks], b + R.a1 + (8 * wd + g) * 24 + 8 * ks + 2 * t4);
                if (Z) pair(bb[(V ? 2 : 0) + ks], b + R.a2 + (8 * wd + g) * 24 + 8 * ks + 2 * t4);
            }
            products<NA>(p, [&](int i) -> const Split& { return V && i < 2 ? v[i & 1] : z[i & 1]; }, bb);
#pragma unroll
            for (int e = 0; e < 4; ++e) held[e] = p[0][e] + p[1][e] + (NA > 2 ? p[NA - 2][e] + p[NA - 1][e] : 0.f);
            if (MODE == CHUNK_HEAD_DECAY) {
                level[0] = b[R.decay + 8 * wd + 2 * t4];
                level[1] = b[R.decay + 8 * wd + 2 * t4 + 1];
            }
            if (Z) store(ci);
        }

        // The state: the chunk's sum by itself, then added.
        if (MODE == CHUNK_HEAD_DECAY) {
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const float2 gain = *(const float2*)(b + R.decay + C + 8 * ks + 2 * t4);
                raw[ks][0] *= gain.x; raw[ks][2] *= gain.x;
                raw[ks][1] *= gain.y; raw[ks][3] *= gain.y;
                v[ks] = as_operand(raw[ks]);
            }
        }
        constexpr int NU = (V ? 2 : 0) + (Z ? 2 : 0), KU = KT < 8 / NU ? KT : 8 / NU;
#pragma unroll
        for (int k0 = 0; k0 < KT; k0 += KU) {
            float bb[KU * NU][2], p[KU * NU][4];
#pragma unroll
            for (int k = 0; k < KU; ++k) {
                const int d = ch0 + 8 * (k0 + k) + g;
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const int t = 8 * ks + 2 * t4;
                    if (V) {
                        bb[k * NU + ks][0] = b[R.k1 + t * (DP + 4) + d];
                        bb[k * NU + ks][1] = b[R.k1 + (t + 1) * (DP + 4) + d];
                    }
                    if (Z) {
                        bb[k * NU + NU - 2 + ks][0] = b[R.k2 + t * (DP + 4) + d];
                        bb[k * NU + NU - 2 + ks][1] = b[R.k2 + (t + 1) * (DP + 4) + d];
                    }
                }
            }
            products<KU * NU>(p, [&](int i) -> const Split& { return V && i % NU < 2 ? v[i & 1] : z[i & 1]; }, bb);
#pragma unroll
            for (int k = 0; k < KU; ++k) {
                const int kt = k0 + k;
#pragma unroll
                for (int i = 1; i < NU; ++i) add4(p[k * NU], p[k * NU + i]);
                const float2 keep = MODE == CHUNK_HEAD_DECAY ? make_float2(b[R.decay + 2 * C], b[R.decay + 2 * C])
                                                             : *(const float2*)(b + R.decay + ch0 + 8 * kt + 2 * t4);
                S[kt][0] = fmaf(keep.x, S[kt][0], p[k * NU][0]);
                S[kt][1] = fmaf(keep.y, S[kt][1], p[k * NU][1]);
                S[kt][2] = fmaf(keep.x, S[kt][2], p[k * NU][2]);
                S[kt][3] = fmaf(keep.y, S[kt][3], p[k * NU][3]);
            }
        }
    }
    if (ci < chunks || bad) {                                  // a record did not come: the copies asked for are waited for (or given up)
        if (tid == 0) {
            for (int i = ci; i < chunks && i < ci + STAGES - 1; ++i) tc::mbar_wait(&full[i % STAGES], (i / STAGES) & 1);
        }
        return;
    }
    if (!Z) {
        __syncthreads();
        if (wd < 2) store(chunks - 1);
    }
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = ch0 + 8 * kt + 2 * t4 + (e & 1);
            if (d < D && (e < 2 ? col0 : col1)) mem[(size_t)d * Dv + col + 8 * (e >> 1)] = S[kt][e];
        }
}

template <int MODE, int NI, int KT, int STAGES>
static int launch_walk(const Rows& in, const Segments& seg, const float* records, int max_chunks, float q_scale, float* memory, float* out,
                       int H, int D, int Dv, int* err, cudaStream_t stream) {
    constexpr int bytes = STAGES * record_of(MODE, 64 * NI).total * (int)sizeof(float);
    if (bytes > 8 * 1024) {                                    // (the kernel has up to 32 KB of its own beside it)
        const cudaError_t e = cudaFuncSetAttribute(chunk_walk_kernel<MODE, NI, KT, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return (int)e;
    }
    // Not as a dependent launch: blocks placed while the records are still being made crowd onto the SMs that are free first, and
    // stay there (7 heads of 64 x 128, 2,048 tokens: 219 us against 112).
    chunk_walk_kernel<MODE, NI, KT, STAGES><<<dim3((Dv + 15) / 16, H, seg.count), 64 * NI / (8 * KT) * 32, bytes, stream>>>(
        in, seg, records, max_chunks, q_scale, memory, out, H, D, Dv, err);
    return kvb_launch_status();
}

template <int MODE, int NI>
static int run(const Rows& in, const Segments& seg, float* records, int max_chunks, float q_scale, float* memory, float* out, int H, int D,
               int Dv, int* err, cudaStream_t stream) {
    if constexpr (MODE == CHUNK_HEAD_DECAY)
        kvb_launch(head_records_kernel<NI>, dim3(max_chunks, H / in.qk_div), dim3(256), 0, stream, in, seg, records, H, D);
    else
    {
        const int wide = ((D | in.stride | in.gate_stride | in.q_col | in.k_col) & 3) == 0 && (((uintptr_t)in.rows | (uintptr_t)in.gates) & 15) == 0;
        kvb_launch(chunk_records_kernel<MODE, NI>, dim3(max_chunks, H), dim3(256), 0, stream, in, seg, records, H, D, wide);
        if constexpr (MODE == CHUNK_DELTA_RULE)
            kvb_launch(chunk_solve_kernel<NI>, dim3(max_chunks, H), dim3(64 * NI), 0, stream, seg, records, H);
    }
    const int rc = kvb_launch_status();
    if (rc != KVB_OK) return rc;
    // Key channels a warp holds: 16 of 64 (four warps), 32 of 128 (four warps); with two warps (eight) a column the same calls take 6
    // to 45 % (8 to 22 %) longer.  A third stage never pays: it costs blocks an SM.
    return launch_walk<MODE, NI, 2 * NI, 2>(in, seg, records, max_chunks, q_scale, memory, out, H, D, Dv, err, stream);
}

// Whether the columns that the heads read lie within a row of `rows` and of `gates` (the decays of CHUNK_CHANNEL_DECAY are rows of
// their own).
static bool rows_fit(int mode, const Rows& in, int H, int G, int D, int Dv) {
    const long long qk = (long long)G * D, a = (long long)H * D;
    if (in.q_col < 0 || in.k_col < 0 || in.v_col < 0 || in.q_col + qk > in.stride || in.k_col + qk > in.stride ||
        in.v_col + (long long)H * Dv > in.stride)
        return false;
    if (mode == CHUNK_CHANNEL_DECAY) return in.gate_stride == a;
    return in.gate_stride >= (mode == CHUNK_GATED_DELTA ? a + H : mode == CHUNK_DELTA_RULE ? 3 * a : 2LL * H);
}

template <int MODE>
static int run(const Rows& in, const Segments& seg, float* records, int max_chunks, float q_scale, float* memory, float* out, int T, int H,
               int G, int D, int Dv, int* err, cudaStream_t stream) {
    if (H < 1 || G < 1 || H % G || D < 1 || Dv < 1 || !rows_fit(MODE, in, H, G, D, Dv)) return KVB_ERR_SHAPE;
    if (seg.count <= 0 || T <= 0) return KVB_OK;
    if (records == nullptr) return KVB_ERR_SHAPE;
    if ((uintptr_t)records & 15) return KVB_ERR_ALIGN;
    if (D > 128 || H > 65535 || seg.count > 65535 || max_chunks < T / C + seg.count) return KVB_ERR_LIMIT;
    if (MODE == CHUNK_CHANNEL_DECAY && Dv > 512) return KVB_ERR_LIMIT;      // as the other forms of this scan
    return D <= 64 ? run<MODE, 1>(in, seg, records, max_chunks, q_scale, memory, out, H, D, Dv, err, stream)
                   : run<MODE, 2>(in, seg, records, max_chunks, q_scale, memory, out, H, D, Dv, err, stream);
}

}  // namespace sc

// Floats of scratch a (chunk of 16 tokens, head) takes; mode 0 gated delta, 1 delta rule, 2 channel decay, 3 head decay.
KVB_API int kvb_chunk_record_floats(int mode, int D) {
    return mode < 0 || mode > 3 || D < 1 ? -1 : sc::record_of(mode, sc::padded(D)).total - sc::record_of(mode, sc::padded(D)).shared;
}
// ... and what a (chunk, group of heads that share q and k) takes besides.
KVB_API int kvb_chunk_shared_floats(int mode, int D) { return mode < 0 || mode > 3 || D < 1 ? -1 : sc::record_of(mode, sc::padded(D)).shared; }

// The scans over portions of prompts.  `rows` [T, stride] holds q, k and v at their columns (head h: number h / (H / G) of D for q and k,
// number h of Dv for v; H a multiple of G), `gates` [T, gate_stride] the mode's own numbers (sc::Rows); `records`: scratch of max_chunks
// (at least T / 16 + S) times the floats above for all H heads and G groups, on 16 bytes.  D up to 128.
KVB_API int kvb_chunk_scan(int mode, const float* rows, int stride, int q_col, int k_col, int v_col, int G, const float* gates,
                           int gate_stride, float q_scale, const int* seg_q_start, const int* seg_q_len, const int* seg_slot, float* memory,
                           float* out, int T, int S, int H, int D, int Dv, int max_chunks, float* records, int* err, cudaStream_t stream) {
    const sc::Rows in = {rows, gates, stride, gate_stride, q_col, k_col, v_col, G > 0 ? H / G : 0};
    const sc::Segments seg = {seg_q_start, seg_q_len, seg_slot, S};
    if (mode == sc::CHUNK_GATED_DELTA) return sc::run<sc::CHUNK_GATED_DELTA>(in, seg, records, max_chunks, q_scale, memory, out, T, H, G, D, Dv, err, stream);
    if (mode == sc::CHUNK_DELTA_RULE) return sc::run<sc::CHUNK_DELTA_RULE>(in, seg, records, max_chunks, q_scale, memory, out, T, H, G, D, Dv, err, stream);
    if (mode == sc::CHUNK_CHANNEL_DECAY) return sc::run<sc::CHUNK_CHANNEL_DECAY>(in, seg, records, max_chunks, q_scale, memory, out, T, H, G, D, Dv, err, stream);
    if (mode == sc::CHUNK_HEAD_DECAY) return sc::run<sc::CHUNK_HEAD_DECAY>(in, seg, records, max_chunks, q_scale, memory, out, T, H, G, D, Dv, err, stream);
    return KVB_ERR_SHAPE;
}
