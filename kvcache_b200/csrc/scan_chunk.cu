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
// chunk): the decays between two tokens are multiplied up one after the other and never divided by, so that any decay down to zero is
// exact.  Launch (2) walks a segment's chunks in order, a block per 16 value channels of a head: S lives in registers, a thread's key
// channels of two value channels; Y S_0 and Q S_0 are summed over a warp's key channels by shuffles and over the warps through shared
// memory, in one order by all of them.  A record lies in scratch as it will lie in shared memory and comes in by one bulk copy, a chunk ahead.
//
// All of it is float32 multiply-adds on the CUDA cores, in an order that rounds no worse than a walk over tokens: decays over the
// chunk are products that are rounded once, and the chunk's last tokens are added to the state one by one.  Against 64 bits results and
// states are off by 0.6 to 1.1 of what the scans over tokens are off by (states of models: 0.5e-7 to 1.1e-7; slow decays 1.6e-7 to 4.3e-7 where those
// are at 1.9e-7 to 4.9e-7).
//
// What bounds it: the latency of a chunk's steps - shared memory, shuffles, two or three barriers, 1.2 to 2.6 us - times the chunks of the longest
// segment.  Measured beside the form each replaces (us; records and walk): gated delta 777 x 14 x 64 x 64: 115 -> 85, 1,500 x 16 x 128 x 128:
// 325 -> 235; delta rule 543 + 905 + 363 x 16 x 128: 660 -> 252, 1,000 x 14 x 64: 196 -> 143; channel decays 600 + 400 x 8 x 128 x 256: 148 -> 68; head
// decays 2,048 x 64 x 128 x 64: 278 -> 262.  Level or up to 5 % behind: 2,048 x 14 x 64 under the delta rule (297 -> 311), 48 tokens beside 63
// single ones under the gated one (46 -> 48), 512 x 28 x 128 x 64 head decays (53 -> 54).  Registers for four blocks an SM: with more, steps of
// several segments take up to 40 % longer, with the compiler's own choice single ones 5 %.
// Where heads are few, runs of a long segment's chunks are walked at once (modes without Z, further down): 2,048 rows of 7 heads of 64 x 128, records
// and walk 147 -> 53 us; of 28 heads of 128 x 64 under head decays 193 -> 133.  From 256 blocks a segment on the walk has warps enough (16 heads of
// 128 x 256: 280 -> 288), and so have steps of many long segments, which pay a third for it (eight of 1,024 rows of the 7 heads: 160 -> 219).
// A weight above a diagonal is zero and is multiplied like any other; only in a chunk whose values are not all finite (a vote) are
// later tokens left out one by one, which takes 15 to 35 % longer where it is done always.
// A segment's result does not depend on what else the step holds (unless their records are more than is held at once: then no segment is cut
// into runs), and a token's not on later ones, whatever they hold (an infinite or undefined
// number of one reaches those after it, as in a walk over tokens).
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

// A product of many decays and what its roundings lost: it counts once for all sixteen tokens, so it is rounded once.
struct Decay {
    float high = 1.f, low = 0.f;
    __device__ __forceinline__ void times(float a) {
        const float p = __fmul_rn(high, a);
        low = fmaf(low, a, fmaf(high, a, -p));
        high = p;
    }
    __device__ __forceinline__ float value() const { return __fadd_rn(high, low); }
};

// ---- launches (1): the records ---------------------------------------------------------------------------------------------
// grid (chunks from `first` on, heads), 256 threads.  Thread (s, part): token s as a key, channels 4 part .. + 3 of every 64.
template <int MODE, int NI>          // NI: 64-channel groups of a row
__global__ void __launch_bounds__(256, MODE == CHUNK_DELTA_RULE && NI == 2 ? 3 : 4) chunk_records_kernel(const Rows in, const Segments seg,
                                                                                                       float* __restrict__ records, int first,
                                                                                                       int H, int D, int wide) {
    constexpr int DP = 64 * NI, PARTS = MODE == CHUNK_DELTA_RULE ? 5 : 3;
    __shared__ __align__(16) float rows_s[PARTS][C][DP];       // q, k, a (, u, c)
    __shared__ float low_s[C][C + 1], mat_s[C][C + 1], b_s[C];
    const int tid = threadIdx.x, s = tid >> 4, part = tid & 15, h = blockIdx.y;
    pdl_wait();
    pdl_launch_dependents();
    int r0, count;
    if (!find_chunk(first + blockIdx.x, seg, r0, count)) return;
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
        Decay run;
#pragma unroll
        for (int t = 0; t < C; ++t) {
            const float before = run.value();
            run.times(rows_s[2][t][d]);
            const float upto = run.value();
            rec[R.q + t * (DP + 8) + d] = rows_s[0][t][d] * upto;
            if (MODE == CHUNK_GATED_DELTA) rows_s[0][t][d] = rows_s[1][t][d] * upto;                   // the key as it meets S_0
            if (MODE == CHUNK_DELTA_RULE) rec[R.y + t * (DP + 8) + d] = rows_s[3][t][d] * before;
        }
        rec[R.decay + d] = run.value();
    } else if (tid < 2 * DP) {
        Decay run;
#pragma unroll
        for (int t = C - 1; t >= 0; --t) {
            const float after = run.value();
            rec[(has_v(MODE) ? R.k1 : R.k2) + t * (DP + 4) + d] = rows_s[1][t][d] * after;
            if (MODE == CHUNK_DELTA_RULE) rec[R.k2 + t * (DP + 4) + d] = -rows_s[4][t][d] * after;
            run.times(rows_s[2][t][d]);
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
__global__ void __launch_bounds__(64 * NI) chunk_solve_kernel(const Segments seg, float* __restrict__ records, int first, int H) {
    constexpr int DP = 64 * NI;
    constexpr Record R = record_of(CHUNK_DELTA_RULE, DP);
    __shared__ float low_s[C][C + 1], mat_s[C][C + 1];
    const int d = threadIdx.x;
    pdl_wait();
    pdl_launch_dependents();
    int r0, count;
    if (!find_chunk(first + blockIdx.x, seg, r0, count)) return;
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

// Head decay: grid (chunks from `first` on, groups of heads with one q and k); `held`: the chunks that `records` has room for.
template <int NI>
__global__ void __launch_bounds__(256) head_records_kernel(const Rows in, const Segments seg, float* __restrict__ records, int first, int held, int H,
                                                           int D) {
    constexpr int DP = 64 * NI, HEADS = 16;
    __shared__ __align__(16) float q_s[C][DP], k_s[C][DP];
    __shared__ float qk_s[C][C + 1], a_s[HEADS][C], d_s[HEADS][C];
    const int tid = threadIdx.x, s = tid >> 4, part = tid & 15, g = blockIdx.y;
    pdl_wait();
    pdl_launch_dependents();
    int r0, count;
    if (!find_chunk(first + blockIdx.x, seg, r0, count)) return;
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
    const int groups = H / in.qk_div, head0 = g * in.qk_div, head1 = head0 + in.qk_div;
    {
        float* rec = records + ((size_t)blockIdx.x * groups + g) * R.shared;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int d = 64 * i + 4 * part;
            *(float4*)(rec + R.q + s * (DP + 8) + d) = *(const float4*)&q_s[s][d];
            *(float4*)(rec + R.k1 + s * (DP + 4) + d) = *(const float4*)&k_s[s][d];
        }
        records += (size_t)held * groups * R.shared;
    }
    for (int h0 = head0; h0 < head1; h0 += HEADS) {
        __syncthreads();
        {                                                          // head h0 + part, token s
            const bool there = h0 + part < head1 && s < count;
            const float* gate = in.gates + (size_t)(r0 + (there ? s : 0)) * in.gate_stride + (there ? h0 + part : 0);
            a_s[part][s] = there ? gate[0] : 1.f;
            d_s[part][s] = there ? gate[H] : 0.f;
        }
        __syncthreads();
        // Thread (head h0 + s, token `part` as a key).
        const int h = h0 + s;
        if (h < head1) {
            float* rec = records + ((size_t)blockIdx.x * H + h) * (R.total - R.shared);
            const float gain = d_s[s][part];
            Decay run, all;
#pragma unroll
            for (int t = 0; t < C; ++t) {
                const float a = a_s[s][t];
                if (t > part) run.times(a);
                else all.times(a);
                const float full = gain * run.high, rest = fmaf(gain, run.low, fmaf(gain, run.high, -full)), qk = qk_s[t][part];
                rec[R.a1 - R.shared + t * 24 + part] = t >= part ? fmaf(qk, full, qk * rest) : 0.f;
            }
            rec[part] = all.value();                               // L_t, t = part
            rec[C + part] = gain * run.value();
            if (part == C - 1) rec[2 * C] = all.value();           // L_C
        }
    }
}

// ---- launch (2): the walk -------------------------------------------------------------------------------------------------
// Two float32 multiply-adds in one instruction, each rounded as `fmaf` rounds.
__device__ __forceinline__ float2 fma2(const float2& a, const float2& b, const float2& c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(*(const uint64_t*)&a), "l"(*(const uint64_t*)&b), "l"(*(const uint64_t*)&c));
    return *(const float2*)&d;
}
__device__ __forceinline__ float2 mul2(const float2& a, const float2& b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(*(const uint64_t*)&a), "l"(*(const uint64_t*)&b));
    return *(const float2*)&d;
}
__device__ __forceinline__ float2 low2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 high2(const float4& v) { return make_float2(v.z, v.w); }

// N neighbouring numbers in shared memory.
template <int N> __device__ __forceinline__ void load(const float* at, float (&v)[N]) {
    if constexpr (N == 2) {
        const float2 x = *(const float2*)at;
        v[0] = x.x; v[1] = x.y;
    } else {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) {
            const float4 x = *(const float4*)(at + 4 * i);
            v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
        }
    }
}
template <int N> __device__ __forceinline__ void keep(float* at, const float (&v)[N]) {
    if constexpr (N == 2) *(float2*)at = make_float2(v[0], v[1]);
    else *(float4*)at = make_float4(v[0], v[1], v[2], v[3]);
}

// Each number twice, for `fma2`.
template <int N> __device__ __forceinline__ void pairs(const float* at, float2 (&v)[N]) {
    float x[N];
    load<N>(at, x);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = make_float2(x[i], x[i]);
}
template <int N> __device__ __forceinline__ bool finite(const float (&v)[N]) {
    bool all = true;
#pragma unroll
    for (int i = 0; i < N; ++i) all &= fabsf(v[i]) <= FLT_MAX;
    return all;
}
// sum += tokens 0 .. t of x [C][16] with the weights of a row of a lower triangular matrix (of two, token by token), in order.  The zeros
// above its diagonal are multiplied too, unless MASKED: zero times an infinite or undefined number of a later token is not zero.
template <int N, bool MASKED>
__device__ __forceinline__ void add_tokens(const float* row, const float* x, int t, float (&sum)[N]) {
    float a[C], v[N];
    load<C>(row, a);
#pragma unroll
    for (int s = 0; s < C; ++s) {
        load<N>(x + 16 * s, v);
#pragma unroll
        for (int c = 0; c < N; ++c) sum[c] = MASKED && s > t ? sum[c] : fmaf(a[s], v[c], sum[c]);
    }
}
template <int N, bool MASKED>
__device__ __forceinline__ void add_tokens(const float* row1, const float* x1, const float* row2, const float* x2, int t, float (&sum)[N]) {
    float a1[C], a2[C], v[N];
    load<C>(row1, a1);
    load<C>(row2, a2);
#pragma unroll
    for (int s = 0; s < C; ++s) {
        load<N>(x1 + 16 * s, v);
#pragma unroll
        for (int c = 0; c < N; ++c) sum[c] = MASKED && s > t ? sum[c] : fmaf(a1[s], v[c], sum[c]);
        load<N>(x2 + 16 * s, v);
#pragma unroll
        for (int c = 0; c < N; ++c) sum[c] = MASKED && s > t ? sum[c] : fmaf(a2[s], v[c], sum[c]);
    }
}

__device__ __forceinline__ void copy_bulk(float* smem, const float* gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(tc::smem_u32(smem)), "l"(gmem), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
}

// What a segment's chunks are cut into where several runs of them are walked at once (see launches (2) below).  By the segment's own
// length: what else the step holds changes nothing.
struct Runs {
    int wanted;                  // runs a segment is cut into at most (0: every segment is one run)
    int least, from;             // chunks a run has at least; chunks from which a segment is cut
    float* starts;               // [runs of segments with several, H, D, Dv]: the states that runs start from
    float* decays;               // [those runs, H, 64 NI or 1]: the product of a run's decays
};
struct Run {
    int seg, number, count;      // the run's segment, its number within it and the segment's count of runs
    int chunks;                  // chunks of each of them but the last
    int place;                   // among the runs of segments that have several
};
__device__ __forceinline__ Run runs_of(int n, const Runs& runs) {
    const int chunks = (n + C - 1) / C;
    Run r = {0, 0, chunks > 0, chunks, 0};
    if (chunks >= runs.from && chunks > 0 && runs.wanted > 1) {
        r.chunks = max(runs.least, (chunks - 1) / runs.wanted + 1);
        r.count = (chunks - 1) / r.chunks + 1;
    }
    return r;
}
// Run `id` of the step, or, with `SEVERAL`, of the segments that have several; false beyond the last.
template <bool SEVERAL>
__device__ __forceinline__ bool find_run(int id, const Segments& seg, const Runs& runs, Run& r) {
    int place = 0;
    for (int s = 0; s < seg.count; ++s) {
        r = runs_of(seg.q_len[s], runs);
        const int mine = SEVERAL && r.count == 1 ? 0 : r.count;
        if (id < mine) {
            r.seg = s;
            r.number = id;
            r.place = place + id;
            return true;
        }
        id -= mine;
        place += r.count > 1 ? r.count : 0;
    }
    return false;
}

// grid (16 value channels, heads, segments or runs), over the chunks first .. first + held - 1 of the step.  A thread holds TD neighbouring key channels of TC value channels of the state; a warp's lanes
// are 2 TC groups of key channels by 16 / TC of value channels.  Beside that, every thread owns one token's OC value channels of Z and O.
template <int MODE, int NI, int TD, int TC, int STAGES>
__global__ void __launch_bounds__(16 * 64 * NI / (TD * TC), 4) chunk_walk_kernel(const Rows in, const Segments seg, const float* __restrict__ records,
                                                                             int first, int held, float q_scale, float* __restrict__ memory,
                                                                             float* __restrict__ out, int H, int D, int Dv, const Runs runs,
                                                                             int* __restrict__ err) {
    constexpr bool Z = has_z(MODE), V = has_v(MODE);
    constexpr int DP = 64 * NI, CG = 16 / TC, DG = 32 / CG, WARPS = DP / (TD * DG), OC = 16 * C / (32 * WARPS);
    constexpr int NR = Z ? 2 * C : C;                          // rows that meet S_0: [Y | Q] or Q
    constexpr Record R = record_of(MODE, DP);
    static_assert((OC == 2 || OC == 4) && (TC == 2 || TC == 4) && TD % 4 == 0, "");
    static_assert(!Z || R.q == R.y + C * (DP + 8), "the rows of Y and Q follow one another");
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(16) float meet[WARPS][NR][16];        // the warps' shares of Y S_0 and Q S_0
    __shared__ __align__(16) float v_s[2][C][16], z_s[Z ? C : 1][16];
    __shared__ __align__(8) uint64_t full[STAGES];
    const int tid = threadIdx.x, lane = tid & 31, wd = tid >> 5, cg = lane % CG, dg = lane / CG;
    const int h = blockIdx.y;
    Run run = {(int)blockIdx.z, 0, 1, 0, 0};
    if (runs.wanted > 0 && !find_run<false>(blockIdx.z, seg, runs, run)) return;
    const int sg = run.seg;
    int n = seg.q_len[sg], r0 = seg.q_start[sg], chunk0 = 0;
    const int slot = seg.slot[sg];
    if (n <= 0) return;
    for (int i = 0; i < sg; ++i) chunk0 += (seg.q_len[i] + C - 1) / C;
    // The segment's chunks from `begin` on that are among the `held` whose records are there.
    const int begin = max(run.number * run.chunks, first - chunk0), d0 = (wd * DG + dg) * TD;
    int chunks = min((n + C - 1) / C, first + held - chunk0) - begin;
    if (run.count > 1) chunks = min(chunks, run.chunks);
    if (chunks <= 0) return;
    n -= begin * C;
    r0 += begin * C;
    chunk0 += begin - first;

    float* mem = memory + ((size_t)slot * H + h) * D * Dv;
    const float* start = run.count > 1 ? runs.starts + ((size_t)run.place * H + h) * D * Dv : mem;
    const int col0 = 16 * blockIdx.x + cg * TC;
    float2 S[TD / 2][TC];                                      // key channels d0 + 2 i and the next
#pragma unroll
    for (int i = 0; i < TD / 2; ++i)
#pragma unroll
        for (int c = 0; c < TC; ++c) {
            const int d = d0 + 2 * i;
            const float* at = start + (size_t)d * Dv + col0 + c;
            S[i][c] = make_float2(d < D && col0 + c < Dv ? at[0] : 0.f, d + 1 < D && col0 + c < Dv ? at[Dv] : 0.f);
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
            copy_bulk(b + R.shared, records + (size_t)held * groups * R.shared + (id * H + h) * (R.total - R.shared), (R.total - R.shared) * 4, bar);
        } else {
            copy_bulk(b, records + (id * H + h) * R.total, R.total * 4, bar);
        }
    };
    // This thread's token of every chunk, and its value channels.
    const int t = tid / (16 / OC), oc = OC * (tid % (16 / OC)), col = 16 * blockIdx.x + oc;
    const float* v_at = in.rows + (size_t)(r0 + t) * in.stride + in.v_col + (size_t)h * Dv + col;
    auto values = [&](int ci, float (&v)[OC]) {
        const bool there = ci * C + t < n;
        const float* at = v_at + (there ? (size_t)ci * C * in.stride : 0);
#pragma unroll
        for (int c = 0; c < OC; ++c) v[c] = there && col + c < Dv ? at[c] : 0.f;
    };
    float next[OC];
    values(0, next);
    keep<OC>(&v_s[0][t][oc], next);
    __syncthreads();
    if (tid == 0)
        for (int i = 0; i < STAGES - 1 && i < chunks; ++i) fetch(i);

    bool bad = false, failed = false;
    int ci = 0;
    for (;; ++ci) {
        // All are done with chunk ci - 1.  A wait that ran out ends the walk; values that are not all finite leave later tokens out one by one.
        bool wild = __syncthreads_or(bad || !finite(next));
        if (wild) failed = __syncthreads_or(bad);
        if (failed || ci == chunks) break;
        if (tid == 0 && ci + STAGES - 1 < chunks) fetch(ci + STAGES - 1);
        values(ci + 1, next);
        if (!tc::mbar_wait(&full[ci % STAGES], (ci / STAGES) & 1)) {
            bad = true;
            atomicOr(err, tc::KVB_DEV_TIMEOUT);
        }
        const float* b = sm + (ci % STAGES) * R.total;
        const float(*v_c)[16] = v_s[ci & 1];
        const int left = n - ci * C;                           // tokens from the chunk's first on: those after them change nothing

        // Y S_0 and Q S_0, eight rows at a time: this thread's key channels, then the warp's.
        const float* rows = b + (Z ? R.y : R.q) + d0;
#pragma unroll
        for (int row0 = 0; row0 < NR; row0 += 8) {
            float2 acc[8][TC];
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int q = 0; q < TD / 4; ++q) {
                    const float4 y = *(const float4*)(rows + (row0 + r) * (DP + 8) + 4 * q);
#pragma unroll
                    for (int c = 0; c < TC; ++c) {
                        acc[r][c] = q ? fma2(low2(y), S[2 * q][c], acc[r][c]) : mul2(low2(y), S[0][c]);
                        acc[r][c] = fma2(high2(y), S[2 * q + 1][c], acc[r][c]);
                    }
                }
            float sum[8][TC];
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int c = 0; c < TC; ++c) sum[r][c] = acc[r][c].x + acc[r][c].y;
            // A lane ends with 8 / DG of the rows, summed over the warp's key channels.
            int mine = 0;
#pragma unroll
            for (int off = 16, count = 4; off >= CG; off >>= 1, count >>= 1) {
                const bool upper = lane & off;
                mine += upper ? count : 0;
#pragma unroll
                for (int r = 0; r < count; ++r)
#pragma unroll
                    for (int c = 0; c < TC; ++c) {
                        const float keep = upper ? sum[r + count][c] : sum[r][c], give = upper ? sum[r][c] : sum[r + count][c];
                        sum[r][c] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                    }
            }
#pragma unroll
            for (int r = 0; r < 8 / DG; ++r)
#pragma unroll
                for (int c = 0; c < TC; ++c) meet[wd][row0 + mine + r][cg * TC + c] = sum[r][c];
        }
        float z_own[OC] = {}, o[OC] = {};
        if (Z) {                                               // W V, while the others get here
            if (!wild) add_tokens<OC, false>(b + R.w + t * 24, &v_c[0][oc], t, z_own);
            else add_tokens<OC, true>(b + R.w + t * 24, &v_c[0][oc], t, z_own);
        }
        __syncthreads();
        {
            float y_sum[OC] = {};
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                float part[OC];
                if (Z) {
                    load<OC>(&meet[w][t][oc], part);
#pragma unroll
                    for (int c = 0; c < OC; ++c) y_sum[c] += part[c];
                }
                load<OC>(&meet[w][NR - C + t][oc], part);
#pragma unroll
                for (int c = 0; c < OC; ++c) o[c] += part[c];
            }
            if (Z) {
#pragma unroll
                for (int c = 0; c < OC; ++c) z_own[c] = t < left ? y_sum[c] + z_own[c] : 0.f;
                keep<OC>(&z_s[t][oc], z_own);
            }
            if (MODE == CHUNK_HEAD_DECAY) {
                const float level = b[R.decay + t];
#pragma unroll
                for (int c = 0; c < OC; ++c) o[c] *= level;
            }
        }
        if (Z) wild |= (bool)__syncthreads_or(!finite(z_own));
        // The results: tokens in order on top of Q S_0.
        {
            const float *a1 = b + R.a1 + t * 24, *a2 = b + R.a2 + t * 24;
            if constexpr (Z && V) {
                if (!wild) add_tokens<OC, false>(a2, &z_s[0][oc], a1, &v_c[0][oc], t, o);
                else add_tokens<OC, true>(a2, &z_s[0][oc], a1, &v_c[0][oc], t, o);
            } else {
                const float *a = Z ? a2 : a1, *x = Z ? &z_s[0][oc] : &v_c[0][oc];
                if (!wild) add_tokens<OC, false>(a, x, t, o);
                else add_tokens<OC, true>(a, x, t, o);
            }
            if (ci * C + t < n) {
                float* at = out + (size_t)(r0 + ci * C + t) * H * Dv + (size_t)h * Dv + col;
#pragma unroll
                for (int c = 0; c < OC; ++c)
                    if (col + c < Dv) at[c] = o[c] * q_scale;
            }
        }
        // The state: earlier tokens by themselves, the decayed state, the chunk's last tokens (eight of sixteen, fewer of fewer) on top, in their
        // order: fewer roundings of a state that decays slowly than a walk over tokens makes, and no others where the last tokens dominate.
        const int split = left > 12 ? 8 : left > 8 ? 4 : 0;
        float2 N[TD / 2][TC];
#pragma unroll
        for (int i = 0; i < TD / 2; ++i)
#pragma unroll
            for (int c = 0; c < TC; ++c) N[i][c] = make_float2(0.f, 0.f);
#pragma unroll
        for (int s = 0; s < C; ++s) {
            if (s % 4 == 0 && s <= 8 && s == split) {
#pragma unroll
                for (int i = 0; i < TD / 4; ++i) {
                    float4 decay;
                    if (MODE == CHUNK_HEAD_DECAY) decay.x = decay.y = decay.z = decay.w = b[R.decay + 2 * C];
                    else decay = *(const float4*)(b + R.decay + d0 + 4 * i);
#pragma unroll
                    for (int c = 0; c < TC; ++c) {
                        N[2 * i][c] = fma2(low2(decay), S[2 * i][c], N[2 * i][c]);
                        N[2 * i + 1][c] = fma2(high2(decay), S[2 * i + 1][c], N[2 * i + 1][c]);
                    }
                }
            }
            float2 v[TC], z[TC];
            if (Z) pairs(&z_s[s][cg * TC], z);
            if (V) pairs(&v_c[s][cg * TC], v);
            if (MODE == CHUNK_HEAD_DECAY) {
                const float gain = b[R.decay + C + s];
#pragma unroll
                for (int c = 0; c < TC; ++c) v[c] = mul2(v[c], make_float2(gain, gain));
            }
#pragma unroll
            for (int i = 0; i < TD / 4; ++i) {
                float4 k1, k2;
                if (Z) k2 = *(const float4*)(b + R.k2 + s * (DP + 4) + d0 + 4 * i);
                if (V) k1 = *(const float4*)(b + R.k1 + s * (DP + 4) + d0 + 4 * i);
#pragma unroll
                for (int c = 0; c < TC; ++c) {
                    float2 &low = N[2 * i][c], &high = N[2 * i + 1][c];
                    if (Z) {
                        low = fma2(low2(k2), z[c], low);
                        high = fma2(high2(k2), z[c], high);
                    }
                    if (V) {
                        low = fma2(low2(k1), v[c], low);
                        high = fma2(high2(k1), v[c], high);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < TD / 2; ++i)
#pragma unroll
            for (int c = 0; c < TC; ++c) S[i][c] = N[i][c];
        keep<OC>(&v_s[(ci + 1) & 1][t][oc], next);
    }
    if (failed) {                                              // the copies asked for are waited for (or given up)
        if (tid == 0)
            for (int i = ci - 1; i < chunks && i < ci + STAGES - 1; ++i) tc::mbar_wait(&full[i % STAGES], (i / STAGES) & 1);
        return;
    }
    if (run.number + 1 < run.count) return;                    // the next run has started from this state already
#pragma unroll
    for (int i = 0; i < TD / 2; ++i)
#pragma unroll
        for (int c = 0; c < TC; ++c) {
            const int d = d0 + 2 * i;
            float* at = mem + (size_t)d * Dv + col0 + c;
            if (d < D && col0 + c < Dv) at[0] = S[i][c].x;
            if (d + 1 < D && col0 + c < Dv) at[Dv] = S[i][c].y;
        }
}

// ---- launches (2) of the modes without Z, where the heads are too few to fill the GPU: several runs of a segment's chunks at once -----
// A run's end is P S_0 + U, with P the product of its decays and U what its tokens leave of a state of zero.  First U and P of every run but a
// segment's last (a thread's share of the state as in the walk, no barrier but the one that hands a stage back), then the states that
// runs start from, one after the other element by element, then the walk with a block for every run.
// grid (16 value channels, heads, runs of segments that have several).  U of run r goes to place r + 1.
template <int MODE, int NI, int TD, int TC, int STAGES>
__global__ void __launch_bounds__(16 * 64 * NI / (TD * TC), 4) chunk_ends_kernel(const Rows in, const Segments seg, const float* __restrict__ records,
                                                                             int held, int H, int D, int Dv, const Runs runs,
                                                                             int* __restrict__ err) {
    static_assert(!has_z(MODE), "");
    constexpr int DP = 64 * NI, CG = 16 / TC, DG = 32 / CG, THREADS = 16 * DP / (TD * TC);
    constexpr Record R = record_of(MODE, DP);
    constexpr bool HEAD = MODE == CHUNK_HEAD_DECAY;
    constexpr int KEYS = C * (DP + 4), PART = KEYS + (HEAD ? 3 * C : DP);      // what is wanted of a record: K1 and the decays
    static_assert(HEAD || R.decay == R.k1 + KEYS, "K1 and the decays follow one another");
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(16) float v_s[2][C][16];
    __shared__ __align__(8) uint64_t full[STAGES];
    const int tid = threadIdx.x, lane = tid & 31, wd = tid >> 5, cg = lane % CG, dg = lane / CG, h = blockIdx.y;
    Run run;
    if (!find_run<true>(blockIdx.z, seg, runs, run) || run.number + 1 == run.count) return;
    int r0 = seg.q_start[run.seg], chunk0 = run.number * run.chunks;
    for (int i = 0; i < run.seg; ++i) chunk0 += (seg.q_len[i] + C - 1) / C;
    r0 += run.number * run.chunks * C;
    const int chunks = run.chunks, d0 = (wd * DG + dg) * TD, col0 = 16 * blockIdx.x + cg * TC, groups = H / in.qk_div;
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) tc::mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    auto fetch = [&](int ci) {
        float* b = sm + (ci % STAGES) * PART;
        uint64_t* bar = &full[ci % STAGES];
        const size_t id = chunk0 + ci;
        tc::mbar_expect_tx(bar, PART * 4);
        if (HEAD) {
            copy_bulk(b, records + (id * groups + h / in.qk_div) * R.shared + R.k1, KEYS * 4, bar);
            copy_bulk(b + KEYS, records + (size_t)held * groups * R.shared + (id * H + h) * (R.total - R.shared), 3 * C * 4, bar);
        } else {
            copy_bulk(b, records + (id * H + h) * R.total + R.k1, PART * 4, bar);
        }
    };
    // 16 x 16 values of a chunk, shared out over the threads.
    auto values = [&](int ci, float (&v)[16 * C / THREADS]) {
#pragma unroll
        for (int e = 0; e < 16 * C / THREADS; ++e) {
            const int at = tid + e * THREADS, t = at >> 4, col = 16 * blockIdx.x + (at & 15);
            v[e] = ci < chunks && col < Dv ? in.rows[(size_t)(r0 + ci * C + t) * in.stride + in.v_col + (size_t)h * Dv + col] : 0.f;
        }
    };
    auto keep_values = [&](int ci, const float (&v)[16 * C / THREADS]) {
#pragma unroll
        for (int e = 0; e < 16 * C / THREADS; ++e) v_s[ci & 1][(tid + e * THREADS) >> 4][(tid + e * THREADS) & 15] = v[e];
    };
    float next[16 * C / THREADS];
    values(0, next);
    keep_values(0, next);
    float2 S[TD / 2][TC];
#pragma unroll
    for (int i = 0; i < TD / 2; ++i)
#pragma unroll
        for (int c = 0; c < TC; ++c) S[i][c] = make_float2(0.f, 0.f);
    Decay product[HEAD ? 1 : TD];
    bool zero[HEAD ? 1 : TD] = {};
    __syncthreads();
    if (tid == 0)
        for (int i = 0; i < STAGES - 1 && i < chunks; ++i) fetch(i);
    bool ok = true, failed = false;
    int ci = 0;
    for (; ci < chunks; ++ci) {
        failed = ci > 0 && __syncthreads_or(!ok);              // all are done with chunk ci - 1, and its values are there
        if (failed) break;
        if (tid == 0 && ci + STAGES - 1 < chunks) fetch(ci + STAGES - 1);
        values(ci + 1, next);
        ok = tc::mbar_wait(&full[ci % STAGES], (ci / STAGES) & 1);
        const float* b = sm + (ci % STAGES) * PART;
        // As in the walk: earlier tokens by themselves, the decayed state, the last eight tokens on top.  A run's chunks are full.
        float2 N[TD / 2][TC];
#pragma unroll
        for (int i = 0; i < TD / 2; ++i)
#pragma unroll
            for (int c = 0; c < TC; ++c) N[i][c] = make_float2(0.f, 0.f);
#pragma unroll
        for (int s = 0; s < C; ++s) {
            if (s == C / 2) {
#pragma unroll
                for (int i = 0; i < TD / 4; ++i) {
                    float4 decay;
                    if (HEAD) decay.x = decay.y = decay.z = decay.w = b[KEYS + 2 * C];
                    else decay = *(const float4*)(b + KEYS + d0 + 4 * i);
                    if (!HEAD || i == 0) {
                        const float a[4] = {decay.x, decay.y, decay.z, decay.w};
#pragma unroll
                        for (int e = 0; e < (HEAD ? 1 : 4); ++e) {
                            product[4 * i + e].times(a[e]);
                            zero[4 * i + e] |= a[e] == 0.f;
                        }
                    }
#pragma unroll
                    for (int c = 0; c < TC; ++c) {
                        N[2 * i][c] = fma2(low2(decay), S[2 * i][c], N[2 * i][c]);
                        N[2 * i + 1][c] = fma2(high2(decay), S[2 * i + 1][c], N[2 * i + 1][c]);
                    }
                }
            }
            float2 v[TC];
            pairs(&v_s[ci & 1][s][cg * TC], v);
            if (HEAD) {
                const float gain = b[KEYS + C + s];
#pragma unroll
                for (int c = 0; c < TC; ++c) v[c] = mul2(v[c], make_float2(gain, gain));
            }
#pragma unroll
            for (int i = 0; i < TD / 4; ++i) {
                const float4 k1 = *(const float4*)(b + s * (DP + 4) + d0 + 4 * i);
#pragma unroll
                for (int c = 0; c < TC; ++c) {
                    N[2 * i][c] = fma2(low2(k1), v[c], N[2 * i][c]);
                    N[2 * i + 1][c] = fma2(high2(k1), v[c], N[2 * i + 1][c]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < TD / 2; ++i)
#pragma unroll
            for (int c = 0; c < TC; ++c) S[i][c] = N[i][c];
        keep_values(ci + 1, next);
    }
    if (!ok || failed) {                                       // the copies asked for are waited for (or given up)
        atomicOr(err, tc::KVB_DEV_TIMEOUT);
        if (failed && tid == 0)
            for (int i = ci - 1; i < chunks && i < ci + STAGES - 1; ++i) tc::mbar_wait(&full[i % STAGES], (i / STAGES) & 1);
        return;
    }
    const size_t place = (size_t)run.place * H + h;
    float* end = runs.starts + (place + H) * D * Dv;
#pragma unroll
    for (int i = 0; i < TD / 2; ++i)
#pragma unroll
        for (int c = 0; c < TC; ++c) {
            const int d = d0 + 2 * i;
            float* at = end + (size_t)d * Dv + col0 + c;
            if (d < D && col0 + c < Dv) at[0] = S[i][c].x;
            if (d + 1 < D && col0 + c < Dv) at[Dv] = S[i][c].y;
        }
    // A product that runs out of exponents is the smallest number there is, not zero, so that an infinite state stays infinite as in a
    // walk; zero only where a chunk's decay is zero.
    auto value = [&](int e) { return zero[e] ? product[e].value() : fmaxf(product[e].value(), 1.4e-45f); };
    if (HEAD) {
        if (blockIdx.x == 0 && tid == 0) runs.decays[place] = value(0);
    } else if (blockIdx.x == 0 && cg == 0) {
#pragma unroll
        for (int e = 0; e < TD; ++e) runs.decays[place * DP + d0 + e] = value(HEAD ? 0 : e);
    }
}

// grid (elements of a state in 256s, heads, segments): the states that a segment's runs start from.
template <bool HEAD, int DP>
__global__ void __launch_bounds__(256) run_starts_kernel(const Segments seg, const float* __restrict__ memory, int H, int D, int Dv, const Runs runs) {
    const int e = blockIdx.x * 256 + threadIdx.x, h = blockIdx.y, sg = blockIdx.z;
    const int count = runs_of(seg.q_len[sg], runs).count, d = e / Dv;
    if (e >= D * Dv || count <= 1) return;
    int first = 0;
    for (int s = 0; s < sg; ++s) {
        const int earlier = runs_of(seg.q_len[s], runs).count;
        first += earlier > 1 ? earlier : 0;
    }
    float S = memory[((size_t)seg.slot[sg] * H + h) * D * Dv + e];
    for (int k = 0; k < count; ++k) {
        const size_t place = (size_t)(first + k) * H + h;
        runs.starts[place * D * Dv + e] = S;
        if (k + 1 < count) S = fmaf(runs.decays[HEAD ? place : place * DP + d], S, runs.starts[(place + H) * D * Dv + e]);
    }
}

template <int MODE, int NI, int TD, int TC, int STAGES>
static int launch_walk(const Rows& in, const Segments& seg, const float* records, int first, int held, float q_scale, float* memory, float* out,
                       int H, int D, int Dv, const Runs& runs, int blocks_z, int* err, cudaStream_t stream) {
    constexpr int bytes = STAGES * record_of(MODE, 64 * NI).total * (int)sizeof(float);
    auto kernel = chunk_walk_kernel<MODE, NI, TD, TC, STAGES>;
    if (bytes > 16 * 1024) {                                   // (the kernel has shared memory of its own beside it)
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return (int)e;
    }
    // Not as a dependent launch: blocks placed while the records are still being made crowd onto the SMs that are free first, and
    // stay there (7 heads of 64 x 128, 2,048 tokens: 219 us against 112).
    kernel<<<dim3((Dv + 15) / 16, H, blocks_z), 16 * 64 * NI / (TD * TC), bytes, stream>>>(in, seg, records, first, held, q_scale, memory, out, H,
                                                                                          D, Dv, runs, err);
    return kvb_launch_status();
}

// The runs' starts: at most `count` runs of segments that have several.
template <int MODE, int NI, int TD, int TC, int STAGES>
static int launch_starts(const Rows& in, const Segments& seg, const float* records, int held, const float* memory, int H, int D, int Dv,
                         const Runs& runs, int count, int* err, cudaStream_t stream) {
    constexpr int bytes = STAGES * (C * (64 * NI + 4) + (MODE == CHUNK_HEAD_DECAY ? 3 * C : 64 * NI)) * (int)sizeof(float);
    auto kernel = chunk_ends_kernel<MODE, NI, TD, TC, STAGES>;
    if (bytes > 16 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return (int)e;
    }
    kernel<<<dim3((Dv + 15) / 16, H, count), 16 * 64 * NI / (TD * TC), bytes, stream>>>(in, seg, records, held, H, D, Dv, runs, err);
    run_starts_kernel<MODE == CHUNK_HEAD_DECAY, 64 * NI><<<dim3((D * Dv + 255) / 256, H, seg.count), 256, 0, stream>>>(seg, memory, H, D, Dv, runs);
    return kvb_launch_status();
}

// `held` chunks at a time, as many as `records` has room for; the states pass from one run of them to the next through `memory`.
template <int MODE, int NI>
static int run(const Rows& in, const Segments& seg, float* records, int total, int held, float q_scale, float* memory, float* out, int H, int D,
               int Dv, const Runs& runs, int run_count, int* err, cudaStream_t stream) {
    for (int first = 0; first < total; first += held) {
        const int count = min(held, total - first);
        if constexpr (MODE == CHUNK_HEAD_DECAY) {
            kvb_launch(head_records_kernel<NI>, dim3(count, H / in.qk_div), dim3(256), 0, stream, in, seg, records, first, held, H, D);
        } else {
            const int wide = ((D | in.stride | in.gate_stride | in.q_col | in.k_col) & 3) == 0 && (((uintptr_t)in.rows | (uintptr_t)in.gates) & 15) == 0;
            kvb_launch(chunk_records_kernel<MODE, NI>, dim3(count, H), dim3(256), 0, stream, in, seg, records, first, H, D, wide);
            if constexpr (MODE == CHUNK_DELTA_RULE)
                kvb_launch(chunk_solve_kernel<NI>, dim3(count, H), dim3(64 * NI), 0, stream, seg, records, first, H);
        }
        int rc = kvb_launch_status();
        if (rc != KVB_OK) return rc;
        // Key and value channels a thread holds: 4 x 2 of 64 (four warps), 8 x 2 of 128 (four warps).  Half of the warps with 4 x 4 or 8 x 2 of 64
        // take 16 to 35 % longer, 4 x 4 and 8 x 4 of 128 8 to 40 %, 8 x 1 30 to 50 %.
        if constexpr (!has_z(MODE))
            if (runs.wanted > 0) {                             // all chunks are held then (kvb_chunk_scan)
                rc = launch_starts<MODE, NI, 4 * NI, 2, 2>(in, seg, records, held, memory, H, D, Dv, runs, run_count, err, stream);
                if (rc != KVB_OK) return rc;
            }
        rc = launch_walk<MODE, NI, 4 * NI, 2, 2>(in, seg, records, first, held, q_scale, memory, out, H, D, Dv, runs,
                                                 runs.wanted > 0 ? run_count + seg.count : seg.count, err, stream);
        if (rc != KVB_OK) return rc;
    }
    return KVB_OK;
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
static int run(const Rows& in, const Segments& seg, float* records, int held, float q_scale, float* memory, float* out, int T, int H,
               int G, int D, int Dv, Runs runs, int run_count, int* err, cudaStream_t stream) {
    if (H < 1 || G < 1 || H % G || D < 1 || Dv < 1 || !rows_fit(MODE, in, H, G, D, Dv)) return KVB_ERR_SHAPE;
    if (seg.count <= 0 || T <= 0) return KVB_OK;
    if (records == nullptr) return KVB_ERR_SHAPE;
    if ((uintptr_t)records & 15) return KVB_ERR_ALIGN;
    if (D > 128 || H > 65535 || seg.count > 65535 || held < 1) return KVB_ERR_LIMIT;
    if (MODE == CHUNK_CHANNEL_DECAY && Dv > 512) return KVB_ERR_LIMIT;      // as the other forms of this scan
    const int total = T / C + seg.count;                       // no step has more chunks than this
    held = min(held, total);
    if (runs.wanted < 0 || (runs.wanted > 0 && (has_z(MODE) || held < total || !runs.starts || runs.least < 1 || runs.from < 0 || run_count < 1)))
        return KVB_ERR_SHAPE;
    if (runs.wanted > 0 && run_count > 65535 - seg.count) return KVB_ERR_LIMIT;
    runs.decays = runs.starts + (size_t)run_count * H * D * Dv;
    return D <= 64 ? run<MODE, 1>(in, seg, records, total, held, q_scale, memory, out, H, D, Dv, runs, run_count, err, stream)
                   : run<MODE, 2>(in, seg, records, total, held, q_scale, memory, out, H, D, Dv, runs, run_count, err, stream);
}

}  // namespace sc

// Floats of scratch a (chunk of 16 tokens, head) takes; mode 0 gated delta, 1 delta rule, 2 channel decay, 3 head decay.
KVB_API int kvb_chunk_record_floats(int mode, int D) {
    return mode < 0 || mode > 3 || D < 1 ? -1 : sc::record_of(mode, sc::padded(D)).total - sc::record_of(mode, sc::padded(D)).shared;
}
// ... and what a (chunk, group of heads that share q and k) takes besides.
KVB_API int kvb_chunk_shared_floats(int mode, int D) { return mode < 0 || mode > 3 || D < 1 ? -1 : sc::record_of(mode, sc::padded(D)).shared; }

// The scans over portions of prompts.  `rows` [T, stride] holds q, k and v at their columns (head h: number h / (H / G) of D for q and k,
// number h of Dv for v; H a multiple of G), `gates` [T, gate_stride] the mode's own numbers (sc::Rows); `records`: scratch of `held` times
// the floats above for all H heads and G groups, on 16 bytes: a step of more chunks (at most T / 16 + S) goes through it `held` chunks at a
// time, with the same results.  D up to 128.
// `wanted` runs a segment (0: one; modes 2 and 3, all chunks held): a segment of at least `run_from` chunks is cut into runs of
// max(run_least, ceil(its chunks / wanted)) of them, which are walked at once; `run_count`: no step of this kind has more runs of segments that have
// several; `starts`: scratch of run_count H (D Dv + D rounded up to 64) floats.
KVB_API int kvb_chunk_scan(int mode, const float* rows, int stride, int q_col, int k_col, int v_col, int G, const float* gates,
                           int gate_stride, float q_scale, const int* seg_q_start, const int* seg_q_len, const int* seg_slot, float* memory,
                           float* out, int T, int S, int H, int D, int Dv, int held, float* records, int* err, cudaStream_t stream, int wanted,
                           int run_least, int run_from, int run_count, float* starts) {
    const sc::Rows in = {rows, gates, stride, gate_stride, q_col, k_col, v_col, G > 0 ? H / G : 0};
    const sc::Segments seg = {seg_q_start, seg_q_len, seg_slot, S};
    const sc::Runs runs = {wanted, run_least, run_from, starts, nullptr};
#define KVB_SCAN(MODE) if (mode == MODE) return sc::run<MODE>(in, seg, records, held, q_scale, memory, out, T, H, G, D, Dv, runs, run_count, err, stream)
    KVB_SCAN(sc::CHUNK_GATED_DELTA);
    KVB_SCAN(sc::CHUNK_DELTA_RULE);
    KVB_SCAN(sc::CHUNK_CHANNEL_DECAY);
    KVB_SCAN(sc::CHUNK_HEAD_DECAY);
#undef KVB_SCAN
    return KVB_ERR_SHAPE;
}
