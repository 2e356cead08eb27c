// Causal attention for portions of prompts on the fifth-generation tensor cores (bfloat16; compiled per head size with
// -DKVB_HEAD_DIM=64 or 128): over cache pages, or (-DKVB_EXPANDED=1) over keys and values that lie in rows one after the
// other and whose last `rot` numbers all heads share.
//
// It computes what the reference's k_paged_attn computes (src/qwen_kernels.cu:146-185).
//
// A stream is two tiles of 128 query rows against the same keys: 256 rows of one head, or, where a segment has at most 128
// rows left, the rows of two heads that share keys.  Two groups of four softmax warps own a tile each, a thread a row:
//   S = Q K^T   tcgen05.mma, M 128 x N 128 keys x K head size; Q and the key tile in 128-byte-swizzled shared memory
//               (K-major), brought by TMA; S lands in tensor memory, 128 lanes x 128 columns for each tile of rows.
//   softmax     a thread reads its row of S, masks it (causal limit, window or chunk), keeps the running maximum and sum in
//               base 2 (the reference's recurrence, src/qwen_kernels.cu:159-176) and writes P = 2^(s - m) as bfloat16 over the
//               first half of the columns that held S.
//   O += P V    P is the A operand, read from tensor memory, the value tile as TMA left it - rows of keys, head size
//               contiguous - is the B operand in MN-major form; O stays in tensor memory for the whole stream.
// While one group's softmax runs, the tensor core multiplies P V and the next Q K^T of the other; the groups take turns at the
// exponentials.  Where a row's maximum grows, four more warps multiply its O by 2^(m_old - m_new) while P is being made: the next
// P V waits for both.  (Head size 64 leaves tensor memory for a P of its own, so the next S does not wait for P V there.)
// What bounds it: a tile of 128 x 128 needs the exponential unit (16 a clock and SM) for 1,024 clocks and the tensor core for 1,024
// at head size 128 (512 at 64), and a pair of them takes a block 3,700 (3,300): reads of S, the maximum and the way between
// barriers stand before and after the exponentials.  2,048 rows of 16 heads of 128 behind 30,000: 1,077 us with the kernel of units
// (csrc/attention_tc.cu: one tile of 128 rows a block, 64 keys at a time, O added up in registers), 488 here (1.07 PFLOP/s); behind
// 2,048: 150 and 76; 14 heads of 64: 443 and 315, 72 and 53.  A launch costs more than that kernel's (its code is met cold, 9,000
// clocks to the first scores, 2,000 for a piece's results, 7,000 where pieces are added), so short work stays there.
// Tried: two threads a row (640 us: what a thread waits for between barriers is paid four times a scheduler), no turns (598), P handed over
// in halves (548), exponentials on the FMA pipe by a polynomial for a quarter of the keys (no change: the unit is not what is waited for),
// O rescaled by the softmax warps only when a maximum had grown by 2^8 (475, but errors against 64 bits up to a fifth larger: P of
// the key with the maximum is then not 1 exactly).
//
// Errors against 64 bits (2-norms, results rounded to bfloat16; this kernel, that of units, mma.sync): 14 heads of 64 without a history 2.030e-3,
// 2.039e-3, 2.021e-3; behind 2,048 tokens 2.256, 2.222, 2.188; behind 16,000 2.322, 2.258, 2.258.  The weights' rounding makes them: of every piece of a
// stream the key with the maximum has the weight 1 exactly, and the other kernels cut long histories into more pieces (that of units with none cut: 2.261
// behind 2,048 and 2.314 behind 16,000).  (Sums in tensor
// memory cut off at 2^-24 a step: 1.9e-5 of a result after 16,384 keys, 5.6e-5 where all terms have one sign.)  Whole layers of attention: 1.0004 to
// 1.0013 times what they were before this kernel on average; of latent attention, expanded and not: 0.995 to 0.999 times.
//
// Work is shared out by key tiles: the streams' tiles, laid end to end, are cut into as many equal runs as there are blocks
// (one an SM), so that all finish together whatever the lengths.  A stream that a cut divides leaves (m, l, O) of its
// pieces in scratch, two places a block, and the last piece to finish adds them in order (a ticket per stream and tile).
// Every mbarrier wait is bounded; on a timeout the error word is set and the block winds down, the warps of a softmax group together.
#include "tc_common.cuh"

#ifndef KVB_HEAD_DIM
#error "compile with -DKVB_HEAD_DIM=64 or 128"
#endif
#ifndef KVB_EXPANDED
#define KVB_EXPANDED 0
#endif

namespace apr {
using namespace tc;

constexpr int D = KVB_HEAD_DIM;
static_assert(D == 64 || D == 128, "head size 64 or 128");
constexpr bool EXPANDED = KVB_EXPANDED != 0;
constexpr int BQ = 128, BK = 128;                    // query rows of a tile, keys of a tile
constexpr int VB = D / 64;                           // 64-wide (128-byte) column blocks of a value
constexpr int QB = VB + (EXPANDED ? 1 : 0);          // ... of a query and a key: the last one holds the shared rotated part
constexpr int BLOCK_BYTES = 128 * 128;               // a [128 rows x 64 columns] bfloat16 block, swizzled
constexpr int Q_BYTES = QB * BLOCK_BYTES, K_BYTES = QB * BLOCK_BYTES, V_BYTES = VB * BLOCK_BYTES;
constexpr int KST = D == 64 && !EXPANDED ? 3 : 2;    // key and value tiles in flight: two rings
constexpr int VST = D == 64 ? (EXPANDED ? 2 : 3) : (EXPANDED ? 1 : 2);
constexpr int TMEM_COLS = 512;                       // S: 2 x 128 columns, O: 2 x D columns; head size 64 has room for P: 2 x 64 columns
constexpr bool OWN_P = D == 64;                      // else P lies over the first half of S
// Warps 0-3 and 4-7: softmax rows of the two tiles; 8-11: rescaling of O; 12 and 14: the tiles' MMAs; 13: copies; 15: little.
constexpr int THREADS = 512;
// Registers a thread: the kernel is launched with 128 (65,536 / 512), of which the others give up what the softmax warps, which
// hold a row of 128 scores, take.
constexpr int SOFTMAX_REGS = 184, RESCALE_REGS = 72, HELPER_REGS = 72;
static_assert(2 * SOFTMAX_REGS + RESCALE_REGS + HELPER_REGS <= 4 * 128, "a split above the launch's registers would wait for good");
constexpr int MAX_TILES = EXPANDED ? 128 : 256;      // pairs of row tiles in a launch
constexpr float NEG_INF = -INFINITY;
// Work is shared out as if every stream had this many key tiles more: what a piece costs beside its tiles (Q, the first scores,
// the results), in tiles.
constexpr int STREAM_COST = 1;
constexpr int TURN_AT = D == 64 ? 64 : 96;            // the thirty-two keys after whose exponentials a group lets the other go on with its own

// 1 / (1 + e^-x), to about 2^-21 of itself; the gated result is rounded to 2^-9.  With expf and a division errors of latent layers against 64 bits are
// the same to 3e-5 of themselves either way (26 steps of 64 to 2,048 rows), and 2,048 rows take 161 us instead of 131 (code that is met cold).
__device__ __forceinline__ float sigmoid(float x) { return __fdividef(1.f, 1.f + ex2(-1.4426950408889634f * x)); }
// Two float32 numbers in one 64-bit register, and the multiply-add of such pairs (one instruction for two results).
__device__ __forceinline__ uint64_t pair(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpair(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// The maximum of a row of scores, over four chains: a maximum does not depend on the order.
__device__ __forceinline__ float row_max(const uint32_t* sv) {
    float mx[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) mx[e] = __uint_as_float(sv[e]);
#pragma unroll
    for (int e = 4; e + 7 < BK; e += 8)
#pragma unroll
        for (int c = 0; c < 4; ++c) mx[c] = max3(mx[c], __uint_as_float(sv[e + c]), __uint_as_float(sv[e + c + 4]));
#pragma unroll
    for (int c = 0; c < 4; ++c) mx[c] = fmaxf(mx[c], __uint_as_float(sv[BK - 4 + c]));
    return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// lo += v's lower bfloat16, hi += its upper one, in float32.
__device__ __forceinline__ void add_bf16x2(float& lo, float& hi, uint32_t v) {
    asm("{.reg .b16 x, y; mov.b32 {x, y}, %2; add.rn.f32.bf16 %0, x, %0; add.rn.f32.bf16 %1, y, %1;}" : "+f"(lo), "+f"(hi) : "r"(v));
}
// Whether all threads of a tile's four softmax warps say so: named barrier `id`.
__device__ __forceinline__ bool all_of_tile(int id, bool mine) {
    uint32_t all;
    __syncwarp();
    asm volatile("{.reg .pred p, q; setp.ne.u32 p, %2, 0; bar.red.and.pred q, %1, 128, p; selp.u32 %0, 1, 0, q;}" : "=r"(all) : "r"(id), "r"((uint32_t)mine) : "memory");
    return all != 0;
}
// The lowest `count` bits (none below 0, all from 32).
__device__ __forceinline__ uint32_t below(int count) { return count >= 32 ? 0xffffffffu : count <= 0 ? 0u : (1u << count) - 1u; }

struct Params {
    bf16* out;                 // [T, Hq * D]
    const int* tiles;          // [n_tiles, 2]: segment, first row of the pair of row tiles
    int n_tiles;
    const int* seg_q_start;
    const int* seg_q_len;
    const int* seg_kv_len;
    const int* block_table;    // [segments, table_stride]
    int table_stride, page_size, page_shift;
    const int* seg_key_row;    // expanded: where key 0 of a segment would lie among the rows of keys
    int rot_steps;             // expanded: the shared part's numbers, in sixteens
    int q_head;                // columns of a head in q
    float* part_o;             // [2 * blocks, 2, D / 4, 128, 4]  unnormalised outputs of pieces of divided streams
    float* part_ml;            // [2 * blocks, 2, 128, 2]  their running maximum and sum
    int* tickets;              // [n_tiles, Hq, 2], zero between launches
    int Hq, Hkv, window;
    float scale_log2;
    int* err;
    const float* sink;         // [Hq] or nullptr: a key without a value in every row's softmax, its score sink[head] (natural units, not scaled)
    int keep;                  // with a window: the request's first `keep` keys stay visible
    // [Hq] or nullptr: with slopes, a score is cap tanh(scale q.k / cap) (cap 0: scale q.k) minus slopes[head] (p - j) for a key p - j back.
    const float* slopes;
    float cap, scale;
    int min_tiles;             // a block takes at least this many key tiles, unless there are fewer
    // Expanded: the result is multiplied by sigmoid(gate[row, gate_col + ...]) (one number a value channel, or one a head).
    const bf16* gate;
    int gate_stride, gate_col, gate_per_head;
};

// Results go out through 32 rows x 64 bytes of shared memory a warp, so that a store covers whole stretches of rows: straight from
// the threads, a row each, 32 lines a store, they took the SM 4,000 clocks a stream.  Where tiles leave no room, the place of
// the rows' Q serves (and the next Q waits for it).
constexpr bool STAGE_IN_Q = EXPANDED;
constexpr int STAGE_BYTES = 32 * 64;
struct Shared {
    uint64_t q_full[2], q_free[2], k_full[KST], k_free[KST], v_full[VST], v_free[VST], s_full[2], s_read[2], p_ready[2], o_full[2], turn[2], top_known[2];
    uint32_t tmem_base;
    int failed;
    int k_copies, v_copies, q_copies[2];   // tiles asked for, as the copying warp leaves them
    int ticket[2];
    float corr[2][BQ];         // what a row's O is multiplied by before the next P V
    int first[MAX_TILES + 1];  // the line of work - every stream's cost and key tiles, one after the other - before this pair of row tiles
};

constexpr int STAGE_AT = 2 * Q_BYTES + KST * K_BYTES + VST * V_BYTES;
constexpr int TILES_BYTES = STAGE_AT + (STAGE_IN_Q ? 0 : 8 * STAGE_BYTES), SMEM_BYTES = TILES_BYTES + (int)sizeof(Shared);
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one block");

// What a pair of row tiles of a segment sees.
struct Tile {
    int seg, row0, rows, pos_first;
    int key_lo, tile_begin, n_keep, keep, n;         // the list of key tiles: n_keep tiles of kept keys, then the window's
    int streams;                                     // heads, or pairs of heads where the second tile of rows would be empty
    bool two_heads;
};
__device__ __forceinline__ Tile make_tile(const Params& p, int t) {
    Tile c;
    c.seg = p.tiles[2 * t];
    c.row0 = p.tiles[2 * t + 1];
    const int q_len = p.seg_q_len[c.seg];
    c.rows = min(2 * BQ, q_len - c.row0);
    c.pos_first = p.seg_kv_len[c.seg] - q_len + c.row0;
    c.key_lo = first_seen_key(c.pos_first, p.window);
    c.keep = p.window > 0 ? p.keep : 0;
    c.tile_begin = c.key_lo / BK;
    c.n_keep = min((c.keep + BK - 1) / BK, c.tile_begin);
    c.n = c.n_keep + (c.pos_first + c.rows - 1) / BK + 1 - c.tile_begin;
    const int group = p.Hq / p.Hkv;
    c.two_heads = !EXPANDED && c.rows <= BQ && group > 1;
    c.streams = c.two_heads ? p.Hkv * ((group + 1) / 2) : p.Hq;
    return c;
}

// A run of a stream's key tiles, for one block; `half` is a tile of 128 rows of the two.
struct Piece {
    int begin, end;            // places in the stream's list of key tiles (none: the block's run ends before the stream's first)
    int first, next;           // where the stream's first key tile lies in the line, and where the block's next piece starts
    int index;                 // the stream's number within its pair of row tiles
    int hk;                    // key/value head
};
__device__ __forceinline__ Piece make_piece(const Params& p, const Tile& c, int tile_first, int w, int w_end) {
    Piece x;
    const int off = w - tile_first;
    x.index = off / (c.n + STREAM_COST);
    const int at = off - x.index * (c.n + STREAM_COST), to = min(c.n + STREAM_COST, at + w_end - w);
    x.first = w - at + STREAM_COST;
    x.next = w + to - at;
    x.begin = max(0, at - STREAM_COST);
    x.end = max(x.begin, to - STREAM_COST);
    const int group = p.Hq / p.Hkv;
    x.hk = c.two_heads ? x.index / ((group + 1) / 2) : x.index / group;
    return x;
}
struct Half {
    int head, row0, rows;      // rows 0: the second of two heads of an odd group, or rows beyond the segment
    int limit;                 // places of the list that any of its rows sees
    int n;                     // key tiles of the piece
};
__device__ __forceinline__ Half make_half(const Params& p, const Tile& c, const Piece& x, int half) {
    Half h;
    if (c.two_heads) {
        const int group = p.Hq / p.Hkv, in_group = 2 * (x.index - x.hk * ((group + 1) / 2)) + half;
        h.head = x.hk * group + in_group;
        h.row0 = c.row0;
        h.rows = in_group < group ? c.rows : 0;
    } else {
        h.head = x.index;
        h.row0 = c.row0 + half * BQ;
        h.rows = max(0, min(BQ, c.rows - half * BQ));
    }
    const int pos_last = c.pos_first + (h.row0 - c.row0) + h.rows - 1;
    h.limit = h.rows > 0 ? c.n_keep + pos_last / BK + 1 - c.tile_begin : 0;
    h.n = max(0, min(x.end, h.limit) - x.begin);
    return h;
}

__global__ void __launch_bounds__(THREADS, 1)
attention_pairs_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ Params p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];   // the kernel has no other shared memory: the swizzle's alignment costs none
    unsigned char* q_s = smem_raw;                                // tile of rows h at q_s + h Q_BYTES
    unsigned char* k_s = q_s + 2 * Q_BYTES;                   // key stage s at k_s + s K_BYTES
    unsigned char* v_s = k_s + KST * K_BYTES;                 // value stage s at v_s + s V_BYTES
    Shared& sh = *reinterpret_cast<Shared*>(smem_raw + TILES_BYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (smem_u32(smem_raw) & 1023) {                          // not on this toolchain and GPU
        if (tid == 0) atomicOr(p.err, KVB_DEV_TIMEOUT);
        return;
    }
    if (tid == 0) {
        for (int h = 0; h < 2; ++h) {
            mbar_init(&sh.q_full[h], 1); mbar_init(&sh.q_free[h], STAGE_IN_Q ? 5 : 1);
            mbar_init(&sh.s_full[h], 1); mbar_init(&sh.s_read[h], 4); mbar_init(&sh.o_full[h], 1);
            mbar_init(&sh.p_ready[h], 8); mbar_init(&sh.turn[h], 4); mbar_init(&sh.top_known[h], 4);
        }
        for (int s = 0; s < KST; ++s) { mbar_init(&sh.k_full[s], 1); mbar_init(&sh.k_free[s], 2); }
        for (int s = 0; s < VST; ++s) { mbar_init(&sh.v_full[s], 1); mbar_init(&sh.v_free[s], 2); }
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sh.tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (warp == 15 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_q) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_k) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_v) : "memory");
    }
    if (warp == 13) {
        // Key tiles before every pair of row tiles.  The step's metadata was written at its start, so none of this waits
        // for the kernel before.
        int before = 0;
        for (int t0 = 0; t0 < p.n_tiles; t0 += 32) {
            int mine = 0;
            if (t0 + lane < p.n_tiles) { const Tile c = make_tile(p, t0 + lane); mine = (c.n + STREAM_COST) * c.streams; }
            int sum = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const int up = __shfl_up_sync(0xffffffffu, sum, d); if (lane >= d) sum += up; }
            if (t0 + lane < p.n_tiles) sh.first[t0 + lane] = before + sum - mine;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) sh.first[p.n_tiles] = before;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_s = sh.tmem_base, tmem_o = sh.tmem_base + 2 * BK;      // S of tile h at + 128 h, O at + D h

    const int total = sh.first[p.n_tiles];
    const int share = max(p.min_tiles, (total + (int)gridDim.x - 1) / (int)gridDim.x);
    const int w_begin = (int)min((long long)total, (long long)blockIdx.x * share), w_end = min(total, w_begin + share);
    int t = 0;
    for (int hi = p.n_tiles; hi - t > 1;) { const int mid = (t + hi) >> 1; if (sh.first[mid] <= w_begin) t = mid; else hi = mid; }

    // Every role walks the block's pieces by itself; barrier phases and stages go by counts that run on from piece to piece.
    if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(HELPER_REGS));
    if (warp == 13) {
        // ---- copies: Q of the two tiles of rows, key and value tiles, page by page; lane i copies page i ----
        const int pages = EXPANDED ? 1 : BK >> p.page_shift;
        bool ok = true, waited = false;
        int count = 0, k_copies = 0, v_copies = 0, q_count[2] = {0, 0};
        for (int w = w_begin; w < w_end && ok;) {
            while (sh.first[t + 1] <= w) ++t;
            const Tile c = make_tile(p, t);
            const Piece x = make_piece(p, c, sh.first[t], w, w_end);
            w = x.next;
            const int n = x.end - x.begin;
            if (n == 0) continue;
            const int pos_last = c.pos_first + c.rows - 1;
            const int* table = p.block_table + (size_t)c.seg * p.table_stride;
            // Lane i's page of place x.begin + j, looked up one tile before it is wanted.  Where the rows can see none of a
            // page's keys, or the table holds none, the copy is aimed before the pool's first row: the TMA unit fills what
            // lies outside the tensor with zeros (0 * NaN would poison the sums) and still counts the bytes.
            auto key_of = [&](int j) -> int { const int i = x.begin + j; return (i < c.n_keep ? i : c.tile_begin - c.n_keep + i) * BK; };
            auto lookup = [&](int j) -> int {
                int page = -1;
                if (!EXPANDED && lane < pages && j < n) {
                    const int first_key = key_of(j) + lane * p.page_size;
                    if (first_key <= pos_last && (first_key + p.page_size > c.key_lo || first_key < c.keep)) page = table[first_key >> p.page_shift];
                }
                return page;
            };
            int page_next = lookup(0);
            // Everything up to here is the step's metadata, which the host wrote at its start.
            if (!waited) { waited = true; pdl_wait(); pdl_launch_dependents(); }
            for (int j = 0; j < n && ok; ++j, ++count) {
                const int page = page_next;
                page_next = lookup(j + 1);
                const int ks = count % KST, vs = count % VST;
                const int row = EXPANDED ? p.seg_key_row[c.seg] + key_of(j) : page >= 0 ? (page * p.Hkv + x.hk) * p.page_size : -p.page_size;
                if (count >= KST) ok = mbar_wait(&sh.k_free[ks], ((count / KST) - 1) & 1);
                if (!ok) break;
                ++k_copies;
                if (lane == 0) mbar_expect_tx(&sh.k_full[ks], K_BYTES);
                __syncwarp();
                if constexpr (EXPANDED) {
                    // Columns of the rows: [keys of all heads | values of all heads]; the shared part has a map of its own.
                    if (lane < VB) tma_load_2d(k_s + (size_t)ks * K_BYTES + lane * BLOCK_BYTES, &map_k, x.hk * D + lane * 64, row, &sh.k_full[ks]);
                    if (lane == VB) tma_load_2d(k_s + (size_t)ks * K_BYTES + VB * BLOCK_BYTES, &map_v, 0, row, &sh.k_full[ks]);
                } else if (lane < pages) {
#pragma unroll
                    for (int b = 0; b < VB; ++b)
                        tma_load_2d(k_s + (size_t)ks * K_BYTES + b * BLOCK_BYTES + lane * p.page_size * 128, &map_k, b * 64, row, &sh.k_full[ks]);
                }
                if (j == 0) {
                    for (int h = 0; h < 2 && ok; ++h) {
                        const Half half = make_half(p, c, x, h);
                        if (half.n == 0) continue;
                        if (q_count[h] > 0) ok = mbar_wait(&sh.q_free[h], (q_count[h] - 1) & 1);
                        if (!ok) break;
                        ++q_count[h];
                        if (lane == 0) mbar_expect_tx(&sh.q_full[h], Q_BYTES);
                        __syncwarp();
                        if (lane < QB)
                            tma_load_2d(q_s + h * Q_BYTES + lane * BLOCK_BYTES, &map_q, half.head * p.q_head + lane * 64, p.seg_q_start[c.seg] + half.row0, &sh.q_full[h]);
                    }
                    if (!ok) break;
                }
                if (count >= VST) ok = mbar_wait(&sh.v_free[vs], ((count / VST) - 1) & 1);
                if (!ok) break;
                ++v_copies;
                if (lane == 0) mbar_expect_tx(&sh.v_full[vs], V_BYTES);
                __syncwarp();
                if constexpr (EXPANDED) {
                    if (lane < VB) tma_load_2d(v_s + (size_t)vs * V_BYTES + lane * BLOCK_BYTES, &map_k, (p.Hq + x.hk) * D + lane * 64, row, &sh.v_full[vs]);
                } else if (lane < pages) {
#pragma unroll
                    for (int b = 0; b < VB; ++b)
                        tma_load_2d(v_s + (size_t)vs * V_BYTES + b * BLOCK_BYTES + lane * p.page_size * 128, &map_v, b * 64, row, &sh.v_full[vs]);
                }
            }
        }
        if (!ok && lane == 0) { atomicOr(p.err, KVB_DEV_TIMEOUT); sh.failed = 1; }
        if (lane == 0) { sh.k_copies = k_copies; sh.v_copies = v_copies; sh.q_copies[0] = q_count[0]; sh.q_copies[1] = q_count[1]; }
        __syncwarp();
    } else if (warp == 12 || warp == 14) {
        // ---- products, a warp for each tile of rows.  Every lane waits on the barriers (a wait by one lane and a broadcast
        // costs twice as much), the first issues.  Where P lies over S, P V of a tile goes out before the next Q K^T into the
        // same columns: the tensor core takes one thread's products in their order. ----
        constexpr uint32_t idesc_s = instr_desc(BQ, BK);
        constexpr uint32_t idesc_o = instr_desc(BQ, D) | (1u << 16);            // B (values) is MN-major
        const int h = warp == 12 ? 0 : 1;
        const int k_steps = D / 16 + (EXPANDED ? p.rot_steps : 0);
        const uint32_t my_s = tmem_s + h * BK, my_p = OWN_P ? tmem_o + 2 * D + h * (BK / 2) : my_s, my_o = tmem_o + h * D;
        bool ok = true;
        int count = 0, s_count = 0, q_count = 0;
        for (int w = w_begin; w < w_end && ok;) {
            while (sh.first[t + 1] <= w) ++t;
            const Tile c = make_tile(p, t);
            const Piece x = make_piece(p, c, sh.first[t], w, w_end);
            w = x.next;
            const int n = x.end - x.begin, nh = make_half(p, c, x, h).n;
            if (n == 0) continue;
            // S = Q K_j^T, or only the word that this warp has no use for K_j.
            auto scores = [&](int j) {
                const int ks = (count + j) % KST;
                if (OWN_P || j == 0 || j >= nh) ok = ok && mbar_wait(&sh.k_full[ks], ((count + j) / KST) & 1);   // else it has been waited for
                if (ok && lane == 0) {
                    if (j < nh) {
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        const uint32_t q_addr = smem_u32(q_s + h * Q_BYTES), k_addr = smem_u32(k_s + (size_t)ks * K_BYTES);
#pragma unroll
                        for (int k = 0; k < QB * 4; ++k)              // 16 numbers of the head a step; 64 a block
                            if (!EXPANDED || k < k_steps)
                                umma(my_s, smem_desc(q_addr + (k / 4) * BLOCK_BYTES) + 2 * (k % 4),
                                     smem_desc(k_addr + (k / 4) * BLOCK_BYTES) + 2 * (k % 4), idesc_s, k != 0 ? 1u : 0u);
                        umma_commit(&sh.s_full[h]);
                        if (j + 1 == nh) umma_commit(&sh.q_free[h]);
                        umma_commit(&sh.k_free[ks]);
                    } else {
                        mbar_arrive(&sh.k_free[ks]);
                    }
                }
                __syncwarp();
            };
            if (nh > 0) { ok = mbar_wait(&sh.q_full[h], q_count & 1); ++q_count; }
            scores(0);
            for (int j = 0; j < n && ok; ++j) {
                const int vs = (count + j) % VST;
                if (j >= nh) {
                    ok = mbar_wait(&sh.v_full[vs], ((count + j) / VST) & 1);
                    if (ok && lane == 0) mbar_arrive(&sh.v_free[vs]);
                    __syncwarp();
                    if (j + 1 < n) scores(j + 1);
                    continue;
                }
                if (OWN_P && j + 1 < n) {                              // the scores are in registers: the next ones may come
                    ok = mbar_wait(&sh.s_read[h], s_count & 1);
                    scores(j + 1);
                }
                // What is mostly there already is asked for first: nothing but P is then waited for on the way to the products.
                ok = ok && mbar_wait(&sh.v_full[vs], ((count + j) / VST) & 1);
                if (!OWN_P && j + 1 < n) ok = ok && mbar_wait(&sh.k_full[(count + j + 1) % KST], ((count + j + 1) / KST) & 1);
                ok = ok && mbar_wait(&sh.p_ready[h], s_count & 1);
                if (ok && lane == 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t v_addr = smem_u32(v_s + (size_t)vs * V_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)                  // 16 keys a step: 8 columns of P in tensor memory, 2048 bytes down V
                        umma_a_tmem(my_o, my_p + 8 * k, smem_desc_mn(v_addr + k * 2048, BLOCK_BYTES), idesc_o, (j != 0 || k != 0) ? 1u : 0u);
                    if (OWN_P || j + 1 == nh) umma_commit(&sh.o_full[h]);
                    umma_commit(&sh.v_free[vs]);
                }
                __syncwarp();
                ++s_count;
                if (!OWN_P && j + 1 < n) scores(j + 1);
            }
            count += n;
        }
        if (!ok && lane == 0) { atomicOr(p.err, KVB_DEV_TIMEOUT); sh.failed = 1; }
        __syncwarp();
    }
    } else if (warp >= 8) {
        // ---- O of a tile is multiplied by 2^(m_old - m_new) where a row's maximum has grown, while the softmax warps make P by
        // the new maximum.  P of the key with the maximum is then 1 exactly; with O rescaled only when the maximum had grown
        // by 2^8 the result's error against 64 bits was up to a fifth larger. ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(RESCALE_REGS));
        const int row = tid & 127;
        const uint32_t my_o = tmem_o + ((uint32_t)((warp & 3) * 32) << 16);
        bool ok = true;
        int count[2] = {0, 0};
        for (int w = w_begin; w < w_end && ok;) {
            while (sh.first[t + 1] <= w) ++t;
            const Tile c = make_tile(p, t);
            const Piece x = make_piece(p, c, sh.first[t], w, w_end);
            w = x.next;
            const int nh[2] = {make_half(p, c, x, 0).n, make_half(p, c, x, 1).n};
            for (int i = 0; i < max(nh[0], nh[1]) && ok; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!ok || i >= nh[h]) continue;
                    ok = mbar_wait(&sh.top_known[h], count[h] & 1);
                    ++count[h];
                    const float corr = sh.corr[h][row];
                    // O holds all earlier tiles and is not being added to: where P lies over S, the S that the maximum is from
                    // was asked for after the P V before it; else the softmax warps have waited for that product.
                    if (i > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
                        for (int d = 0; d < D; d += 32) {
                            uint32_t r[32];
                            tmem_ld32(my_o + h * D + d, r);
#pragma unroll
                            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * corr);
                            tmem_st16(my_o + h * D + d, r);
                            tmem_st16(my_o + h * D + d + 16, r + 16);
                        }
                        tmem_st_wait();
                        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.p_ready[h]);
                }
        }
        if (!ok && lane == 0) { atomicOr(p.err, KVB_DEV_TIMEOUT); sh.failed = 1; }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(SOFTMAX_REGS));
        pdl_wait();                                                 // results and scratch: the kernels before may still read theirs
        pdl_launch_dependents();
        // ---- softmax: warps 0-3 the first tile of rows, 4-7 the second; thread = row ----
        const int wg = warp >> 2, row = tid & 127;
        const uint32_t lane_base = ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t my_s = tmem_s + wg * BK + lane_base, my_o = tmem_o + wg * D + lane_base;
        const uint32_t my_p = OWN_P ? tmem_o + 2 * D + wg * (BK / 2) + lane_base : my_s;
        bool ok = true;
        int s_count = 0, pieces = 0, turns = 0;
        for (int w = w_begin; w < w_end && ok;) {
            while (sh.first[t + 1] <= w) ++t;
            const Tile c = make_tile(p, t);
            const Piece x = make_piece(p, c, sh.first[t], w, w_end);
            w = x.next;
            const Half hf = make_half(p, c, x, wg);
            if (hf.n == 0) continue;
            const int both = min(hf.n, make_half(p, c, x, wg ^ 1).n);      // tiles that the two groups take in turns
            const int h = hf.head;
            const int pos = row < hf.rows ? c.pos_first + (hf.row0 - c.row0) + row : -1;
            const int lo = first_seen_key(pos, p.window);           // the first key the row sees
            // The row's running maximum and sum.
            float m = NEG_INF, l = 0.f;
            if (p.sink && x.begin == 0) { m = p.sink[h] * 1.4426950408889634f; l = 1.f; }   // the sink, once per row: in its first piece
            for (int i = 0; i < hf.n; ++i, ++s_count) {
                ok = mbar_wait(&sh.s_full[wg], s_count & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const int place = x.begin + i, key0 = (place < c.n_keep ? place : c.tile_begin - c.n_keep + place) * BK;
                // Whether every row of this warp sees every key of the tile (then no element needs its mask).
                const bool open = pos >= 0 && key0 + BK - 1 <= pos && key0 >= lo;
                const bool warp_open = __all_sync(0xffffffffu, open);
                const bool biased = !EXPANDED && p.slopes;
                const float scale_log2 = biased ? 1.f : p.scale_log2;
                if (biased || !warp_open) {
                    // Scores that are not used as they are go back to tensor memory once they are made, 32 at a time in a loop
                    // that is not unrolled, as is all that a tile or a stream does once: a launch finds the instruction cache
                    // cold and pays about six clocks for every instruction it meets for the first time.
                    const float slope = biased ? p.slopes[h] : 0.f, inv_cap = p.cap > 0.f ? 1.f / p.cap : 0.f;
#pragma unroll 1
                    for (int e0 = 0; e0 < BK; e0 += 32) {
                        // Bit e: key k0 + e is seen - up to the row's position, and from the window's first key or among the kept.
                        const int k0 = key0 + e0;
                        const uint32_t seen = below(pos + 1 - k0) & (~below(lo - k0) | below(c.keep - k0));
                        if (!biased && __all_sync(0xffffffffu, seen == 0xffffffffu)) continue;
                        uint32_t r[32];
                        tmem_ld32(my_s + e0, r);
                        if (biased) {
                            // Capped and biased scores: the whole score is made here, in base-2 units, and the exponent multiplies
                            // by 1.  tanh by one exponential, 1 - 2 / (1 + e^{2 y}): exact at both ends, absolute error about 1e-7.
#pragma unroll
                            for (int e = 0; e < 32; ++e) {
                                float v = __uint_as_float(r[e]) * p.scale;
                                if (p.cap > 0.f) v = p.cap * (1.f - __fdividef(2.f, 1.f + ex2(v * inv_cap * 2.885390081777927f)));
                                r[e] = __float_as_uint((v - slope * (float)(pos - k0 - e)) * 1.4426950408889634f);
                            }
                        }
#pragma unroll
                        for (int e = 0; e < 32; ++e)
                            if (!((seen >> e) & 1u)) r[e] = __float_as_uint(NEG_INF);
                        tmem_st16(my_s + e0, r);
                        tmem_st16(my_s + e0 + 16, r + 16);
                    }
                    tmem_st_wait();
                }
                uint32_t sv[BK];
#pragma unroll
                for (int e = 0; e < BK; e += 32) tmem_ld32_nowait(my_s + e, sv + e);
                tmem_ld_wait();
                if (OWN_P) {                                          // S is in registers
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.s_read[wg]);
                }
                const float top = fmaxf(m, row_max(sv) * scale_log2);
                if (OWN_P && s_count > 0) ok = ok && mbar_wait(&sh.o_full[wg], (s_count - 1) & 1);    // the product that reads the P before
                const float corr = ex2(m - (top == NEG_INF ? 0.f : top));
                m = top;
                l *= corr;
                sh.corr[wg][row] = corr;
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.top_known[wg]);
                // P = 2^(s * scale - m) as bfloat16: keys 2c and 2c + 1 of the row in column c.  A masked score is -inf and gives
                // 0.  The sum is taken of the rounded numbers, in float32 over four chains: the weights that V gets then add up to 1 (from the
                // unrounded ones errors against 64 bits were up to 1 % larger, where few keys take most of the weight).
                const float base_m = m == NEG_INF ? 0.f : m;
                const uint64_t scale2 = pair(scale_log2, scale_log2), minus2 = pair(-base_m, -base_m);
                float l4[4] = {0.f, 0.f, 0.f, 0.f};
                // The groups take turns at the exponentials: side by side each would take twice as long, and both would then want
                // the tensor core at once and leave the exponentials idle meanwhile.
                // From the block's first turn to its last, across pieces: a group that ran ahead of the other by a piece of one tile
                // would pass its turn on twice before the other had looked.
                if (i < both) {
                    if (wg == 1 || turns > 0) ok = ok && mbar_wait(&sh.turn[wg], (turns - (wg ^ 1)) & 1);
                    ++turns;
                }
#pragma unroll
                for (int e0 = 0; e0 < BK; e0 += 32) {
                    uint32_t packed[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const float2 y = unpair(fma2(pair(__uint_as_float(sv[e0 + 2 * e]), __uint_as_float(sv[e0 + 2 * e + 1])), scale2, minus2));
                        const float p0 = ex2(y.x), p1 = ex2(y.y);
                        __nv_bfloat162 v = __floats2bfloat162_rn(p0, p1);
                        packed[e] = *reinterpret_cast<uint32_t*>(&v);
                        add_bf16x2(l4[(2 * e) & 3], l4[(2 * e + 1) & 3], packed[e]);
                    }
                    tmem_st16(my_p + e0 / 2, packed);
                    if (e0 == TURN_AT) {
                        __syncwarp();
                        if (lane == 0 && i < both) mbar_arrive(&sh.turn[wg ^ 1]);
                    }
                }
                l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
                tmem_st_wait();
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.p_ready[wg]);
                if (!ok) break;
            }
            // The blocks whose runs hold a part of what these rows see of the stream.
            const int block0 = x.first / share, block1 = (x.first + hf.limit - 1) / share;
            int* ticket = p.tickets + ((size_t)t * p.Hq + x.index) * 2 + wg;
            if (EXPANDED && pos >= 0) {                               // the row's gates, while the last product runs
                const bf16* g = p.gate + (size_t)(p.seg_q_start[c.seg] + hf.row0 + row) * p.gate_stride + p.gate_col + (p.gate_per_head ? h : h * D);
                for (int d = 0; d < (p.gate_per_head ? 1 : D); d += 64) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(g + d));
            }
            ok = ok && mbar_wait(&sh.o_full[wg], (OWN_P ? s_count - 1 : pieces) & 1);
            // All four warps have handed over P of this piece, so none still looks at the word of the piece before.
            if (ok && block0 != block1 && row == 0) sh.ticket[wg] = *reinterpret_cast<volatile int*>(ticket);
            // The tile's warps give up together: one whose wait ran out comes here as well, and only here do they leave the line of work, so
            // that none is left alone at one of the barriers below, which have no limit.
            ok = all_of_tile(1 + wg, ok);
            if (!ok) break;
            ++pieces;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");

            const int q_row0 = p.seg_q_start[c.seg] + hf.row0, q_row = q_row0 + row;
            unsigned char* stage = STAGE_IN_Q ? q_s + wg * Q_BYTES + (warp & 3) * STAGE_BYTES : smem_raw + STAGE_AT + warp * STAGE_BYTES;
            // 32 results of the row from column d.  The warp's rows go into its stage, 16 bytes at a time, in an order that spreads
            // the banks, and out of it with four lanes a row.
            auto store32 = [&](int d, float* f) {
                if (EXPANDED && pos >= 0) {
                    const bf16* g = p.gate + (size_t)q_row * p.gate_stride + p.gate_col + (p.gate_per_head ? h : h * D + d);
                    if (p.gate_per_head) {
                        const float s = sigmoid(__bfloat162float(g[0]));
#pragma unroll
                        for (int e = 0; e < 32; ++e) f[e] *= s;
                    } else {                                          // rows that start on 16 bytes
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const uint4 v = *reinterpret_cast<const uint4*>(g + 8 * q);
                            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                f[8 * q + e] *= sigmoid(__uint_as_float(e & 1 ? u[e / 2] & 0xffff0000u : u[e / 2] << 16));
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t w4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        __nv_bfloat162 v = __floats2bfloat162_rn(f[8 * q + 2 * e], f[8 * q + 2 * e + 1]);
                        w4[e] = *reinterpret_cast<uint32_t*>(&v);
                    }
                    *reinterpret_cast<uint4*>(stage + lane * 64 + ((q ^ (lane >> 1)) & 3) * 16) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                }
                __syncwarp();
#pragma unroll
                for (int r0 = 0; r0 < 32; r0 += 8) {
                    const int r = r0 + (lane >> 2), q = lane & 3, tile_row = (warp & 3) * 32 + r;
                    const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 64 + ((q ^ (r >> 1)) & 3) * 16);
                    if (tile_row < hf.rows) *reinterpret_cast<uint4*>(p.out + ((size_t)(q_row0 + tile_row) * p.Hq + h) * D + d + 8 * q) = v;
                }
            };
            if (block0 == block1) {
                const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
                for (int d = 0; d < D; d += 32) {
                    uint32_t r[32];
                    tmem_ld32(my_o + d, r);
                    float f[32];
#pragma unroll
                    for (int e = 0; e < 32; ++e) f[e] = __uint_as_float(r[e]) * inv;
                    store32(d, f);
                }
            } else {
                auto place_of = [&](int b) -> size_t { return (size_t)(2 * b + (b * share > x.first ? 0 : 1)) * 2 + wg; };
                // Whether all other pieces have left their sums already: then this one's need not be written down.
                bool last = sh.ticket[wg] == block1 - block0;
                if (!last) {
                    // Leave this piece's (m, l, O), [D / 4][128 rows] of float4, so that a warp's rows make one contiguous store.
                    const size_t mine = place_of(blockIdx.x);
                    float4* po = reinterpret_cast<float4*>(p.part_o + mine * BQ * D) + row;
#pragma unroll 1
                    for (int d = 0; d < D; d += 64) {
                        uint32_t r[64];
                        tmem_ld32_nowait(my_o + d, r);
                        tmem_ld32_nowait(my_o + d + 32, r + 32);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 64; e += 4)
                            po[((d + e) / 4) * BQ] = make_float4(__uint_as_float(r[e]), __uint_as_float(r[e + 1]), __uint_as_float(r[e + 2]), __uint_as_float(r[e + 3]));
                    }
                    *reinterpret_cast<float2*>(p.part_ml + (mine * BQ + row) * 2) = make_float2(m, l);
                    __threadfence();
                    asm volatile("bar.sync %0, 128;\n" ::"r"(1 + wg) : "memory");
                    if (row == 0) sh.ticket[wg] = atomicAdd(ticket, 1);
                    asm volatile("bar.sync %0, 128;\n" ::"r"(1 + wg) : "memory");
                    last = sh.ticket[wg] == block1 - block0;
                }
                if (last) {
                    // The last piece to finish adds all of them in order, its own from tensor memory: the same numbers in the same
                    // order whichever is last.  weight_s = 2^(m_s - M) / sum_s 2^(m_s - M) l_s, out = sum_s weight_s O_s.
                    __threadfence();
                    if (row == 0) *ticket = 0;
                    const int me = blockIdx.x;
                    auto ml_of = [&](int b) -> float2 {
                        return b == me ? make_float2(m, l) : __ldcg(reinterpret_cast<const float2*>(p.part_ml + (place_of(b) * BQ + row) * 2));
                    };
                    float M = NEG_INF, L = 0.f;                    // L belongs to the scale M throughout
                    for (int b0 = block0; b0 <= block1; b0 += 4) {
                        float2 v[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) v[k] = b0 + k <= block1 ? ml_of(b0 + k) : make_float2(NEG_INF, 0.f);
                        const float before = M;
#pragma unroll
                        for (int k = 0; k < 4; ++k) M = fmaxf(M, v[k].x);
                        const float base = M == NEG_INF ? 0.f : M;
                        L *= before == NEG_INF ? 0.f : ex2(before - base);
#pragma unroll
                        for (int k = 0; k < 4; ++k) L += ex2(v[k].x - base) * v[k].y;
                    }
                    const float base_m = M == NEG_INF ? 0.f : M;
                    const float inv = L > 0.f ? 1.f / L : 0.f;
#pragma unroll 1
                    for (int d = 0; d < D; d += 64) {
                        float acc[64];
#pragma unroll
                        for (int e = 0; e < 64; ++e) acc[e] = 0.f;
#pragma unroll 1
                        for (int b = block0; b <= block1; ++b) {
                            uint32_t r[64];
                            const float ws = ex2(ml_of(b).x - base_m) * inv;
                            if (b == me) {
                                tmem_ld32_nowait(my_o + d, r);
                                tmem_ld32_nowait(my_o + d + 32, r + 32);
                                tmem_ld_wait();
                            } else {
                                const uint4* from = reinterpret_cast<const uint4*>(p.part_o + place_of(b) * BQ * D) + row + (d / 4) * BQ;
#pragma unroll
                                for (int e = 0; e < 16; ++e) {
                                    const uint4 v = __ldcg(from + e * BQ);
                                    r[4 * e] = v.x; r[4 * e + 1] = v.y; r[4 * e + 2] = v.z; r[4 * e + 3] = v.w;
                                }
                            }
#pragma unroll
                            for (int e = 0; e < 64; ++e) acc[e] = fmaf(ws, __uint_as_float(r[e]), acc[e]);
                        }
                        store32(d, acc);
                        store32(d + 32, acc + 32);
                    }
                }
            }
            if (STAGE_IN_Q) {
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");    // the next Q comes by TMA
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.q_free[wg]);
            }
        }
        if (!ok && lane == 0) { atomicOr(p.err, KVB_DEV_TIMEOUT); sh.failed = 1; }
        __syncwarp();
    }

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (sh.failed && tid == 0) {      // give copies that may still be in flight a bounded chance to land: the last ones into every place
        for (int h = 0; h < 2; ++h)
            if (sh.q_copies[h] > 0) mbar_wait(&sh.q_full[h], (sh.q_copies[h] - 1) & 1);
        for (int c = max(0, sh.k_copies - KST); c < sh.k_copies; ++c) mbar_wait(&sh.k_full[c % KST], (c / KST) & 1);
        for (int c = max(0, sh.v_copies - VST); c < sh.v_copies; ++c) mbar_wait(&sh.v_full[c % VST], (c / VST) & 1);
    }
    __syncthreads();
    if (warp == 12) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(sh.tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

static int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, Params& p, float* scratch, int blocks, cudaStream_t stream) {
    if (p.n_tiles > MAX_TILES || p.min_tiles < 1 || blocks < 1) return KVB_ERR_SHAPE;
    p.part_o = scratch;
    p.part_ml = scratch + (size_t)4 * blocks * BQ * D;
    p.scale_log2 = p.scale * 1.4426950408889634f;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attention_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    kvb_launch(attention_pairs_kernel, dim3(blocks), dim3(THREADS), (size_t)SMEM_BYTES, stream, mq, mk, mv, p);
    return kvb_launch_status();
}

}  // namespace apr

#if !KVB_EXPANDED
// q, out: [T, Hq * D] bfloat16; k_pages, v_pages: [num_pages, Hkv, page_size, D]; tiles: int32 [n_tiles, 2] (segment, first
// of up to 256 rows); scratch: 4 * blocks * 128 * (D + 2) floats; tickets: 2 * n_tiles * Hq ints, zero before the first
// launch (the kernel leaves them zero); blocks: the GPU's SMs.  page_size a power of two, 8..64.
KVB_API int kvb_attention_pairs(const void* q, void* out, const void* k_pages, const void* v_pages, int num_pages,
                             const int* block_table, int table_stride, const int* tiles, int n_tiles, float* scratch,
                             int* tickets, int blocks, const int* seg_q_start, const int* seg_q_len, const int* seg_kv_len, int T,
                             int Hq, int Hkv, int page_size, int window, float scale, const float* sink, int keep_first,
                             const float* slopes, float cap, int min_tiles, int* err, cudaStream_t stream) {
    using namespace apr;
    if (n_tiles <= 0) return KVB_OK;
    if (Hkv < 1 || Hq % Hkv != 0 || Hq > 65535) return KVB_ERR_SHAPE;
    if (page_size < 8 || page_size > 64 || (page_size & (page_size - 1)) != 0) return KVB_ERR_SHAPE;
    if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) return KVB_ERR_ALIGN;
    CUtensorMap mq, mk, mv;
    int rc = make_bf16_map(&mq, q, T, Hq * D, (long long)Hq * D, BQ);
    if (rc != KVB_OK) return rc;
    const long long pool_rows = (long long)num_pages * Hkv * page_size;
    rc = make_bf16_map(&mk, k_pages, pool_rows, D, D, page_size);
    if (rc != KVB_OK) return rc;
    rc = make_bf16_map(&mv, v_pages, pool_rows, D, D, page_size);
    if (rc != KVB_OK) return rc;
    Params p = {};
    p.out = (bf16*)out; p.block_table = block_table; p.tiles = tiles; p.n_tiles = n_tiles;
    p.seg_q_start = seg_q_start; p.seg_q_len = seg_q_len; p.seg_kv_len = seg_kv_len;
    p.tickets = tickets;
    p.table_stride = table_stride; p.Hq = Hq; p.Hkv = Hkv; p.page_size = page_size; p.q_head = D;
    while ((1 << p.page_shift) < page_size) ++p.page_shift;
    p.window = window; p.min_tiles = min_tiles;
    p.sink = sink; p.keep = keep_first;
    p.slopes = slopes; p.cap = cap; p.scale = scale;
    p.err = err;
    return launch(mq, mk, mv, p, scratch, blocks, stream);
}
#else
// The same attention over keys and values that a latent was expanded to (csrc/latent.cu, kvb_latent_expand_prepare): kv [key_rows,
// 2 * H * D] - the heads' keys, then the heads' values - and rot [key_rows, 64], the keys' rotated part that all heads share (`rot`
// numbers of it).  q: rows of `q_ld` numbers, head h's D + rot at column h (D + rot).  seg_key_row: the row of kv that a segment's key 0
// has, or would have.  gate: out *= sigmoid(gate[t, gate_col + h D + d]), or, with `gate_per_head`, sigmoid(gate[t, gate_col + h]).
KVB_API int kvb_attention_pairs_expanded(const void* q, int q_ld, void* out, const void* kv, const void* rot_rows, int key_rows, const int* tiles,
                                         int n_tiles, float* scratch, int* tickets, int blocks, const int* seg_key_row,
                                         const int* seg_q_start, const int* seg_q_len, const int* seg_kv_len, int T, int H, int rot, int window,
                                         float scale, const float* sink, const void* gate, int gate_stride, int gate_col, int gate_per_head,
                                         int min_tiles, int* err, cudaStream_t stream) {
    using namespace apr;
    if (n_tiles <= 0) return KVB_OK;
    if (H < 1 || H > 65535 || rot < 16 || rot > 64 || rot % 16 != 0 || q_ld % 8 != 0 || H * (D + rot) > q_ld || key_rows < 1 || !gate) return KVB_ERR_SHAPE;
    if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)kv | (uintptr_t)rot_rows) & 15) return KVB_ERR_ALIGN;
    if (!gate_per_head && (((uintptr_t)gate & 15) || gate_stride % 8 != 0 || gate_col % 8 != 0)) return KVB_ERR_ALIGN;
    CUtensorMap mq, mk, mr;
    int rc = make_bf16_map(&mq, q, T, q_ld, q_ld, BQ);
    if (rc != KVB_OK) return rc;
    rc = make_bf16_map(&mk, kv, key_rows, 2 * H * D, 2LL * H * D, BK);
    if (rc != KVB_OK) return rc;
    rc = make_bf16_map(&mr, rot_rows, key_rows, 64, 64, BK);
    if (rc != KVB_OK) return rc;
    Params p = {};
    p.out = (bf16*)out; p.tiles = tiles; p.n_tiles = n_tiles;
    p.seg_q_start = seg_q_start; p.seg_q_len = seg_q_len; p.seg_kv_len = seg_kv_len; p.seg_key_row = seg_key_row;
    p.tickets = tickets;
    p.Hq = p.Hkv = H; p.q_head = D + rot; p.rot_steps = rot / 16;
    p.window = window; p.min_tiles = min_tiles; p.sink = sink; p.scale = scale;
    p.gate = (const bf16*)gate; p.gate_stride = gate_stride; p.gate_col = gate_col; p.gate_per_head = gate_per_head;
    p.err = err;
    return launch(mq, mk, mr, p, scratch, blocks, stream);
}
#endif
