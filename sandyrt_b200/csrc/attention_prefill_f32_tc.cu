// Causal attention of prompt portions in float32 on the tensor cores, every operand in three bfloat16 pieces (split_f32.cuh); heads
// above 32, up to 128.  The formula, the cache layout and the rules are those of attention.cu and attention_prefill_f32.cu.
//
// A block takes 128 queries of one head and walks the keys they see 64 at a time.  A warp issues the products (each instruction waits for
// the tensor cores to take it: a warp with other work held the rest up for longer than the products take); of sixteen others four
// threads share a query's row, each 16 keys of the scores and a quarter of the output's columns.  Per tile of keys:
//   S = Q K^T      both operands' pieces in shared memory, an accumulator in tensor memory (k is the head: 64 or 128)
//   softmax        in float registers, with the row's exact maximum; the four threads of a row exchange theirs
//   O = P V        the probabilities' pieces go to tensor memory (a thread its row), the values' lie in shared memory as the cache has
//                  them (keys along k); one accumulator for this tile alone, added into float registers with the rescaled sum
// so no accumulator takes more than one chunk of k (two for heads above 64).  S of the next tile runs beside a tile's softmax, O beside the
// next tile's; keys and values are fetched into registers a tile ahead.
//
// What is not finite, or so large that its product could leave the pieces' range (2^39 and more), the tensor cores can't take: the scores
// of such a query or key are formed with float arithmetic from the cache, such a value is left out of its tile's sum and added in float
// arithmetic at the end, so that a NaN or an infinity reaches the queries that see it and no others.
//
// What bounds it: the issue slots of the sixteen warps (splitting keys, values and probabilities, softmax: 3,500 a tile and scheduler of
// the 5,000 clocks a tile takes) and the chain from a tile's scores to the next; the products are a quarter of that.  Alone, us, the fma
// tiles of attention_prefill_f32.cu -> this kernel: two prompts of 1,024 tokens, 12 heads of 64 132 -> 52; four of 100 to 412, 12 heads
// of 64 54 -> 25, 12 heads of 128 on one key/value head 92 -> 40; one of 16 14 -> 9; four tokens behind 300 33 -> 19.  Error against 64
// bits (2-norm) of the first 2.8e-7 -> 1.5e-7, with values of one sign 2.4e-7 -> 1.0e-7, sharp scores 5.5e-7 -> 3.0e-7 (the exponentials are
// the hardware's base-2 ones, good to 2^-22, on a difference rounded to a float, as expf's argument was).  One query of NaN in the first 88 us,
// one key or value 56, nothing but NaN keys 144, values 94 (fma tiles 132 to 254); one infinite query 445.  With eight warps, one of them issuing the products too, it took 100 us.
//
// Every wait on an mbarrier is bounded: on expiry the kernel raises `*status` (bit 8) and runs to its end (its output is then not valid).
#include "attention_rules.h"
#include "split_f32.cuh"

namespace {

constexpr int KEYS = 64, WORKERS = 512, THREADS = WORKERS + 32, SHARE = 4;         // SHARE: threads a row
constexpr int ROW_SLOTS = 8;            // tiles whose keys' rows are kept
constexpr float LOG2E = 1.4426950408889634f;
constexpr uint32_t TOO_LARGE = 0x53000000u;     // 2^39: products of two, 128 of them, at SCALE twice stay below 2^127

struct PromptArgs {
    const float* q;
    int ld_q;
    const float* k;
    const float* v;
    long long page_stride;
    const int* block_table;
    int max_blocks;
    const int* q_start;
    const int* kv_before;
    float* out;
    int ld_out, n_heads, n_kv_heads, head_dim, page_size;
    float scale;
    SandyAttentionRules rules;
    int portions;           // 0 every request, 2 those of more than one token
    int num_pages, q_pieces, wide;          // q's rows, out's rows start on 16-byte boundaries
    int* status;
};

template <int D>
struct Form {
    static constexpr int BLOCKS = D / 64;                       // of 64 entries of the head: 128 bytes of a piece's row
    static constexpr int Q_PIECE = BLOCKS * BM * 128, KV_PIECE = BLOCKS * KEYS * 128;
    static constexpr int OFF_K = N_PIECES * Q_PIECE, OFF_V = OFF_K + N_PIECES * KV_PIECE, BODY = OFF_V + N_PIECES * KV_PIECE;
    static constexpr int SMEM = BODY + 1024;                    // room to align
    static constexpr uint32_t S_COL = 0, O_COL = 2 * KEYS, P_COL = O_COL + D;      // two accumulators of scores
    static constexpr int ITEMS = KEYS * D / 8 / WORKERS;        // of eight floats, a thread's share of a tile of keys
    static constexpr int COLS = D / SHARE;                      // output columns a thread
};

__device__ __forceinline__ bool is_large(float x) { return (__float_as_uint(x) & 0x7fffffffu) >= TOO_LARGE; }
__device__ __forceinline__ bool too_large(const float4& v) {
    const uint32_t a = __float_as_uint(v.x) & 0x7fffffffu, b = __float_as_uint(v.y) & 0x7fffffffu, c = __float_as_uint(v.z) & 0x7fffffffu,
                   d = __float_as_uint(v.w) & 0x7fffffffu;
    return max(max(a, b), max(c, d)) >= TOO_LARGE;
}

__device__ __forceinline__ bool has_nan(const float4& v) { return v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w; }
__device__ __forceinline__ void keep_small(float4& v) {
    v = make_float4(is_large(v.x) ? 0.0f : v.x, is_large(v.y) ? 0.0f : v.y, is_large(v.z) ? 0.0f : v.z, is_large(v.w) ? 0.0f : v.w);
}

// A query times a key in float arithmetic; the key's row starts on 16 bytes, the query's if `pieces`.
__device__ __forceinline__ float plain_score(const float* q, int pieces, const float* k, int d) {
    float x = 0.0f;
#pragma unroll 1
    for (int c = 0; c < d; c += 4) {
        const float4 a = pieces ? *reinterpret_cast<const float4*>(q + c) : make_float4(q[c], q[c + 1], q[c + 2], q[c + 3]);
        const float4 b = *reinterpret_cast<const float4*>(k + c);
        x = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, x))));
    }
    return x;
}

__device__ __forceinline__ float exp2_of(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// grid (heads, requests, tiles of queries): every request's longest tiles start first.
template <int D>
__global__ void __launch_bounds__(THREADS, 1)
prefill_attention_f32_tc_kernel(const PromptArgs p) {
    using F = Form<D>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ long long key_row[ROW_SLOTS][KEYS];  // row of the cache (in rows of a head) of each key of a tile; -1: none
    __shared__ float part_of[2][SHARE][BM];         // what the threads of a row exchange
    __shared__ uint64_t bars[4];                    // scores are there; a weighted sum is; keys' pieces are; probabilities and values are
    // What the tensor cores can't take: the queries (ODD, and NAN_TOO where one of its entries is a NaN); the keys by the last tile (of
    // those whose number ends in the same bits: other warps leave the keys of two tiles on) in which there was one, and in which this one
    // was one; the first and the last tile with such a value.
    enum { ODD = 1, NAN_TOO = 2 };
    __shared__ int odd_q[BM], odd_k[4], odd_key[4][KEYS], nan_key[4][KEYS], odd_v[2];
    __shared__ uint32_t tmem_slot;
    enum { SCORES, SUM, KEYS_IN, PROBS_IN };
    const int seq = blockIdx.y, head = blockIdx.x;
    const int q0 = p.q_start[seq], n_q = p.q_start[seq + 1] - q0;
    const int tile = (n_q + BM - 1) / BM - 1 - (int)blockIdx.z;
    if (tile < 0 || (p.portions == 2 && n_q == 1)) return;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int part = warp >> 2, row = (warp & 3) * 32 + lane;           // this thread's part of its query's row
    const int d = p.head_dim;
    const int kv_head = head / (p.n_heads / p.n_kv_heads);
    const int rows = min(BM, n_q - tile * BM);
    const int pos0 = p.kv_before[seq] + tile * BM, t0 = q0 + tile * BM, pos = pos0 + row;

    // Keys the tile sees: those kept in front of a window (0 .. kept - 1), then first .. pos0 + rows - 1.
    const SandyAttentionRules& r = p.rules;
    const VisibleKeys of_first = visible_keys(pos0, r.window, r.keep_first, r.chunk);
    const int first = of_first.lo, kept = of_first.kept, last = pos0 + rows - 1;
    const int kept_tiles = (kept + KEYS - 1) / KEYS, tiles = kept_tiles + (last - first + KEYS) / KEYS;
    const int* table = p.block_table + (size_t)seq * p.max_blocks;
    const long long rows_per_page = p.page_stride / d;
    auto tile_start = [&](int t) { return t < kept_tiles ? t * KEYS : first + (t - kept_tiles) * KEYS; };
    auto tile_end = [&](int t) { return t < kept_tiles ? kept : last + 1; };         // the first key behind the tile's part
    // Where the key tid of tile t lies, in two steps: the page, whose entry is a trip to memory, and the row.
    int next_page = -1;
    auto ask_page = [&](int t) {
        const int j = tile_start(t) + tid, block = j / p.page_size;
        next_page = tid < KEYS && t < tiles && j < tile_end(t) && block < p.max_blocks ? table[block] : -1;
    };
    auto keep_row = [&](int t) {
        if (tid < KEYS && t < tiles) {
            const int j = tile_start(t) + tid;
            long long at = -1;
            if (j < tile_end(t)) {
                if (next_page >= 0 && next_page < p.num_pages)
                    at = next_page * rows_per_page + (long long)kv_head * p.page_size + j % p.page_size;
                else if (p.status)
                    atomicOr(p.status, 16);         // a visible key with no page behind it: report it, read nothing
            }
            key_row[t % ROW_SLOTS][tid] = at;
        }
    };
    // A thread's items of a tile: eight entries, from entry `at_d`, of the keys at_key + i * APART.
    constexpr int APART = WORKERS * 8 / D;
    const int at_key = tid / (D / 8), at_d = tid % (D / 8) * 8;
    float4 kv[F::ITEMS][2], vv[F::ITEMS][2];
    auto fetch = [&](int t, const float* cache, float4 (&to)[F::ITEMS][2]) {
#pragma unroll
        for (int i = 0; i < F::ITEMS; i++) {
            const long long at = key_row[t % ROW_SLOTS][at_key + i * APART];
            const bool there = at >= 0 && at_d < d;
            const float4* src = reinterpret_cast<const float4*>(cache + (there ? at * d + at_d : 0));
            to[i][0] = there ? src[0] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            to[i][1] = there ? src[1] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    // Rows of 128 bytes (64 entries), 128-byte swizzle.
    auto leave = [&](const float4 (&x)[2], uint8_t* to, int at_row, int at_entry, int block_bytes, int piece_bytes) {
        uint4 piece[N_PIECES];
        split_eight(x[0], x[1], piece);
        uint8_t* dst = to + (at_entry >> 6) * block_bytes + at_row * 128 + ((((at_entry & 63) >> 3) ^ (at_row & 7)) << 4);
#pragma unroll
        for (int j = 0; j < N_PIECES; j++) *reinterpret_cast<uint4*>(dst + j * piece_bytes) = piece[j];
    };
    auto leave_keys = [&](int t) {
#pragma unroll
        for (int i = 0; i < F::ITEMS; i++) {
            leave(kv[i], smem + F::OFF_K, at_key + i * APART, at_d, KEYS * 128, F::KV_PIECE);
            if (too_large(kv[i][0]) || too_large(kv[i][1])) {
                odd_k[t & 3] = odd_key[t & 3][at_key + i * APART] = t;
                if (has_nan(kv[i][0]) || has_nan(kv[i][1])) nan_key[t & 3][at_key + i * APART] = t;
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // my pieces, before the tensor core reads them
    };
    // (what the tensor cores can't take of the values is added at the end)
    auto leave_values = [&](int t) {
#pragma unroll
        for (int i = 0; i < F::ITEMS; i++) {
            if (too_large(vv[i][0]) || too_large(vv[i][1])) {
                atomicMin(&odd_v[0], t);
                atomicMax(&odd_v[1], t);
                keep_small(vv[i][0]);
                keep_small(vv[i][1]);
            }
            leave(vv[i], smem + F::OFF_V, at_key + i * APART, at_d, KEYS * 128, F::KV_PIECE);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    bool expired = false;
    auto wait = [&](int bar, int phase) {
        if (!expired && !mbar_wait(&bars[bar], phase & 1)) {
            if (p.status) atomicOr(p.status, 256);
            expired = true;
        }
        tc_fence_after();
    };

    if (tid == 0) {
        mbar_init(&bars[SCORES], 1);
        mbar_init(&bars[SUM], 1);
        mbar_init(&bars[KEYS_IN], WORKERS / 32);
        mbar_init(&bars[PROBS_IN], WORKERS / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        odd_v[0] = tiles;
        odd_v[1] = -1;
    }
    if (tid < BM) odd_q[tid] = 0;
    if (tid < 4) odd_k[tid] = -1;
    if (tid < 4 * KEYS) odd_key[tid & 3][tid >> 2] = nan_key[tid & 3][tid >> 2] = -1;
    if (warp == WORKERS / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int t = 0; t < 3; t++) {
        ask_page(t);
        keep_row(t);
    }
    ask_page(3);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, lanes = (uint32_t)((warp & 3) * 32) << 16;
    auto issue_s = [&](int t) {
        constexpr uint32_t idesc = make_instr_desc(KEYS);
#pragma unroll
        for (int i = 0; i < N_PRODUCTS; i++)
#pragma unroll
            for (int b = 0; b < F::BLOCKS; b++) {
                const uint64_t dq = make_smem_desc(smem_u32(smem) + PIECE_OF_A[i] * F::Q_PIECE + b * BM * 128);
                const uint64_t dk = make_smem_desc(smem_u32(smem) + F::OFF_K + PIECE_OF_W[i] * F::KV_PIECE + b * KEYS * 128);
#pragma unroll
                for (int k = 0; k < 64 / UMMA_K; k++)
                    umma_bf16(tmem + F::S_COL + (t & 1) * KEYS, dq + (uint64_t)(2 * k), dk + (uint64_t)(2 * k), idesc, i > 0 || b > 0 || k > 0 ? 1u : 0u);
            }
        umma_commit(&bars[SCORES]);
    };
    auto issue_o = [&] {
        constexpr uint32_t idesc = make_instr_desc(64) | (1u << 16);        // the values' pieces: keys along k, columns contiguous
#pragma unroll
        for (int b = 0; b < F::BLOCKS; b++)
#pragma unroll
            for (int i = 0; i < N_PRODUCTS; i++) {
                const uint32_t v = smem_u32(smem) + F::OFF_V + PIECE_OF_W[i] * F::KV_PIECE + b * KEYS * 128;
#pragma unroll
                for (int k = 0; k < KEYS / UMMA_K; k++)
                    umma_bf16_ta(tmem + F::O_COL + 64 * b, tmem + F::P_COL + PIECE_OF_A[i] * (KEYS / 2) + 8 * k, make_smem_desc(v + k * (UMMA_K * 128)),
                                 idesc, i > 0 || k > 0 ? 1u : 0u);
            }
        umma_commit(&bars[SUM]);
    };

    if (warp == WORKERS / 32) {
        if (elect_one()) {
            for (int t = -1; t < tiles && !expired; t++) {
                if (t + 1 < tiles) {
                    wait(KEYS_IN, t + 1);
                    if (!expired) issue_s(t + 1);
                }
                if (t < 0) continue;
                wait(PROBS_IN, t);
                if (expired) break;
                issue_o();
            }
        }
        __syncwarp();
        pdl_launch_dependents();
        __syncthreads();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
        return;
    }
    auto arrive = [&](int bar) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[bar]);
    };

    pdl_wait();
    fetch(0, p.k, kv);
    for (int i = tid; i < BM * D / 8; i += WORKERS) {
        const int at_row = i / (D / 8), at = i % (D / 8) * 8;
        float4 x[2] = {make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f)};
        if (at_row < rows && at < d) {
            const float* src = p.q + (size_t)(t0 + at_row) * p.ld_q + head * d + at;
            if (p.q_pieces) {
                x[0] = *reinterpret_cast<const float4*>(src);
                x[1] = *reinterpret_cast<const float4*>(src + 4);
            } else {
                x[0] = make_float4(src[0], src[1], src[2], src[3]);
                x[1] = make_float4(src[4], src[5], src[6], src[7]);
            }
        }
        leave(x, smem, at_row, at, BM * 128, F::Q_PIECE);
        if (too_large(x[0]) || too_large(x[1])) atomicOr(&odd_q[at_row], has_nan(x[0]) || has_nan(x[1]) ? ODD | NAN_TOO : ODD);
    }
    leave_keys(0);
    arrive(KEYS_IN);
    if (tiles > 1) fetch(1, p.k, kv);
    fetch(0, p.v, vv);

    const bool ruled = r.window > 0 || r.chunk > 0 || r.softcap > 0.0f || r.dist_bias;
    const int my_lo = visible_keys(pos, r.window, r.keep_first, r.chunk).lo;
    auto meet = [&] {
        __syncwarp();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp & 3)) : "memory");        // the four warps of these rows
    };
    // m: the row's maximum.  It is taken from a score before the product with log2(e): of scores of 2^31 and more that product alone is
    // off by more than an exponential's range.
    float m = -INFINITY, l = 0.0f, corr = 0.0f;     // l: of this thread's keys alone, until the end
    float o[F::COLS];
#pragma unroll
    for (int c = 0; c < F::COLS; c++) o[c] = 0.0f;
    // Tile t's weighted sum into o.
    auto add_sum = [&](int t) {
        wait(SUM, t);
#pragma unroll
        for (int c = 0; c < F::COLS; c += 16) {
            uint32_t raw[16];
            tmem_ld_32x16(tmem + lanes + F::O_COL + part * F::COLS + c, raw);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i++) o[c + i] = fmaf(o[c + i], corr, __uint_as_float(raw[i]) * UNSCALE);
        }
    };

    const float unscale = UNSCALE * p.scale;
    for (int t = 0; t < tiles; t++) {
        constexpr int MINE = KEYS / SHARE;          // keys of a thread: from part * MINE on
        keep_row(t + 3);
        ask_page(t + 4);
        wait(SCORES, t);
        float s[MINE];
        {
            uint32_t raw[MINE];
            tmem_ld_32x16(tmem + lanes + F::S_COL + (t & 1) * KEYS + part * MINE, raw);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < MINE; j++) s[j] = __uint_as_float(raw[j]) * unscale;
        }
        if (t + 1 < tiles) {
            leave_keys(t + 1);
            arrive(KEYS_IN);
            if (t + 2 < tiles) fetch(t + 2, p.k, kv);
        }
        const int start = tile_start(t), end = tile_end(t);
        const long long* key_rows = &key_row[t % ROW_SLOTS][part * MINE];
        const bool found = key_rows[lane % MINE] >= 0;
        const bool odd = odd_q[row] | (odd_k[t & 3] == t);
        if (!__all_sync(0xffffffffu, !odd && !ruled && found && start + KEYS - 1 <= pos0)) {
            // (in a branch that is there anyway: one of its own, never taken, costs heads of 128 5 %)
            if (odd) {
#pragma unroll 1
                for (int j = 0; j < MINE; j++) {
                    const int key = part * MINE + j;
                    if (!odd_q[row] && odd_key[t & 3][key] != t) continue;
                    float x = 0.0f;
                    if ((odd_q[row] & NAN_TOO) || nan_key[t & 3][key] == t) x = NAN;
                    else if (key_rows[j] >= 0 && row < rows)
                        x = plain_score(p.q + (size_t)(t0 + row) * p.ld_q + head * d, p.q_pieces, p.k + key_rows[j] * d, d) * p.scale;
#pragma unroll
                    for (int i = 0; i < MINE; i++) s[i] = i == j ? x : s[i];
                }
            }
            __syncwarp();
            const unsigned there = __ballot_sync(0xffffffffu, found);        // (behind the tile's end no row was found)
            if (r.softcap > 0.0f) {
#pragma unroll
                for (int j = 0; j < MINE; j++) s[j] = r.softcap * tanhf(s[j] / r.softcap);
            }
#pragma unroll
            for (int j = 0; j < MINE; j++) {
                const int key = start + part * MINE + j;
                const bool seen = (there >> j & 1) && key <= pos && (key >= my_lo || key < r.keep_first);
                if (r.dist_bias && seen) s[j] += r.dist_bias[(size_t)head * r.n_dist + min(pos - key, r.n_dist - 1)];
                s[j] = seen ? s[j] : -INFINITY;
            }
        }
        float top = s[0];
#pragma unroll
        for (int j = 1; j < MINE; j++) top = fmaxf(top, s[j]);
        part_of[t & 1][part][row] = top;
        meet();
        const float(&tops)[SHARE][BM] = part_of[t & 1];
        top = fmaxf(fmaxf(tops[0][row], tops[1][row]), fmaxf(tops[2][row], tops[3][row]));
        if (t > 0) add_sum(t - 1);
        const float m_new = fmaxf(m, top), base = m_new == -INFINITY ? 0.0f : m_new;
        corr = exp2_of((m - base) * LOG2E);
        m = m_new;
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < MINE; j++) {
            s[j] = exp2_of((s[j] - base) * LOG2E);          // (a score that is NaN stays one)
            sum += s[j];
        }
        l = l * corr + sum;
        {
            uint4 low[N_PIECES], high[N_PIECES];
            split_eight(make_float4(s[0], s[1], s[2], s[3]), make_float4(s[4], s[5], s[6], s[7]), low);
            split_eight(make_float4(s[8], s[9], s[10], s[11]), make_float4(s[12], s[13], s[14], s[15]), high);
#pragma unroll
            for (int i = 0; i < N_PIECES; i++) tmem_st_32x8(tmem + lanes + F::P_COL + i * (KEYS / 2) + part * (MINE / 2), low[i], high[i]);
        }
        leave_values(t);
        tmem_wait_st();
        arrive(PROBS_IN);
        if (t + 1 < tiles) fetch(t + 1, p.v, vv);
    }
    add_sum(tiles - 1);
    part_of[tiles & 1][part][row] = l;
    pdl_launch_dependents();
    tc_fence_before();
    __syncthreads();
    // What was left out of the values, with the weights that its keys' scores give; what a query does not see must not reach it (0 times
    // it is not 0).  (In the loop over the tiles this code, never taken, took heads of 128 from 82 to 106 us for two prompts of 1,024.)
    for (int t = odd_v[0]; t <= odd_v[1]; t++) {
        bool all_nan = row < rows;
#pragma unroll
        for (int c = 0; c < F::COLS; c++) all_nan &= o[c] != o[c];
        if (__all_sync(0xffffffffu, all_nan || row >= rows)) break;         // nothing changes that any more
        const int end = min(tile_start(t) + KEYS, tile_end(t));
        for (int k0 = tile_start(t); k0 < end; k0 += 32) {
            // a lane a key: whether there is such a value among this warp's columns, and one that is no NaN (which is one under any weight)
            const int block = (k0 + lane) / p.page_size, page = k0 + lane < end && block < p.max_blocks ? table[block] : -1;
            long long at = 0;
            bool large = false, weighed = false;
            if (page >= 0 && page < p.num_pages) {
                at = page * rows_per_page + (long long)kv_head * p.page_size + (k0 + lane) % p.page_size;
                for (int c = part * F::COLS; c < min((part + 1) * F::COLS, d); c += 4) {
                    const float4 y = *reinterpret_cast<const float4*>(p.v + at * d + c);
                    large |= too_large(y);
                    weighed |= (is_large(y.x) && y.x == y.x) || (is_large(y.y) && y.y == y.y) || (is_large(y.z) && y.z == y.z) || (is_large(y.w) && y.w == y.w);
                }
            }
            const unsigned weigh = __ballot_sync(0xffffffffu, weighed);
            for (unsigned keys = __ballot_sync(0xffffffffu, large); keys; keys &= keys - 1) {
                const int j = __ffs(keys) - 1, key = k0 + j;
                const long long of = __shfl_sync(0xffffffffu, at, j) * d;
                if (row >= rows || key > pos || (key < my_lo && key >= r.keep_first)) continue;
                float weight = NAN;
                if (weigh >> j & 1) {
                    float x = plain_score(p.q + (size_t)(t0 + row) * p.ld_q + head * d, p.q_pieces, p.k + of, d) * p.scale;
                    if (r.softcap > 0.0f) x = r.softcap * tanhf(x / r.softcap);
                    if (r.dist_bias) x += r.dist_bias[(size_t)head * r.n_dist + min(pos - key, r.n_dist - 1)];
                    weight = exp2_of((x - (m == -INFINITY ? 0.0f : m)) * LOG2E);
                }
#pragma unroll
                for (int c = 0; c < F::COLS; c += 4) {
                    if (part * F::COLS + c >= d) break;
                    const float4 y = *reinterpret_cast<const float4*>(p.v + of + part * F::COLS + c);
                    o[c] = is_large(y.x) ? fmaf(weight, y.x, o[c]) : o[c];
                    o[c + 1] = is_large(y.y) ? fmaf(weight, y.y, o[c + 1]) : o[c + 1];
                    o[c + 2] = is_large(y.z) ? fmaf(weight, y.z, o[c + 2]) : o[c + 2];
                    o[c + 3] = is_large(y.w) ? fmaf(weight, y.w, o[c + 3]) : o[c + 3];
                }
            }
        }
    }
    if (row >= rows) return;
    const float(&ls)[SHARE][BM] = part_of[tiles & 1];
    l = (ls[0][row] + ls[1][row]) + (ls[2][row] + ls[3][row]);
    const int token = t0 + row;
    const float den = r.sink ? l + expf(r.sink[head] - m) : l;
    const float gate = r.out_gate ? r.out_gate[(size_t)token * p.n_heads + head] : 1.0f;
    float* out = p.out + (size_t)token * p.ld_out + head * d + part * F::COLS;
#pragma unroll
    for (int c = 0; c < F::COLS; c += 4) {
        const int col = part * F::COLS + c;
        if (col >= d) break;
        float x[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            x[i] = o[c + i] / den * gate * elem_gate_of((const float*)r.elem_gate, r.ld_elem_gate, r.gate_dim, token, head, col + i);
        if (p.wide) {
            *reinterpret_cast<float4*>(out + c) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) out[c + i] = x[i];
        }
    }
}

template <int D>
int launch(const PromptArgs& p, int n_seqs, int max_q_len, cudaStream_t stream) {
    const cudaError_t set = cudaFuncSetAttribute(prefill_attention_f32_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, Form<D>::SMEM);
    if (set != cudaSuccess) return (int)set;
    const dim3 grid(p.n_heads, n_seqs, (max_q_len + BM - 1) / BM);
    return sandy_launch(prefill_attention_f32_tc_kernel<D>, grid, dim3(THREADS), Form<D>::SMEM, stream, p);
}

}  // namespace

// Arguments as in sandy_prefill_attention_f32_rules; portions: 0 every request, 2 those that bring more than one token.  Head sizes that are multiples of 16, above 32 and up to 128.
SANDY_API int sandy_prefill_attention_f32_tc_rules(const float* q, int ld_q, const float* k_cache, const float* v_cache,
                                                   long long page_stride, const int* block_table, int max_blocks,
                                                   const int* q_start, const int* kv_before, float* out, int ld_out, int n_seqs,
                                                   int max_q_len, int n_heads, int n_kv_heads, int head_dim, int page_size,
                                                   float scale, const SandyAttentionRules* rules, int portions, int num_pages, int* status,
                                                   cudaStream_t stream) {
    if (n_seqs == 0 || max_q_len == 0) return SANDY_OK;
    if (!rules || !q || !k_cache || !v_cache || !block_table || !q_start || !kv_before || !out) return SANDY_ERR_ARGUMENT;
    if (rules->dist_bias && rules->n_dist < 1) return SANDY_ERR_ARGUMENT;
    if (rules->keep_first < 0 || (rules->keep_first > 0 && rules->chunk > 0) || (rules->elem_gate && rules->gate_dim < 1))
        return SANDY_ERR_UNSUPPORTED;
    if (head_dim <= 32 || head_dim % 16 != 0 || head_dim > 128) return SANDY_ERR_UNSUPPORTED;
    if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0 || page_size <= 0 || rules->window < 0 || n_seqs > 65535 || max_q_len > 65535 * BM || (portions != 0 && portions != 2))
        return SANDY_ERR_UNSUPPORTED;
    if (page_stride % head_dim != 0 || rules->softcap < 0.0f || rules->chunk < 0) return SANDY_ERR_UNSUPPORTED;
    if (((uintptr_t)k_cache & 15) || ((uintptr_t)v_cache & 15)) return SANDY_ERR_UNSUPPORTED;
    const PromptArgs p = {q, ld_q, k_cache, v_cache, page_stride, block_table, max_blocks, q_start, kv_before, out, ld_out, n_heads,
                          n_kv_heads, head_dim, page_size, scale, *rules, portions, num_pages, !((uintptr_t)q & 15) && ld_q % 4 == 0,
                          !((uintptr_t)out & 15) && ld_out % 4 == 0, status};
    return head_dim <= 64 ? launch<64>(p, n_seqs, max_q_len, stream) : launch<128>(p, n_seqs, max_q_len, stream);
}
