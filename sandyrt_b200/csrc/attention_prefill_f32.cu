// Causal attention of prompt portions in float32, heads of up to 128, on the 32-bit pipes: heads up to 32, and steps of very many
// single tokens that the decode kernel has no form for (attention_prefill_f32_tc.cu takes the others).  A tile of queries of one head
// against tiles of keys, every product and sum on the 32-bit pipes.  The formula, the cache layout and the rules are those of the
// general kernel (attention.cu), which gives a warp one (token, head) pair and so reads every key once per query: 2 TFLOP/s.
//
// What bounds it is the fma rate.  A block of four warps takes 64 queries of one head and walks the keys they see 64 at a time,
// with an online softmax.  A warp owns 16 queries (its rows of the scores and of the output never leave it), a thread 8
// queries x 4 keys, then 8 queries x 4 (or 8) output columns: a load of 16 bytes from shared memory feeds 16 to 64 packed
// fmas.  Scores pair two entries of the head (queries and keys run along it), the output pairs two columns.  Keys and values
// come by cp.async from the request's pages, values under the scores, the next keys under the output; for heads above 64 the
// probabilities take the keys' place, so that two blocks fit an SM.
// Alone, us, the general kernel -> this one: two prompts of 1,024 tokens, 12 heads of 64: 1,607 -> 132 (24 TFLOP/s of the pairs a
// causal mask leaves); four of 100 to 412 tokens, 12 heads of 128 on one key/value head: 470 -> 99; 32 single tokens behind
// 100 to 700 beside a portion of 480, 16 heads of 64: 573 -> 119.  What is left is instructions beside the fmas (softmax, loads
// from shared memory) and, in short steps, a block's serial start.
#include "attention_rules.h"
#include "common.cuh"

namespace {

constexpr int BQ = 64, BKEYS = 64, THREADS = 128;
constexpr int P_PITCH = BKEYS + 4;
constexpr float NOT_SEEN = -0.0f;       // the probability of a key that a query does not see (one it sees has at least +0)

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
    int num_pages, q_pieces;
    int* status;
};

__device__ __forceinline__ void copy_16(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;       // 0: the sixteen bytes are filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Head sizes in between run as the next wider form, whose further entries are zeros in shared memory.
template <int D>
struct Form {
    static constexpr int PITCH = D + 4;             // floats: the rows of eight neighbouring lanes start in eight groups of banks
    static constexpr int COLS = D < 64 ? 4 : D / 16;            // output columns a thread
    static constexpr int BLOCKS = D > 64 ? 2 : 3;               // on an SM
    static constexpr bool P_IN_KEYS = D > 64;
    static constexpr int TILE = 64 * PITCH, KEYS = P_IN_KEYS && TILE < BQ * P_PITCH ? BQ * P_PITCH : TILE;
    static constexpr int SMEM = (TILE + KEYS + TILE + (P_IN_KEYS ? 0 : BQ * P_PITCH)) * 4;
};

// grid (heads, requests, tiles of queries): every request's longest tiles start first.
template <int D>
__global__ void __launch_bounds__(THREADS, Form<D>::BLOCKS)
prefill_attention_f32_kernel(const PromptArgs p) {
    using F = Form<D>;
    constexpr int PITCH = F::PITCH, COLS = F::COLS;
    extern __shared__ __align__(128) float smem[];
    __shared__ long long key_row[2][BKEYS];         // row of the cache (in rows of a head) of each key of a tile; -1: none
    const int seq = blockIdx.y, head = blockIdx.x;
    const int q0 = p.q_start[seq], n_q = p.q_start[seq + 1] - q0;
    const int tile = (n_q + BQ - 1) / BQ - 1 - (int)blockIdx.z;
    if (tile < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = lane >> 4, tx = lane & 15;
    const int d = p.head_dim;
    const int kv_head = head / (p.n_heads / p.n_kv_heads);
    const int rows = min(BQ, n_q - tile * BQ);
    const int pos0 = p.kv_before[seq] + tile * BQ, t0 = q0 + tile * BQ;
    float* q_s = smem;
    float* k_s = q_s + F::TILE;
    float* v_s = k_s + F::KEYS;
    float* p_s = F::P_IN_KEYS ? k_s : v_s + F::TILE;

    // Keys the tile sees: those kept in front of a window (0 .. kept - 1), then first .. pos0 + rows - 1.
    const SandyAttentionRules& r = p.rules;
    const VisibleKeys of_first = visible_keys(pos0, r.window, r.keep_first, r.chunk);
    const int first = of_first.lo, kept = of_first.kept, last = pos0 + rows - 1;
    const int kept_tiles = (kept + BKEYS - 1) / BKEYS, tiles = kept_tiles + (last - first + BKEYS) / BKEYS;
    const int* table = p.block_table + (size_t)seq * p.max_blocks;
    const long long rows_per_page = p.page_stride / d;
    auto tile_start = [&](int t) { return t < kept_tiles ? t * BKEYS : first + (t - kept_tiles) * BKEYS; };
    auto tile_end = [&](int t) { return t < kept_tiles ? kept : last + 1; };         // the first key behind the tile's part
    auto find_rows = [&](int t) {
        if (tid < BKEYS) {
            const int j = tile_start(t) + tid;
            long long row = -1;
            if (j < tile_end(t)) {
                const int block = j / p.page_size, page = block < p.max_blocks ? table[block] : -1;
                if (page >= 0 && page < p.num_pages)
                    row = page * rows_per_page + (long long)kv_head * p.page_size + (j - block * p.page_size);
                else if (p.status)
                    atomicOr(p.status, 16);         // a visible key with no page behind it: report it, read nothing
            }
            key_row[t & 1][tid] = row;
        }
    };
    // a thread copies one piece of every (THREADS / (D / 4))-th row
    constexpr int APART = THREADS / (D / 4);
    const int copy_row = tid / (D / 4), copy_col = tid % (D / 4) * 4;
    auto copy_tile = [&](int t, const float* cache, float* to) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(to + copy_row * PITCH + copy_col);
#pragma unroll 8
        for (int i = 0; i < BKEYS / APART; i++) {
            const long long at = key_row[t & 1][copy_row + i * APART];
            const bool there = at >= 0 && copy_col < d;
            copy_16(dst + i * APART * PITCH * 4, cache + (there ? at * d + copy_col : 0), there);
        }
        commit_group();
    };

    pdl_wait();
    if (p.q_pieces) {                               // the queries' rows start on 16-byte boundaries
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(q_s + copy_row * PITCH + copy_col);
#pragma unroll 8
        for (int i = 0; i < BQ / APART; i++) {
            const bool there = copy_row + i * APART < rows && copy_col < d;
            copy_16(dst + i * APART * PITCH * 4, p.q + (there ? (size_t)(t0 + copy_row + i * APART) * p.ld_q + head * d + copy_col : 0), there);
        }
    } else {
        for (int i = tid; i < BQ * D; i += THREADS) {
            const int row = i / D, c = i % D;
            q_s[row * PITCH + c] = row < rows && c < d ? p.q[(size_t)(t0 + row) * p.ld_q + head * d + c] : 0.0f;
        }
    }
    find_rows(0);
    __syncthreads();
    copy_tile(0, p.k, k_s);
    const int row0 = warp * 16 + ty;                // this thread's queries: row0 + 2 i
    const bool idle = warp * 16 >= rows;            // a warp without queries only helps with the copies
    const bool ruled = r.window > 0 || r.chunk > 0 || r.softcap > 0.0f || r.dist_bias;
    float m[8], l[8];                               // l: of this thread's keys alone, until the end
    float2 o[8][COLS / 2];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < COLS / 2; c++) o[i][c] = make_float2(0.0f, 0.0f);
    }

    for (int t = 0; t < tiles; t++) {
        if (t + 1 < tiles) find_rows(t + 1);
        wait_groups<0>();
        __syncthreads();                            // these keys are there, and nobody reads the last values any more
        copy_tile(t, p.v, v_s);
        const int start = tile_start(t), end = tile_end(t);
        float s[8][4];
        if (!idle) {
            float2 acc[8][4];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
            const float* qp = q_s + row0 * PITCH;
            const float* kp = k_s + tx * PITCH;
#pragma unroll 4
            for (int c = 0; c < D; c += 4) {
                float4 kv[4];
#pragma unroll
                for (int j = 0; j < 4; j++) kv[j] = *reinterpret_cast<const float4*>(kp + 16 * j * PITCH + c);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 qv = *reinterpret_cast<const float4*>(qp + 2 * i * PITCH + c);
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(make_float2(qv.x, qv.y), make_float2(kv[j].x, kv[j].y), acc[i][j]);
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(make_float2(qv.z, qv.w), make_float2(kv[j].z, kv[j].w), acc[i][j]);
                }
            }
            // keys that a page is missing for are not seen either
            const bool found = key_row[t & 1][tx] >= 0 && key_row[t & 1][tx + 16] >= 0 && key_row[t & 1][tx + 32] >= 0 && key_row[t & 1][tx + 48] >= 0;
            const bool whole = __all_sync(0xffffffffu, !ruled && found && start + BKEYS - 1 <= pos0);
            bool rose = false;
            float corr[8];
            unsigned hidden = 0;                    // bit 8 j + i: query i does not see key j, whatever its score is
#pragma unroll
            for (int i = 0; i < 8; i++) {
#pragma unroll
                for (int j = 0; j < 4; j++) s[i][j] = (acc[i][j].x + acc[i][j].y) * p.scale;
            }
            if (!whole) {
#pragma unroll 1
                for (int j = 0; j < 4; j++) {       // one code for the four keys: it runs for the tiles at the edges only
                    const int at = tx + 16 * j, key = start + at;
                    const bool there = key < end && key_row[t & 1][at] >= 0;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int pos = pos0 + row0 + 2 * i;
                        const int lo = visible_keys(pos, r.window, r.keep_first, r.chunk).lo;
                        const bool seen = there && key <= pos && (key >= lo || key < r.keep_first);
                        float x = j == 0 ? s[i][0] : j == 1 ? s[i][1] : j == 2 ? s[i][2] : s[i][3];
                        if (r.softcap > 0.0f) x = r.softcap * tanhf(x / r.softcap);
                        if (r.dist_bias && seen) x += r.dist_bias[(size_t)head * r.n_dist + min(pos - key, r.n_dist - 1)];
                        x = seen ? x : -INFINITY;
                        hidden |= seen ? 0u : 1u << (8 * j + i);
                        s[i][0] = j == 0 ? x : s[i][0];
                        s[i][1] = j == 1 ? x : s[i][1];
                        s[i][2] = j == 2 ? x : s[i][2];
                        s[i][3] = j == 3 ? x : s[i][3];
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float top = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
                const float m_new = fmaxf(m[i], top), base = m_new == -INFINITY ? 0.0f : m_new;
                corr[i] = expf(m[i] - base);
                rose |= m_new != m[i];
                m[i] = m_new;
#pragma unroll
                for (int j = 0; j < 4; j++) s[i][j] = expf(s[i][j] - base);      // (a score that is NaN stays one)
                l[i] = l[i] * corr[i] + ((s[i][0] + s[i][1]) + (s[i][2] + s[i][3]));
            }
            if (!whole) {
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (hidden >> (8 * j + i) & 1) s[i][j] = NOT_SEEN;
            }
            if (__any_sync(0xffffffffu, rose)) {
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int c = 0; c < COLS / 2; c++) o[i][c] = __fmul2_rn(o[i][c], make_float2(corr[i], corr[i]));
            }
        }
        __syncthreads();                            // nobody reads these keys any more
        if (!F::P_IN_KEYS && t + 1 < tiles) copy_tile(t + 1, p.k, k_s);
        else commit_group();
        if (!idle) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) p_s[(row0 + 2 * i) * P_PITCH + tx + 16 * j] = s[i][j];
        }
        wait_groups<1>();
        __syncthreads();                            // the values are there
        // A value that some queries of the tile do not see must not reach them, were it not finite (0 times it is not 0).
        bool odd = false;
        if (end - 1 > pos0 || r.window > 0 || r.chunk > 0) {
            for (int i = tid; i < BKEYS * D / 4; i += THREADS) {
                const float4 v = *reinterpret_cast<const float4*>(v_s + i / (D / 4) * PITCH + i % (D / 4) * 4);
                odd |= !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w));
            }
            odd = __syncthreads_or(odd);
        }
        const bool with_columns = D >= 64 || tx * 4 < D;
        if (odd && !idle && with_columns) {
            for (int k = 0; k < BKEYS; k++)
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float pr = p_s[(row0 + 2 * i) * P_PITCH + k];
                    if (__float_as_uint(pr) == __float_as_uint(NOT_SEEN)) continue;
#pragma unroll
                    for (int c = 0; c < COLS; c++) {
                        float& to = c % 2 ? o[i][c / 2].y : o[i][c / 2].x;
                        to = fmaf(pr, v_s[k * PITCH + (c / 4) * 64 + tx * 4 + c % 4], to);
                    }
                }
        } else if (!idle && with_columns) {
            const float* pp = p_s + row0 * P_PITCH;
            const float* vp = v_s + tx * 4;
            const int keys = min(BKEYS, end - start);       // behind them the probabilities are zero
#pragma unroll 2
            for (int k = 0; k < keys; k += 4) {
                float4 pr[8];
#pragma unroll
                for (int i = 0; i < 8; i++) pr[i] = *reinterpret_cast<const float4*>(pp + 2 * i * P_PITCH + k);
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    float4 vv[COLS / 4];
#pragma unroll
                    for (int b = 0; b < COLS / 4; b++) vv[b] = *reinterpret_cast<const float4*>(vp + (k + e) * PITCH + 64 * b);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const float x = e == 0 ? pr[i].x : e == 1 ? pr[i].y : e == 2 ? pr[i].z : pr[i].w;
                        const float2 twice = make_float2(x, x);
#pragma unroll
                        for (int b = 0; b < COLS / 4; b++) {
                            o[i][2 * b] = __ffma2_rn(twice, make_float2(vv[b].x, vv[b].y), o[i][2 * b]);
                            o[i][2 * b + 1] = __ffma2_rn(twice, make_float2(vv[b].z, vv[b].w), o[i][2 * b + 1]);
                        }
                    }
                }
            }
        }
        if (F::P_IN_KEYS) {
            __syncthreads();                        // nobody reads the probabilities any more: the next keys may come
            if (t + 1 < tiles) copy_tile(t + 1, p.k, k_s);
        }
    }
    pdl_launch_dependents();
    if (idle) return;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = row0 + 2 * i, token = t0 + row;
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], w);
        if (row >= rows) continue;
        const float den = r.sink ? l[i] + expf(r.sink[head] - m[i]) : l[i];
        const float gate = r.out_gate ? r.out_gate[(size_t)token * p.n_heads + head] : 1.0f;
#pragma unroll
        for (int c = 0; c < COLS; c++) {
            const int col = (c / 4) * 64 + tx * 4 + c % 4;
            const float sum = c % 2 ? o[i][c / 2].y : o[i][c / 2].x;
            if (col < d)
                p.out[(size_t)token * p.ld_out + head * d + col] =
                    sum / den * gate * elem_gate_of((const float*)r.elem_gate, r.ld_elem_gate, r.gate_dim, token, head, col);
        }
    }
}

template <int D>
int launch(const PromptArgs& p, int n_seqs, int max_q_len, cudaStream_t stream) {
    const cudaError_t set = cudaFuncSetAttribute(prefill_attention_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, Form<D>::SMEM);
    if (set != cudaSuccess) return (int)set;
    const dim3 grid(p.n_heads, n_seqs, (max_q_len + BQ - 1) / BQ);
    return sandy_launch(prefill_attention_f32_kernel<D>, grid, dim3(THREADS), Form<D>::SMEM, stream, p);
}

}  // namespace

// q: [n_tokens, H*D] with row stride ld_q; request s has the tokens q_start[s] .. q_start[s + 1] - 1 at positions from
// kv_before[s] on; out like q with row stride ld_out; float32 throughout.  Head sizes that are multiples of 16 up to 128.
SANDY_API int sandy_prefill_attention_f32_rules(const float* q, int ld_q, const float* k_cache, const float* v_cache,
                                                long long page_stride, const int* block_table, int max_blocks,
                                                const int* q_start, const int* kv_before, float* out, int ld_out, int n_seqs,
                                                int max_q_len, int n_heads, int n_kv_heads, int head_dim, int page_size,
                                                float scale, const SandyAttentionRules* rules, int num_pages, int* status,
                                                cudaStream_t stream) {
    if (n_seqs == 0 || max_q_len == 0) return SANDY_OK;
    if (!rules || !q || !k_cache || !v_cache || !block_table || !q_start || !kv_before || !out) return SANDY_ERR_ARGUMENT;
    if (rules->dist_bias && rules->n_dist < 1) return SANDY_ERR_ARGUMENT;
    if (rules->keep_first < 0 || (rules->keep_first > 0 && rules->chunk > 0) || (rules->elem_gate && rules->gate_dim < 1))
        return SANDY_ERR_UNSUPPORTED;
    if (head_dim <= 0 || head_dim % 16 != 0 || head_dim > 128) return SANDY_ERR_UNSUPPORTED;
    if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0 || page_size <= 0 || rules->window < 0 || n_seqs > 65535 || max_q_len > 65535 * BQ)
        return SANDY_ERR_UNSUPPORTED;
    if (page_stride % head_dim != 0 || rules->softcap < 0.0f || rules->chunk < 0) return SANDY_ERR_UNSUPPORTED;
    if (((uintptr_t)k_cache & 15) || ((uintptr_t)v_cache & 15)) return SANDY_ERR_UNSUPPORTED;
    const PromptArgs p = {q, ld_q, k_cache, v_cache, page_stride, block_table, max_blocks, q_start, kv_before, out, ld_out, n_heads,
                          n_kv_heads, head_dim, page_size, scale, *rules, num_pages, !((uintptr_t)q & 15) && ld_q % 4 == 0, status};
    if (head_dim <= 32) return launch<32>(p, n_seqs, max_q_len, stream);
    return head_dim <= 64 ? launch<64>(p, n_seqs, max_q_len, stream) : launch<128>(p, n_seqs, max_q_len, stream);
}
