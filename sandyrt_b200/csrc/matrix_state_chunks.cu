// The gated delta rule and the matrix memory (the formulas stand in matrix_state.cu) for requests that bring many tokens, with
// query/key sizes up to 64: everything that does not need the state is formed for all chunks of 32 tokens side by side, and what
// goes from chunk to chunk is reduced to one small product.
//
// delta rule     With G the running sum of the decays' logarithms inside a chunk, r(t, j) = exp(G_t - G_j), and L the unit
//                lower triangular system of matrix_state.cu solved for both right-hand sides,
//                    U = L^-1 (beta v),   W = L^-1 (beta exp(G) k),   u = U - W S0
//                the rest is linear in the state before the chunk, S0:
//                    S  = exp(G_31) S0 + (N - A S0),   A = K'^T W,  N = K'^T U,  K'_j = exp(G_31 - G_j) k_j
//                    o  = Q S0 + P U,     Q_t = exp(G_t) q_t - sum_j P(t, j) W_j,  P(t, j) = r(t, j) (q_t . k_j)
//                so a chunk costs the walk one [d, d] x [d, columns] product and no triangular system.  A S0 is summed
//                by itself: started from N, or with exp(G_31) inside A, each of its 64 products would be rounded at the size
//                of the whole state (error of the state against 64 bits beside the walk's, mean over 144 settings of length,
//                keys, write strength and decay: 1.12 times, up to 1.65; so 0.74 times, up to 1.03).
//   delta_chunk_prepare_kernel   a block a (chunk, head, request): A, N, Q, exp(G_31), and P U into the output
//   delta_chunk_states_kernel    a block a (request, head, 16 columns) walks the chunks and leaves S0 of each
//   delta_chunk_output_kernel    a block a (chunk, head, request): the output plus Q S0
//
// matrix memory  The decay is one number a token, so the state before a chunk is an element-wise recurrence over the chunks'
//                own sums (with each chunk's own maximum a as its exponents' zero; none that is formed is above zero):
//                    N = sum_j exp(a_j - a) k_j v_j^T;   m' = F + max(m, a);   S' = exp(F + m - m') S + exp(F + a - m') N
//   mlstm_chunk_prepare_kernel   N, n and (F, a) of every chunk
//   mlstm_chunk_states_kernel    four elements a thread, chunk after chunk
//   mlstm_chunk_output_kernel    the read-out from S0 and the chunk's own tokens
//
// All float32, the inputs in the projection's type.  The kernels that walk with everything in one block (matrix_state.cu) spend 9
// and 6 us a chunk, whatever the head count; they keep sizes above 64.  Alone, us, those -> these: 2 x 1,024 tokens, 12 heads, delta
// rule 278 -> 115, 24 heads 400 -> 201; 3 heads of 64 x 128, matrix memory 179 -> 37; one request of 96 tokens 29 -> 25
// and 22 -> 21, of 64 21 / 23 and 16 / 21.  The walk is bound by its chain (a product of 64 x 64 x 16 and two barriers a chunk), the
// others by shared-memory loads beside the fmas.
#include "common.cuh"
#include "matrix_state.h"

namespace {

constexpr int COLS = SANDY_MATRIX_STATE_COLS;
constexpr int CC = 32;                  // tokens a chunk: one warp's scan
constexpr int D = 64;                   // rows of the state; smaller heads run with rows of zeros
constexpr int LD = D + 4;               // row pitch in shared memory: eight neighbouring rows start in eight groups of banks
constexpr int LT = CC + 4;

__device__ __forceinline__ float log_sigmoid_f(float z) { return fminf(z, 0.0f) - log1pf(expf(-fabsf(z))); }

__device__ __forceinline__ float scan_sum(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}
__device__ __forceinline__ float scan_max(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = fmaxf(v, u);
    }
    return v;
}
__device__ __forceinline__ float4 at4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void put4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }
__device__ __forceinline__ void copy_16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc[r][c] += x[r] * y[c]
template <int R>
__device__ __forceinline__ void outer(float2 (&acc)[R][2], const float (&x)[R], const float4& y) {
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float2 xx = make_float2(x[r], x[r]);
        acc[r][0] = __ffma2_rn(xx, make_float2(y.x, y.y), acc[r][0]);
        acc[r][1] = __ffma2_rn(xx, make_float2(y.z, y.w), acc[r][1]);
    }
}
template <int R>
__device__ __forceinline__ void clear(float2 (&acc)[R][2]) {
#pragma unroll
    for (int r = 0; r < R; r++) acc[r][0] = acc[r][1] = make_float2(0.0f, 0.0f);
}

// The four tokens' own corner of a triangular product: token r takes y[0 .. r] and nothing of the later ones (zero times what is
// not finite is not zero).  Pt: weights [token of y][token], pitch LT.
__device__ __forceinline__ void corner(float2 (&acc)[4][2], const float* Pt, const float* y, int ldy) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float4 v = at4(y + j * ldy);
#pragma unroll
        for (int r = j; r < 4; r++) {
            const float2 w = make_float2(Pt[j * LT + r], Pt[j * LT + r]);
            acc[r][0] = __ffma2_rn(w, make_float2(v.x, v.y), acc[r][0]);
            acc[r][1] = __ffma2_rn(w, make_float2(v.z, v.w), acc[r][1]);
        }
    }
}

// x . y_b for four rows y_b of Y that lie eight rows apart (rows of D floats at pitch LD).
__device__ __forceinline__ void dots(const float* X, const float* Y, float (&out)[4]) {
    float2 acc[4];
#pragma unroll
    for (int b = 0; b < 4; b++) acc[b] = make_float2(0.0f, 0.0f);
#pragma unroll 4
    for (int i = 0; i < D; i += 4) {
        const float4 x = at4(X + i);
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const float4 y = at4(Y + b * 8 * LD + i);
            acc[b] = __ffma2_rn(make_float2(x.z, x.w), make_float2(y.z, y.w), __ffma2_rn(make_float2(x.x, x.y), make_float2(y.x, y.y), acc[b]));
        }
    }
#pragma unroll
    for (int b = 0; b < 4; b++) out[b] = acc[b].x + acc[b].y;
}

// Chunk c of request s has place q_start[s] / 32 + s + c in the scratch: no two requests' chunks meet, and n_tokens / 32 + n_seqs
// places hold them all.
__device__ __forceinline__ long long place(int t0, int s, int chunk) { return (long long)(t0 / CC + s + chunk); }

// ---- delta rule ----------------------------------------------------------------------------------------------
// Of a (place, head): -A transposed [column][row] (D * D), Q transposed [row of the state][token] (D * CC), N [D][ep], ep the value
// size in whole 64s, and exp(G_31) (and 31 floats that keep the parts on 128-byte boundaries); the states overwrite N.
__host__ __device__ constexpr long long delta_floats(int ep) { return (long long)D * D + D * CC + (long long)D * ep + 32; }

// grid (chunks x 64s of columns, heads, requests), 256 threads.
__global__ void __launch_bounds__(256, 2)
delta_chunk_prepare_kernel(const float* __restrict__ qkv, int ld, const float* __restrict__ bg, const int* __restrict__ q_start,
                           float* __restrict__ scratch, float* __restrict__ out, int ld_out, int n_heads, int n_qk_heads, int d,
                           int e, int long_from) {
    __shared__ __align__(16) float q[CC * LD], k[CC * LD], uw[CC][2 * D + 4], L[CC * LT], Pt[CC * LT], beta[CC], G[CC];
    const int tiles = (e + 63) / 64, chunk = blockIdx.x / tiles, col0 = blockIdx.x % tiles * 64, h = blockIdx.y, s = blockIdx.z;
    const int t0 = q_start[s], n = q_start[s + 1] - t0, tc = t0 + chunk * CC, n_tok = min(CC, n - chunk * CC);
    pdl_wait();
    if (n < long_from || n_tok <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int qh = h / (n_heads / n_qk_heads);
    const bool with_w = col0 == 0;
    float* mine = scratch + (place(t0, s, chunk) * n_heads + h) * delta_floats(tiles * 64);

    if (tid < CC) {
        const bool live = tid < n_tok;          // behind the last token: nothing is written (beta 0), nothing decays
        beta[tid] = live ? bg[(size_t)(tc + tid) * 2 * n_heads + h] : 0.0f;
        G[tid] = scan_sum(live ? bg[(size_t)(tc + tid) * 2 * n_heads + n_heads + h] : 0.0f, tid);
    }
#pragma unroll
    for (int u = 0; u < CC * D / 256; u++) {
        const int x = tid + u * 256, t = x / D, i = x % D;
        const float* row = qkv + (size_t)(tc + t) * ld;
        const bool live = t < n_tok;
        q[t * LD + i] = live && i < d ? row[qh * d + i] : 0.0f;
        k[t * LD + i] = live && i < d ? row[(n_qk_heads + qh) * d + i] : 0.0f;
        uw[t][i] = live && col0 + i < e ? row[2 * n_qk_heads * d + h * e + col0 + i] : 0.0f;
    }
    __syncthreads();
    {
        const int t = tid / 8, j0 = tid % 8;
        float a[4], b[4];
        dots(q + t * LD, k + j0 * LD, a);
        dots(k + t * LD, k + j0 * LD, b);
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int j = j0 + 8 * x;
            const float r = j <= t ? expf(G[t] - G[j]) : 0.0f;
            Pt[j * LT + t] = j <= t ? r * a[x] : 0.0f;
            L[t * LT + j] = j < t ? beta[t] * r * b[x] : 0.0f;
        }
    }
    __syncthreads();
    // the triangular system, a column a thread: 64 of U, 64 of W
    if (tid < (with_w ? 2 * D : D)) {
        float y[CC];
#pragma unroll
        for (int t = 0; t < CC; t++) y[t] = 0.0f;
#pragma unroll
        for (int t = 0; t < CC; t++) {
            float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int j = 0; j < t; j += 4) {    // (from t on L is zero)
                const float4 l = at4(L + t * LT + j);
                sum = __ffma2_rn(make_float2(l.z, l.w), make_float2(y[j + 2], y[j + 3]), __ffma2_rn(make_float2(l.x, l.y), make_float2(y[j], y[j + 1]), sum));
            }
            const float right = tid < D ? beta[t] * uw[t][tid] : beta[t] * expf(G[t]) * k[t * LD + tid - D];
            y[t] = right - (sum.x + sum.y);
        }
#pragma unroll
        for (int t = 0; t < CC; t++) uw[t][tid] = y[t];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < CC * D / 256; u++) {
        const int x = tid + u * 256, t = x / D, i = x % D;
        k[t * LD + i] *= expf(G[CC - 1] - G[t]);
    }
    __syncthreads();
    const int c4 = lane * 4;                    // this lane's four columns of U (0 .. 63) or W
    if (c4 < D || with_w) {
        const int r0 = warp * 4;                // four tokens
        float2 acc[4][2];
        clear(acc);
        for (int j = 0; j < r0; j++) {
            const float4 p = at4(Pt + j * LT + r0);
            const float x[4] = {p.x, p.y, p.z, p.w};
            outer(acc, x, at4(&uw[j][c4]));
        }
        corner(acc, Pt + r0 * LT + r0, &uw[r0][c4], 2 * D + 4);
        if (c4 < D) {
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float o[4] = {acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y};
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (r0 + r < n_tok && col0 + c4 + c < e) out[(size_t)(tc + r0 + r) * ld_out + h * e + col0 + c4 + c] = o[c];
            }
        } else {
            float* qt = mine + D * D;
            float w[4][4], g[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                w[r][0] = acc[r][0].x; w[r][1] = acc[r][0].y; w[r][2] = acc[r][1].x; w[r][3] = acc[r][1].y;
                g[r] = expf(G[r0 + r]);
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int i = c4 - D + c;
                put4(qt + i * CC + r0, g[0] * q[r0 * LD + i] - w[0][c], g[1] * q[(r0 + 1) * LD + i] - w[1][c],
                     g[2] * q[(r0 + 2) * LD + i] - w[2][c], g[3] * q[(r0 + 3) * LD + i] - w[3][c]);
            }
        }
        const int i0 = warp * 8;                // eight rows of the state
        float2 sum[8][2];
        clear(sum);
#pragma unroll 4
        for (int j = 0; j < CC; j++) {
            const float4 k0 = at4(k + j * LD + i0), k1 = at4(k + j * LD + i0 + 4);
            const float x[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
            outer(sum, x, at4(&uw[j][c4]));
        }
        if (c4 < D) {
            float* N = mine + D * D + D * CC;
#pragma unroll
            for (int r = 0; r < 8; r++) put4(N + (size_t)(i0 + r) * tiles * 64 + col0 + c4, sum[r][0].x, sum[r][0].y, sum[r][1].x, sum[r][1].y);
        } else {
            float a[4][8];
#pragma unroll
            for (int r = 0; r < 8; r++) { a[0][r] = sum[r][0].x; a[1][r] = sum[r][0].y; a[2][r] = sum[r][1].x; a[3][r] = sum[r][1].y; }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int i = c4 - D + c;
#pragma unroll
                for (int r = 0; r < 8; r++) a[c][r] = -a[c][r];
                put4(mine + i * D + i0, a[c][0], a[c][1], a[c][2], a[c][3]);
                put4(mine + i * D + i0 + 4, a[c][4], a[c][5], a[c][6], a[c][7]);
            }
            if (tid == D / 4) put4(mine + D * D + D * CC + D * tiles * 64, expf(G[CC - 1]), 0.0f, 0.0f, 0.0f);     // the first such thread
        }
    }
    pdl_launch_dependents();
}

constexpr int WALK_STAGES = 3, WALK_STAGE = D * D + D * COLS + 32;   // floats: A, 16 columns of N, the decay

// grid (requests, heads, 16s of columns), 128 threads: four rows and two columns of the state each.
__global__ void __launch_bounds__(128)
delta_chunk_states_kernel(float* __restrict__ scratch, float* __restrict__ state, long long state_stride,
                          const int* __restrict__ q_start, const int* __restrict__ seq_slots, int n_heads, int d, int e,
                          int long_from) {
    extern __shared__ __align__(16) float ring[];
    __shared__ __align__(16) float S[D * COLS];
    const int s = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * COLS, ep = (e + 63) / 64 * 64;
    const int t0 = q_start[s], n = q_start[s + 1] - t0, chunks = (n + CC - 1) / CC;
    pdl_wait();
    if (n < long_from || n <= 0) return;
    const int tid = threadIdx.x, r0 = tid % 16 * 4, c0 = tid / 16 * 2;
    float* St = state + (long long)seq_slots[s] * state_stride + (long long)h * e * d;
    auto of = [&](int c) { return scratch + (place(t0, s, c) * n_heads + h) * delta_floats(ep); };
    auto load = [&](int c) {
        if (c < chunks) {
            const float* from = of(c);
            float* to = ring + c % WALK_STAGES * WALK_STAGE;
#pragma unroll
            for (int u = 0; u < D * D / 512; u++) copy_16(to + (tid + u * 128) * 4, from + (tid + u * 128) * 4);
#pragma unroll
            for (int u = 0; u < D * COLS / 512; u++) {
                const int x = tid + u * 128, i = x / (COLS / 4), c4 = x % (COLS / 4) * 4;
                copy_16(to + D * D + x * 4, from + D * D + D * CC + (size_t)i * ep + col0 + c4);
            }
            if (tid == 0) copy_16(to + D * D + D * COLS, from + D * D + D * CC + D * ep);
        }
        commit_group();
    };
    load(0);
    load(1);
    for (int x = tid; x < D * COLS; x += 128) {
        const int c = x / D, i = x % D;
        S[i * COLS + c] = (i < d && col0 + c < e) ? St[(size_t)(col0 + c) * d + i] : 0.0f;
    }
    auto at = [&](int i, int c) { return i < d && col0 + c < e ? St[(size_t)(col0 + c) * d + i] : 0.0f; };
    float2 own[4];                              // this thread's part of the state
#pragma unroll
    for (int r = 0; r < 4; r++) own[r] = make_float2(at(r0 + r, c0), at(r0 + r, c0 + 1));
    for (int c = 0; c < chunks; c++) {
        wait_groups<1>();
        __syncthreads();                        // this chunk's A and N are there, the state is whole
        load(c + 2);
        const float* A = ring + c % WALK_STAGES * WALK_STAGE;
        const float* N = A + D * D;
        float* S0 = of(c) + D * D + D * CC;
#pragma unroll
        for (int u = 0; u < D * COLS / 512; u++) {
            const int x = tid + u * 128, i = x / (COLS / 4), c4 = x % (COLS / 4) * 4;
            *reinterpret_cast<float4*>(S0 + (size_t)i * ep + col0 + c4) = at4(S + x * 4);
        }
        float2 acc[4], n4[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            acc[r] = make_float2(0.0f, 0.0f);
            n4[r] = *reinterpret_cast<const float2*>(N + (r0 + r) * COLS + c0);
        }
        const float2 decay = make_float2(N[D * COLS], N[D * COLS]);
#pragma unroll 8
        for (int i = 0; i < D; i++) {
            const float4 a = at4(A + i * D + r0);
            const float2 sv = *reinterpret_cast<const float2*>(S + i * COLS + c0);
            acc[0] = __ffma2_rn(make_float2(a.x, a.x), sv, acc[0]);
            acc[1] = __ffma2_rn(make_float2(a.y, a.y), sv, acc[1]);
            acc[2] = __ffma2_rn(make_float2(a.z, a.z), sv, acc[2]);
            acc[3] = __ffma2_rn(make_float2(a.w, a.w), sv, acc[3]);
        }
#pragma unroll
        for (int r = 0; r < 4; r++) own[r] = __ffma2_rn(decay, own[r], __fadd2_rn(n4[r], acc[r]));
        __syncthreads();                        // everyone has read the state
#pragma unroll
        for (int r = 0; r < 4; r++) *reinterpret_cast<float2*>(S + (r0 + r) * COLS + c0) = own[r];
    }
    pdl_launch_dependents();
    __syncthreads();
    for (int x = tid; x < D * COLS; x += 128) {
        const int c = x / D, i = x % D;
        if (i < d && col0 + c < e) St[(size_t)(col0 + c) * d + i] = S[i * COLS + c];
    }
}

// grid (chunks x 64s of columns, heads, requests), 128 threads: four tokens and four columns each.
__global__ void __launch_bounds__(128)
delta_chunk_output_kernel(const float* __restrict__ scratch, const int* __restrict__ q_start, float* __restrict__ out, int ld_out,
                          int n_heads, int e, int long_from) {
    __shared__ __align__(16) float qt[D * CC], S0[D * 64];
    const int tiles = (e + 63) / 64, chunk = blockIdx.x / tiles, col0 = blockIdx.x % tiles * 64, h = blockIdx.y, s = blockIdx.z;
    const int t0 = q_start[s], n = q_start[s + 1] - t0, tc = t0 + chunk * CC, n_tok = min(CC, n - chunk * CC);
    pdl_wait();
    if (n < long_from || n_tok <= 0) return;
    const int tid = threadIdx.x, r0 = tid / 16 * 4, c0 = tid % 16 * 4;
    const float* mine = scratch + (place(t0, s, chunk) * n_heads + h) * delta_floats(tiles * 64) + D * D;
#pragma unroll
    for (int u = 0; u < D * CC / 512; u++) copy_16(qt + (tid + u * 128) * 4, mine + (tid + u * 128) * 4);
#pragma unroll
    for (int u = 0; u < D * 64 / 512; u++) {
        const int x = tid + u * 128, i = x / 16, c4 = x % 16 * 4;
        copy_16(S0 + x * 4, mine + D * CC + (size_t)i * tiles * 64 + col0 + c4);
    }
    commit_group();
    wait_groups<0>();
    __syncthreads();
    float2 acc[4][2];
    clear(acc);
#pragma unroll 8
    for (int i = 0; i < D; i++) {
        const float4 qv = at4(qt + i * CC + r0);
        const float x[4] = {qv.x, qv.y, qv.z, qv.w};
        outer(acc, x, at4(S0 + i * 64 + c0));
    }
    pdl_launch_dependents();
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const float o[4] = {acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y};
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (r0 + r < n_tok && col0 + c0 + c < e) out[(size_t)(tc + r0 + r) * ld_out + h * e + col0 + c0 + c] += o[c];
    }
}

// ---- matrix memory -------------------------------------------------------------------------------------------
// Of a (place, head): N [D][ep] and n [D], ep the value size in whole fours, then F, a and the m before the chunk.  The states
// overwrite N and n.
__host__ __device__ constexpr long long mlstm_floats(int ep) { return (long long)D * (ep + 1) + 4; }

struct MemoryArgs {
    int ld, q_off, k_off, v_off;
    const float* gates;
    int ld_gates;
    const float* gate_bias;
    float cap, q_scale;
    const int* q_start;
    const int* seq_slots;
    float* scratch;
    int n_heads, d, e, long_from;
};

// Of token `lane` of a chunk: a = log i - F and F, the running sum of log f.  Tokens behind the last: -inf and no decay.
__device__ __forceinline__ float2 memory_gates(const MemoryArgs& p, int h, int tc, int n_tok, int lane) {
    float li = -INFINITY, lf = 0.0f;
    if (lane < n_tok) {
        const float* g = p.gates + (size_t)(tc + lane) * p.ld_gates;
        li = p.cap * tanhf((g[h] + p.gate_bias[h]) / p.cap);
        lf = log_sigmoid_f(p.cap * tanhf((g[p.n_heads + h] + p.gate_bias[p.n_heads + h]) / p.cap));
    }
    const float F = scan_sum(lf, lane);
    return make_float2(li - F, F);
}

// grid (chunks x 128s of columns, heads, requests), 256 threads: eight rows and four columns of N each.
template <typename T>
__global__ void __launch_bounds__(256)
mlstm_chunk_prepare_kernel(const T* __restrict__ proj, const MemoryArgs p) {
    __shared__ __align__(16) float k[CC * LD], v[CC][128 + 4], a[CC];
    const int tiles = (p.e + 127) / 128, chunk = blockIdx.x / tiles, col0 = blockIdx.x % tiles * 128, h = blockIdx.y, s = blockIdx.z;
    const int t0 = p.q_start[s], n = p.q_start[s + 1] - t0, tc = t0 + chunk * CC, n_tok = min(CC, n - chunk * CC);
    pdl_wait();
    if (n < p.long_from || n_tok <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ep = (p.e + 3) / 4 * 4;
    float* mine = p.scratch + (place(t0, s, chunk) * p.n_heads + h) * mlstm_floats(ep);
#pragma unroll
    for (int u = 0; u < CC * D / 256; u++) {
        const int x = tid + u * 256, t = x / D, i = x % D;
        k[t * LD + i] = t < n_tok && i < p.d ? to_f32(proj[(size_t)(tc + t) * p.ld + p.k_off + h * p.d + i]) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < CC * 128 / 256; u++) {
        const int x = tid + u * 256, t = x / 128, c = x % 128;
        v[t][c] = t < n_tok && col0 + c < p.e ? to_f32(proj[(size_t)(tc + t) * p.ld + p.v_off + h * p.e + col0 + c]) : 0.0f;
    }
    if (warp == 0) {
        const float2 g = memory_gates(p, h, tc, n_tok, lane);
        const float top = warp_max(g.x);
        a[lane] = expf(g.x - top);
        if (lane == CC - 1 && col0 == 0) {
            mine[(size_t)D * (ep + 1)] = g.y;
            mine[(size_t)D * (ep + 1) + 1] = top;
        }
    }
    __syncthreads();
    const int i0 = warp * 8, c4 = lane * 4;
    float2 sum[8][2];
    float ones[8];
    clear(sum);
#pragma unroll
    for (int r = 0; r < 8; r++) ones[r] = 0.0f;
#pragma unroll 4
    for (int j = 0; j < CC; j++) {
        const float w = a[j];
        const float4 k0 = at4(k + j * LD + i0), k1 = at4(k + j * LD + i0 + 4);
        const float x[8] = {w * k0.x, w * k0.y, w * k0.z, w * k0.w, w * k1.x, w * k1.y, w * k1.z, w * k1.w};
        outer(sum, x, at4(&v[j][c4]));
#pragma unroll
        for (int r = 0; r < 8; r++) ones[r] += x[r];
    }
    pdl_launch_dependents();
    if (col0 + c4 < ep)
#pragma unroll
        for (int r = 0; r < 8; r++) put4(mine + (size_t)(i0 + r) * ep + col0 + c4, sum[r][0].x, sum[r][0].y, sum[r][1].x, sum[r][1].y);
    if (col0 == 0 && lane == 0)
#pragma unroll
        for (int r = 0; r < 8; r++) mine[(size_t)D * ep + i0 + r] = ones[r];
}

constexpr int AHEAD = 8;                // chunks on their way at once

// grid (1,024s of the state's elements, heads, requests), 256 threads: four of the D * (ep + 1) elements each.
__global__ void __launch_bounds__(256)
mlstm_chunk_states_kernel(const MemoryArgs p, float* __restrict__ state, long long state_stride) {
    const int h = blockIdx.y, s = blockIdx.z, d = p.d, e = p.e, ep = (e + 3) / 4 * 4, Z = (e + COLS - 1) / COLS;
    const int t0 = p.q_start[s], n = p.q_start[s + 1] - t0, chunks = (n + CC - 1) / CC;
    pdl_wait();
    if (n < p.long_from || n <= 0) return;
    const int x = (blockIdx.x * 256 + threadIdx.x) * 4;
    if (x >= D * (ep + 1)) return;
    float* base = state + (long long)p.seq_slots[s] * state_stride;
    float* n_st = base + (long long)p.n_heads * e * d + (long long)h * Z * d;
    float* m_st = base + (long long)p.n_heads * e * d + (long long)p.n_heads * Z * d + (long long)h * Z;
    // elements x .. x + 3: columns of one row of S, or rows of n
    auto home = [&](int y) -> float* {
        const int at = x + y;
        if (at >= D * ep) return at - D * ep < d ? n_st + (at - D * ep) : nullptr;
        return at / ep < d && at % ep < e ? base + (long long)h * e * d + (long long)(at % ep) * d + at / ep : nullptr;
    };
    float S[4];
#pragma unroll
    for (int y = 0; y < 4; y++) S[y] = home(y) ? *home(y) : 0.0f;
    float m = m_st[0];
    float* at = p.scratch + (place(t0, s, 0) * p.n_heads + h) * mlstm_floats(ep);
    const long long apart = p.n_heads * mlstm_floats(ep);
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 N[AHEAD];
        float2 g[AHEAD];
#pragma unroll
        for (int c = 0; c < AHEAD; c++)
            if (c0 + c < chunks) {
                N[c] = at4(at + (c0 + c) * apart + x);
                g[c] = *reinterpret_cast<const float2*>(at + (c0 + c) * apart + (long long)D * (ep + 1));
            }
#pragma unroll
        for (int c = 0; c < AHEAD; c++)
            if (c0 + c < chunks) {
                float* to = at + (c0 + c) * apart;
                put4(to + x, S[0], S[1], S[2], S[3]);
                if (x == 0) to[(long long)D * (ep + 1) + 2] = m;
                const float top = fmaxf(m, g[c].y), old = expf(m - top), own = expf(g[c].y - top);
                S[0] = old * S[0] + own * N[c].x; S[1] = old * S[1] + own * N[c].y;
                S[2] = old * S[2] + own * N[c].z; S[3] = old * S[3] + own * N[c].w;
                m = g[c].x + top;
            }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int y = 0; y < 4; y++)
        if (float* to = home(y)) {
            *to = S[y];
            if (x >= D * ep)                    // n and m are kept once per block of columns
                for (int z = 1; z < Z; z++) to[(long long)z * d] = S[y];
        }
    // (m itself is written by the last chunk's read-out: every block here reads the old one)
}

struct OutputSmem { float q[CC * LD], k[CC * LD], qT[D * LT], v[CC][128 + 4], Pt[CC * LT], S0[D][128], n0[D], a[CC], M[CC], F[CC], c[CC], den[CC]; };

// grid (chunks x 128s of columns, heads, requests), 256 threads: four tokens and four columns each.
template <typename T>
__global__ void __launch_bounds__(256, 2)
mlstm_chunk_output_kernel(const T* __restrict__ proj, const MemoryArgs p, float* __restrict__ state, long long state_stride,
                          float* __restrict__ out, int ld_out) {
    extern __shared__ __align__(16) unsigned char raw[];
    OutputSmem& m = *reinterpret_cast<OutputSmem*>(raw);
    const int tiles = (p.e + 127) / 128, chunk = blockIdx.x / tiles, col0 = blockIdx.x % tiles * 128, h = blockIdx.y, s = blockIdx.z;
    const int t0 = p.q_start[s], n = p.q_start[s + 1] - t0, tc = t0 + chunk * CC, n_tok = min(CC, n - chunk * CC);
    pdl_wait();
    if (n < p.long_from || n_tok <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ep = (p.e + 3) / 4 * 4;
    const float* mine = p.scratch + (place(t0, s, chunk) * p.n_heads + h) * mlstm_floats(ep);
#pragma unroll
    for (int u = 0; u < D * 128 / 1024; u++) {
        const int x = tid + u * 256, i = x / 32, c4 = x % 32 * 4;
        if (col0 + c4 < ep) copy_16(&m.S0[i][c4], mine + (size_t)i * ep + col0 + c4);
        else put4(&m.S0[i][c4], 0.0f, 0.0f, 0.0f, 0.0f);
    }
    commit_group();
#pragma unroll
    for (int u = 0; u < CC * D / 256; u++) {
        const int x = tid + u * 256, t = x / D, i = x % D;
        const T* row = proj + (size_t)(tc + t) * p.ld + h * p.d + i;
        const bool live = t < n_tok && i < p.d;
        const float qv = live ? to_f32(row[p.q_off]) * p.q_scale : 0.0f;
        m.q[t * LD + i] = qv;
        m.qT[i * LT + t] = qv;
        m.k[t * LD + i] = live ? to_f32(row[p.k_off]) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < CC * 128 / 256; u++) {
        const int x = tid + u * 256, t = x / 128, c = x % 128;
        m.v[t][c] = t < n_tok && col0 + c < p.e ? to_f32(proj[(size_t)(tc + t) * p.ld + p.v_off + h * p.e + col0 + c]) : 0.0f;
    }
    if (tid < D) m.n0[tid] = mine[(size_t)D * ep + tid];
    if (warp == 0) {
        const float m0 = mine[(size_t)D * (ep + 1) + 2];
        const float2 g = memory_gates(p, h, tc, n_tok, lane);
        const float M = fmaxf(scan_max(g.x, lane), m0);
        m.a[lane] = g.x;
        m.F[lane] = g.y;
        m.M[lane] = M;
        m.c[lane] = expf(m0 - M);
        if (tc + CC >= t0 + n && col0 == 0) {           // the last chunk: m of the state behind it
            const int Z = (p.e + COLS - 1) / COLS;
            float* m_st = state + (long long)p.seq_slots[s] * state_stride + (long long)p.n_heads * p.e * p.d +
                          (long long)p.n_heads * Z * p.d + (long long)h * Z;
            const float last = __shfl_sync(0xffffffffu, g.y + M, CC - 1);
            for (int z = lane; z < Z; z += 32) m_st[z] = last;
        }
    }
    wait_groups<0>();
    __syncthreads();
    {
        const int t = tid / 8, j0 = tid % 8;
        float w[4], nq = 0.0f, own = 0.0f;
        dots(m.q + t * LD, m.k + j0 * LD, w);
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int j = j0 + 8 * x;
            w[x] = j <= t ? w[x] * expf(m.a[j] - m.M[t]) : 0.0f;
            m.Pt[j * LT + t] = w[x];
            own += w[x];
        }
#pragma unroll
        for (int x = 0; x < D / 8; x++) nq = fmaf(m.q[t * LD + j0 + 8 * x], m.n0[j0 + 8 * x], nq);
        nq = m.c[t] * nq + own;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) nq += __shfl_xor_sync(0xffffffffu, nq, o);
        if (j0 == 0) m.den[t] = fmaxf(fabsf(nq), expf(-(m.F[t] + m.M[t]))) + 1e-6f;
    }
    __syncthreads();
    const int r0 = warp * 4, c4 = lane * 4;
    float2 acc[4][2];
    clear(acc);
#pragma unroll 8
    for (int i = 0; i < D; i++) {
        const float4 qv = at4(m.qT + i * LT + r0);
        const float x[4] = {qv.x, qv.y, qv.z, qv.w};
        outer(acc, x, at4(&m.S0[i][c4]));
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const float2 c = make_float2(m.c[r0 + r], m.c[r0 + r]);
        acc[r][0] = __fmul2_rn(acc[r][0], c);
        acc[r][1] = __fmul2_rn(acc[r][1], c);
    }
    for (int j = 0; j < r0; j++) {
        const float4 pv = at4(m.Pt + j * LT + r0);
        const float x[4] = {pv.x, pv.y, pv.z, pv.w};
        outer(acc, x, at4(&m.v[j][c4]));
    }
    corner(acc, m.Pt + r0 * LT + r0, &m.v[r0][c4], 128 + 4);
    pdl_launch_dependents();
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const float o[4] = {acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y};
        const float den = m.den[r0 + r];
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (r0 + r < n_tok && col0 + c4 + c < p.e) out[(size_t)(tc + r0 + r) * ld_out + h * p.e + col0 + c4 + c] = o[c] / den;
    }
}

bool sizes_fit(int n_tokens, int n_seqs, int max_q_len, int n_heads, int d, int e, int long_from) {
    return n_tokens > 0 && n_seqs > 0 && n_seqs <= 65535 && n_heads > 0 && n_heads <= 65535 && max_q_len > 0 && d > 0 && d <= D && e > 0 &&
           e <= 1024 && long_from >= 1;
}

}  // namespace

// Floats of scratch of a step of n_tokens tokens of n_seqs requests; kind 0 the delta rule, 1 the matrix memory.
SANDY_API long long sandy_matrix_chunks_scratch(int kind, int n_tokens, int n_seqs, int n_heads, int v_dim) {
    const long long places = (long long)n_tokens / CC + n_seqs;
    return places * n_heads * (kind == 0 ? delta_floats((v_dim + 63) / 64 * 64) : mlstm_floats((v_dim + 3) / 4 * 4));
}

// Requests that bring at least `long_from` tokens (sandy_delta_scan, given the same number, takes the others); arguments as there.
// scratch: sandy_matrix_chunks_scratch floats on a 16-byte boundary.  max_q_len: the most tokens a request brings.
SANDY_API int sandy_delta_chunks(const float* qkv, int ld, const float* bg, float* state, long long state_stride, const int* q_start,
                                 const int* seq_slots, float* scratch, float* out, int ld_out, int n_tokens, int n_seqs,
                                 int max_q_len, int n_heads, int n_qk_heads, int qk_dim, int v_dim, int long_from,
                                 cudaStream_t stream) {
    if (n_seqs == 0) return SANDY_OK;
    if (!qkv || !bg || !state || !q_start || !seq_slots || !scratch || !out) return SANDY_ERR_ARGUMENT;
    if (!sizes_fit(n_tokens, n_seqs, max_q_len, n_heads, qk_dim, v_dim, long_from) || n_qk_heads <= 0 || n_heads % n_qk_heads ||
        ((uintptr_t)scratch & 15))
        return SANDY_ERR_UNSUPPORTED;
    const int chunks = (max_q_len + CC - 1) / CC, tiles = (v_dim + 63) / 64;
    const dim3 wide(chunks * tiles, n_heads, n_seqs), walk(n_seqs, n_heads, (v_dim + COLS - 1) / COLS);
    const int ring = WALK_STAGES * WALK_STAGE * (int)sizeof(float);
    const cudaError_t set = cudaFuncSetAttribute(delta_chunk_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ring);
    if (set != cudaSuccess) return (int)set;
    int code = sandy_launch(delta_chunk_prepare_kernel, wide, dim3(256), 0, stream, qkv, ld, bg, q_start, scratch, out, ld_out, n_heads,
                            n_qk_heads, qk_dim, v_dim, long_from);
    if (code == 0)
        code = sandy_launch(delta_chunk_states_kernel, walk, dim3(128), ring, stream, scratch, state, state_stride, q_start, seq_slots,
                            n_heads, qk_dim, v_dim, long_from);
    if (code == 0)
        code = sandy_launch(delta_chunk_output_kernel, wide, dim3(128), 0, stream, scratch, q_start, out, ld_out, n_heads, v_dim, long_from);
    return code;
}

// Likewise for sandy_mlstm_scan.
SANDY_API int sandy_mlstm_chunks(const void* proj, int ld, int dtype, int q_off, int k_off, int v_off, const float* gates, int ld_gates,
                                 const float* gate_bias, float cap, float q_scale, float* state, long long state_stride,
                                 const int* q_start, const int* seq_slots, float* scratch, float* out, int ld_out, int n_tokens,
                                 int n_seqs, int max_q_len, int n_heads, int qk_dim, int v_dim, int long_from, cudaStream_t stream) {
    if (n_seqs == 0) return SANDY_OK;
    if (!proj || !gates || !gate_bias || !state || !q_start || !seq_slots || !scratch || !out) return SANDY_ERR_ARGUMENT;
    if (!sizes_fit(n_tokens, n_seqs, max_q_len, n_heads, qk_dim, v_dim, long_from) || !(cap > 0.0f) || ((uintptr_t)scratch & 15) ||
        (dtype != SANDY_F32 && dtype != SANDY_BF16))
        return SANDY_ERR_UNSUPPORTED;
    const MemoryArgs p = {ld, q_off, k_off, v_off, gates, ld_gates, gate_bias, cap, q_scale, q_start, seq_slots, scratch, n_heads,
                          qk_dim, v_dim, long_from};
    const int chunks = (max_q_len + CC - 1) / CC, tiles = (v_dim + 127) / 128, ep = (v_dim + 3) / 4 * 4;
    const dim3 wide(chunks * tiles, n_heads, n_seqs), walk((D * (ep + 1) + 1023) / 1024, n_heads, n_seqs);
    auto go = [&](auto zero) {
        using T = decltype(zero);
        const cudaError_t set = cudaFuncSetAttribute(mlstm_chunk_output_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OutputSmem));
        if (set != cudaSuccess) return (int)set;
        int code = sandy_launch(mlstm_chunk_prepare_kernel<T>, wide, dim3(256), 0, stream, (const T*)proj, p);
        if (code == 0) code = sandy_launch(mlstm_chunk_states_kernel, walk, dim3(256), 0, stream, p, state, state_stride);
        if (code == 0)
            code = sandy_launch(mlstm_chunk_output_kernel<T>, wide, dim3(256), sizeof(OutputSmem), stream, (const T*)proj, p, state,
                                state_stride, out, ld_out);
        return code;
    };
    return dtype == SANDY_F32 ? go(float()) : go(bf16());
}
