// Matrix product of float32 operands on the 32-bit pipes, for weights stored [N, K] whose rows start on 16-byte
// boundaries, with bias / activation / residual folded into the write-back.
//
//   out[m, n] = act( sum_k a[m, k] * w[n, k] + bias[n] ) + residual[m, n]
//
// Every product and sum is an IEEE float operation (no tensor core, no reduced-precision mode).  Both operands run along
// k, so two k at a time go through one packed fma (sums of the even and of the odd k apart, added at the end): half the
// instructions of plain FFMA for the same rate, which leaves issue slots for the loads.  The order of an element's sum is
// fixed by the launch's shape (M, N, K), never by the other rows' values.
//
// Measured alone, weights from HBM, against the general kernel (gemm_simt.cu), us: 8 rows, 2,304 x 768 94 -> 4.1, 768 x 3,072
// 361 -> 5.2, 50,257 x 768 242 -> 46 (3.4 TB/s); 2,048 rows, 2,304 x 768 239 -> 164, 768 x 768 98 -> 68, 3,072 x 768 328 ->
// 246, 768 x 3,072 379 -> 240 (44 TFLOP/s of the 74 the fma units could do: with three 64-bit operands a packed fma takes
// about three cycles of the register file, not two).
//
// Three kernels:
//
// short    small products with a short k (a tiny model's), where a launch's start and end are all there is: tiles of 16 x 16 whose
//          whole k is brought at once, the weights' part before the kernel in front has ended; four warps split k.  57 rows, us:
//          192 x 64 2.5, 64 x 256 3.5 (tiles of 64 x 64 8.6 and 5.3, gemm_f32_tc.cu 5.3 and 5.1).
// stream   few rows.  What bounds it is the weights' way from memory, so nothing is staged: a warp owns four rows of w and
//          a part of k, its lanes run along k in float4 steps (512 contiguous bytes of each row), and the first of them
//          are on their way before the kernel in front has ended (weights are written by no kernel).  Four rows of w
//          share each load of a.  The sums cross the lanes in a halving exchange (31 shuffles for 32 sums), then the
//          warps that share a row in shared memory.
// tile     up to 64 rows of narrow products, where the tensor cores (gemm_f32_tc.cu) do not pay.  Tiles of 32*WM x 8*TN*WN outputs
//          behind a ring of cp.async stages of 32 k; 8 x TN outputs a thread.  Where the tiles are too few for the SMs, the blocks
//          of a cluster split k and add up through shared memory.  What is left to it takes tiles of 64 x 64 in as many parts as k
//          allows; 128 x 128 and 64 x 128, and the rule that weighs them, serve comparisons (microbench.py) and tests.
#include <cooperative_groups.h>

#include <algorithm>

#include "epilogue.cuh"

namespace cg = cooperative_groups;

namespace {

// Two floats that go through one instruction.
__device__ __forceinline__ float2 low(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 high(const float4& v) { return make_float2(v.z, v.w); }

struct Product {
    const float* a;
    const float* w;
    const float* bias;
    const float* residual;
    float* out;
    int M, N, K, lda, ldw, ldr, ldc, act;
};

__device__ __forceinline__ void write_back(const Product& p, int m, int n, float v) {
    if (p.bias) v += p.bias[n];
    v = apply_act(v, p.act);
    if (p.residual) v += p.residual[(size_t)m * p.ldr + n];
    p.out[(size_t)m * p.ldc + n] = v;
}

// ---- few rows ------------------------------------------------------------------------------------------------
constexpr int ROWS = 4;             // rows of w a warp
constexpr int STEP = 128;           // k a warp takes in one step (32 lanes of four)
constexpr int STREAM_WARPS = 8;

// Adds V sums over the 32 lanes; lane i is left with sums [i * V / 32, ...) where V >= 32, else every lane with sum
// i * V / 32.
template <int V>
__device__ __forceinline__ void lane_exchange(float* v, int lane) {
    int width = V;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (width > 1) {
            const bool upper = lane & o;
            const int half = width / 2;
#pragma unroll
            for (int i = 0; i < V / 2; i++) {
                if (i < half) {
                    const float give = upper ? v[i] : v[i + half];
                    const float keep = upper ? v[i + half] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            }
            width = half;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
}

// blockDim (32, parts, groups): threadIdx.z picks four rows of w, threadIdx.y a share of k (steps y, y + parts, ...).
// blockIdx.x picks MB rows of a (blocks that read the same rows of w are neighbours), blockIdx.y the first rows of w; a block
// goes on to the rows gridDim.y blocks further, whose first steps are loaded before the sums of the last ones are added up.
template <int MB, int AHEAD, int BLOCKS>
__global__ void __launch_bounds__(STREAM_WARPS * 32, BLOCKS)
gemm_f32_stream_kernel(const Product p) {
    constexpr int V = MB * ROWS;
    __shared__ float sums[STREAM_WARPS][V];
    const int lane = threadIdx.x, part = threadIdx.y, parts = blockDim.y, group = threadIdx.z, groups = blockDim.z;
    const int m0 = blockIdx.x * MB;
    const int steps = (p.K + STEP - 1) / STEP, whole = p.K / STEP;
    const float* w;             // the first of the four rows
    int row_offset[ROWS];
    auto at_rows = [&](int quad) {
        const int n0 = min(quad * ROWS, p.N - 1);
        w = p.w + (size_t)n0 * p.ldw;
#pragma unroll
        for (int r = 0; r < ROWS; r++) row_offset[r] = min(r, p.N - 1 - n0) * p.ldw;
    };
    // Lanes behind the end of a row load and add nothing: a zero weight there would turn an infinite activation into NaN.  Only a
    // row's last part of a step asks lane by lane, whole steps the warp at once (8 rows of 768 x 3,072: 5.2 us, lane by lane 6.7).
    float4 wv[AHEAD][ROWS];
    auto inside = [&](int step) { return step * STEP + lane * 4 < p.K; };
    auto load_w = [&](int slot, int step) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) wv[slot][r] = __ldg(reinterpret_cast<const float4*>(w + row_offset[r] + step * STEP + lane * 4));
    };
    auto load_first = [&]() {
#pragma unroll
        for (int i = 0; i < AHEAD; i++)
            if (inside(part + i * parts)) load_w(i, part + i * parts);
    };
    pdl_launch_dependents();
    int first = blockIdx.y * groups;
    at_rows(first + group);
    load_first();
    pdl_wait();

    const int n_quads = (p.N + ROWS - 1) / ROWS;
    const float* a = p.a + (size_t)m0 * p.lda;
    for (; first < n_quads; first += gridDim.y * groups) {
        float2 acc[MB][ROWS];
#pragma unroll
        for (int m = 0; m < MB; m++)
#pragma unroll
            for (int r = 0; r < ROWS; r++) acc[m][r] = make_float2(0.0f, 0.0f);
        for (int base = part; base < steps; base += AHEAD * parts) {
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const int step = base + i * parts;
                auto add = [&]() {
                    const float* ak = a + step * STEP + lane * 4;
#pragma unroll
                    for (int m = 0; m < MB; m++) {
                        const float4 av = *reinterpret_cast<const float4*>(ak + (size_t)min(m, p.M - 1 - m0) * p.lda);
#pragma unroll
                        for (int r = 0; r < ROWS; r++)
                            acc[m][r] = __ffma2_rn(high(av), high(wv[i][r]), __ffma2_rn(low(av), low(wv[i][r]), acc[m][r]));
                    }
                };
                if (step < whole) {
                    add();
                    if (step + AHEAD * parts < whole) load_w(i, step + AHEAD * parts);
                    else if (inside(step + AHEAD * parts)) load_w(i, step + AHEAD * parts);
                } else if (inside(step)) {
                    add();
                }
            }
        }
        const int quad = first + group;
        if (first + gridDim.y * groups < n_quads) {
            at_rows(quad + gridDim.y * groups);
            load_first();
        }
        float v[V];
#pragma unroll
        for (int m = 0; m < MB; m++)
#pragma unroll
            for (int r = 0; r < ROWS; r++) v[m * ROWS + r] = acc[m][r].x + acc[m][r].y;
        lane_exchange<V>(v, lane);
        if (parts == 1) {           // nothing to add up across warps: the lanes write their sums, no warp waits for another
#pragma unroll
            for (int i = 0; i < (V + 31) / 32; i++) {
                const int at = V >= 32 ? lane * (V / 32) + i : lane * V / 32;
                const int m = m0 + at / ROWS, n = quad * ROWS + at % ROWS;
                if ((V >= 32 || lane * V % 32 == 0) && m < p.M && n < p.N) write_back(p, m, n, v[i]);
            }
            continue;
        }
        const int warp = group * parts + part;
        __syncthreads();            // the sums of the rows before have been read
        if constexpr (V >= 32) {
#pragma unroll
            for (int i = 0; i < V / 32; i++) sums[warp][lane * (V / 32) + i] = v[i];
        } else {
            if (lane % (32 / V) == 0) sums[warp][lane / (32 / V)] = v[0];
        }
        __syncthreads();
        for (int i = part * 32 + lane; i < V; i += parts * 32) {
            float s = 0.0f;
            for (int k = 0; k < parts; k++) s += sums[group * parts + k][i];
            const int m = m0 + i / ROWS, n = quad * ROWS + i % ROWS;
            if (m < p.M && n < p.N) write_back(p, m, n, s);
        }
    }
}

// ---- tiles ---------------------------------------------------------------------------------------------------
constexpr int BK = 32, STAGES = 3, PIECES = BK / 4, MAX_SPLITS = 8;

__device__ __forceinline__ void copy_16(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;       // 0: the sixteen bytes are filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Bytes from one row of a stage to the next.  128 are used; with 144, eight rows one after another start in eight different
// groups of banks, and every address is a thread's own base plus a constant (an exclusive-or of row and piece instead cost
// 0.45 address instructions for each packed fma).
constexpr int PITCH = BK * 4 + 16;

template <int WM, int WN, int TN>
struct Tile {
    static constexpr int BM = WM * 32, BN = WN * 8 * TN, THREADS = WM * WN * 32;
    static constexpr int STAGE_BYTES = (BM + BN) * PITCH;
    static constexpr int SMEM = STAGES * STAGE_BYTES > BM * BN * 4 ? STAGES * STAGE_BYTES : BM * BN * 4;
};

// grid (tiles of N, tiles of M, splits); the blocks of one tile's splits are a cluster.
template <int WM, int WN, int TN>
__global__ void __launch_bounds__(WM * WN * 32)
gemm_f32_tile_kernel(const Product p) {
    using T = Tile<WM, WN, TN>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ty = lane >> 3, tx = lane & 7;
    const int wm = warp % WM, wn = warp / WM;
    const int n0 = blockIdx.x * T::BN, m0 = blockIdx.y * T::BM;
    const int splits = gridDim.z, split = blockIdx.z;
    const int steps_all = (p.K + BK - 1) / BK;
    const int first = (int)((long long)steps_all * split / splits), last = (int)((long long)steps_all * (split + 1) / splits);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    pdl_launch_dependents();

    // a thread copies one piece of the rows tid / PIECES + i * ROWS_APART of both operands; addresses behind the operands'
    // ends are formed and not read
    constexpr int ROWS_APART = T::THREADS / PIECES, A_COPIES = T::BM / ROWS_APART, W_COPIES = T::BN / ROWS_APART;
    const int copy_row = tid / PIECES, copy_k = tid % PIECES * 4;
    const float* a_src = p.a + (size_t)(m0 + copy_row) * p.lda + copy_k;
    const float* w_src = p.w + (size_t)(n0 + copy_row) * p.ldw + copy_k;
    const long long a_apart = (long long)ROWS_APART * p.lda, w_apart = (long long)ROWS_APART * p.ldw;
    const int a_rows = p.M - m0 - copy_row, w_rows = p.N - n0 - copy_row;       // rows there are, counted from copy_row
    const uint32_t copy_dst = base + copy_row * PITCH + copy_k * 4;
    auto load = [&](int step, bool a_too, bool w_too) {
        const int k0 = step * BK;
        const uint32_t stage = copy_dst + ((step - first) % STAGES) * T::STAGE_BYTES;
        const int a_there = k0 + copy_k < p.K ? a_rows : 0, w_there = k0 + copy_k < p.K ? w_rows : 0;
        if (w_too) {
#pragma unroll
            for (int i = 0; i < W_COPIES; i++)
                copy_16(stage + (T::BM + i * ROWS_APART) * PITCH, w_src + k0 + i * w_apart, i * ROWS_APART < w_there);
        }
        if (a_too) {
#pragma unroll
            for (int i = 0; i < A_COPIES; i++)
                copy_16(stage + i * ROWS_APART * PITCH, a_src + k0 + i * a_apart, i * ROWS_APART < a_there);
        }
    };
    // the weights of the first stages are written by no kernel: they come before the kernel in front has ended
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++)
        if (first + s < last) load(first + s, false, true);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (first + s < last) load(first + s, true, false);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    float2 acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = make_float2(0.0f, 0.0f);
    const int a_row = wm * 32 + ty, w_row = wn * 8 * TN + tx;
    for (int step = first; step < last; step++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        if (step + STAGES - 1 < last) load(step + STAGES - 1, true, true);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const unsigned char* stage = smem + ((step - first) % STAGES) * T::STAGE_BYTES;
        const unsigned char* a_piece = stage + a_row * PITCH;
        const unsigned char* w_piece = stage + (T::BM + w_row) * PITCH;
#pragma unroll
        for (int c = 0; c < PIECES; c++) {
            float4 av[8];
#pragma unroll
            for (int i = 0; i < 8; i++) av[i] = *reinterpret_cast<const float4*>(a_piece + 4 * i * PITCH + 16 * c);
#pragma unroll
            for (int j = 0; j < TN; j++) {
                const float4 wv = *reinterpret_cast<const float4*>(w_piece + 8 * j * PITCH + 16 * c);
#pragma unroll
                for (int i = 0; i < 8; i++) acc[i][j] = __ffma2_rn(low(av[i]), low(wv), acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; i++) acc[i][j] = __ffma2_rn(high(av[i]), high(wv), acc[i][j]);
            }
        }
    }
    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int m = m0 + a_row + 4 * i;
            if (m >= p.M) continue;
#pragma unroll
            for (int j = 0; j < TN; j++) {
                const int n = n0 + w_row + 8 * j;
                if (n < p.N) write_back(p, m, n, acc[i][j].x + acc[i][j].y);
            }
        }
        return;
    }
    // the blocks of the cluster leave their sums in their own shared memory; block r adds up every splits-th row
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float* mine = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) mine[(a_row + 4 * i) * T::BN + w_row + 8 * j] = acc[i][j].x + acc[i][j].y;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int at = tid; at < T::BM / splits * (T::BN / 4); at += T::THREADS) {
        const int row = at / (T::BN / 4) * splits + split, col = at % (T::BN / 4) * 4;
        if (m0 + row >= p.M) continue;
        float4 v[MAX_SPLITS];           // all on their way before the first is needed
#pragma unroll
        for (int r = 0; r < MAX_SPLITS; r++)
            if (r < splits) v[r] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(mine + row * T::BN + col, r));
        float4 s = v[0];
#pragma unroll
        for (int r = 1; r < MAX_SPLITS; r++) {
            if (r < splits) s = make_float4(s.x + v[r].x, s.y + v[r].y, s.z + v[r].z, s.w + v[r].w);
        }
        const float sums[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (n0 + col + c < p.N) write_back(p, m0 + row, n0 + col + c, sums[c]);
    }
    cluster.sync();         // nobody leaves while a peer may still read its shared memory
}

// ---- short k -------------------------------------------------------------------------------------------------
constexpr int SHORT_TILE = 16, SHORT_WARPS = 4, SHORT_K = 256;

// grid (tiles of N, tiles of M).  A warp takes every fourth piece of four k, a lane 2 x 4 outputs; the warps' sums are added in pairs.
__global__ void __launch_bounds__(SHORT_WARPS * 32)
gemm_f32_short_kernel(const Product p) {
    extern __shared__ __align__(16) float operands[];
    __shared__ float sums[SHORT_WARPS][SHORT_TILE][SHORT_TILE + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * SHORT_TILE, m0 = blockIdx.y * SHORT_TILE;
    const int pieces = p.K / 4, pitch = p.K + 4;            // eight rows one after another start in eight groups of banks
    float* as = operands;
    float* ws = operands + SHORT_TILE * pitch;
    pdl_launch_dependents();
    auto bring = [&](float* to, const float* from, int ld, int rows) {
        for (int i = tid; i < SHORT_TILE * pieces; i += SHORT_WARPS * 32) {
            const int row = i / pieces, at = i % pieces * 4;
            copy_16((uint32_t)__cvta_generic_to_shared(to + row * pitch + at), from + (size_t)(row < rows ? row : 0) * ld + at, row < rows);
        }
    };
    bring(ws, p.w + (size_t)n0 * p.ldw, p.ldw, p.N - n0);       // weights are written by no kernel
    pdl_wait();
    bring(as, p.a + (size_t)m0 * p.lda, p.lda, p.M - m0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int ty = lane >> 2, tx = lane & 3;
    float2 acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll 4
    for (int c = warp; c < pieces; c += SHORT_WARPS) {
        float4 av[2], wv[4];
#pragma unroll
        for (int i = 0; i < 2; i++) av[i] = *reinterpret_cast<const float4*>(as + (ty + 8 * i) * pitch + 4 * c);
#pragma unroll
        for (int j = 0; j < 4; j++) wv[j] = *reinterpret_cast<const float4*>(ws + (tx + 4 * j) * pitch + 4 * c);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(high(av[i]), high(wv[j]), __ffma2_rn(low(av[i]), low(wv[j]), acc[i][j]));
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) sums[warp][ty + 8 * i][tx + 4 * j] = acc[i][j].x + acc[i][j].y;
    __syncthreads();
    for (int i = tid; i < SHORT_TILE * SHORT_TILE; i += SHORT_WARPS * 32) {
        const int row = i / SHORT_TILE, col = i % SHORT_TILE;
        const float v = (sums[0][row][col] + sums[1][row][col]) + (sums[2][row][col] + sums[3][row][col]);
        if (m0 + row < p.M && n0 + col < p.N) write_back(p, m0 + row, n0 + col, v);
    }
}

int launch_short(const Product& p, cudaStream_t stream) {
    const dim3 grid((p.N + SHORT_TILE - 1) / SHORT_TILE, (p.M + SHORT_TILE - 1) / SHORT_TILE);
    return sandy_launch(gemm_f32_short_kernel, grid, dim3(SHORT_WARPS * 32), (size_t)2 * SHORT_TILE * (p.K + 4) * 4, stream, p);
}

template <int MB, int AHEAD, int BLOCKS>
int launch_stream(const Product& p, cudaStream_t stream) {
    // Groups of four rows of w in a block: few enough that there are blocks for every SM; the warps left over share k.
    const int quads = (p.N + ROWS - 1) / ROWS, steps = (p.K + STEP - 1) / STEP, m_blocks = (p.M + MB - 1) / MB;
    const int resident = std::max(1, BLOCKS * sandy_sm_count() / m_blocks);
    int groups = STREAM_WARPS;
    while (groups > 1 && (quads + groups - 1) / groups < resident) groups /= 2;
    const int parts = std::max(1, std::min(STREAM_WARPS / groups, steps));
    dim3 grid(m_blocks, std::min((quads + groups - 1) / groups, resident)), block(32, parts, groups);
    return sandy_launch(gemm_f32_stream_kernel<MB, AHEAD, BLOCKS>, grid, block, 0, stream, p);
}

// Up to here the weights are streamed (alone, weights from HBM, us, stream / best tile: 24 rows 768 x 768 4.0 / 5.7, 3,072 x
// 768 8.4 / 11.4, 768 x 3,072 8.9 / 15.3, 50,257 x 768 99 / 120; 28 rows 5.7 / 5.8, 12.7 / 11.5, 14.7 / 15.4, 125 / 121).
constexpr int STREAM_MAX_ROWS = 24;

// SMs that clusters of s blocks, one block an SM, can cover: groups of SMs that share a crossbar are not all multiples of s
// (144 blocks in clusters of 4 took two rounds where the same blocks two an SM took one).
int coverable(int s) {
    const int sms = sandy_sm_count();
    return s <= 2 ? sms : s == 4 ? sms * 9 / 10 : sms * 8 / 10;
}

template <int WM, int WN, int TN>
int launch_tile(const Product& p, int splits, cudaStream_t stream) {
    using T = Tile<WM, WN, TN>;
    constexpr int SM_BYTES = 220 * 1024;
    const cudaError_t set = cudaFuncSetAttribute(gemm_f32_tile_kernel<WM, WN, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_BYTES);
    if (set != cudaSuccess) return (int)set;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + T::BN - 1) / T::BN, (p.M + T::BM - 1) / T::BM, splits);
    // The blocks of a cluster may be stacked on one SM while others idle: each asks for as much shared memory as leaves no
    // room for more of them than an SM has to take.
    const int sms = coverable(splits), blocks = cfg.gridDim.x * cfg.gridDim.y * splits, share = (blocks + sms - 1) / sms;
    cfg.dynamicSmemBytes = std::max(T::SMEM, SM_BYTES / share - 2048);
    cfg.blockDim = dim3(T::THREADS);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = splits;
        n++;
    }
    if (sandy_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<WM, WN, TN>, p);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// Which tile, in how many parts of k.  A block is as fast as the blocks beside it on its SM let it be: for 768 k, one, two
// and three blocks of 64 x 64 on an SM take 30, 49 and 68 us, one and two of 64 x 128 48 and 84, one of 128 x 128 82; more
// than that take turns.  A block's start counts as 16 k more, a cluster's exchange as 24.
int choose(int M, int N, int K, int& splits) {
    struct Shape { int bm, bn, together; float us[3]; };
    const Shape shapes[3] = {{128, 128, 1, {82, 0, 0}}, {64, 128, 2, {48, 84, 0}}, {64, 64, 3, {30, 49, 68}}};
    float best = 0.0f;
    int which = 0;
    splits = 1;
    for (int i = 0; i < 3; i++) {
        const Shape& h = shapes[i];
        const long long tiles = (long long)((N + h.bn - 1) / h.bn) * ((M + h.bm - 1) / h.bm);
        for (int s = 1; s <= MAX_SPLITS; s *= 2) {
            if (s > 1 && K / s < 64) break;
            const long long blocks = (tiles * s + coverable(s) - 1) / coverable(s);         // on the busiest SM
            const float us = blocks <= h.together ? h.us[blocks - 1] : h.us[h.together - 1] * (float)blocks / h.together;
            const float cost = us * ((float)K / s + (s > 1 ? 40.0f : 16.0f));
            if (best == 0.0f || cost < best) {
                best = cost;
                which = i;
                splits = s;
            }
        }
    }
    return which;
}

}  // namespace

// a: [M, K] (row stride lda), w: [N, K] (row stride ldw), bias: [N] or null, residual: [M, N] (row stride ldr) or null,
// out: [M, N] (row stride ldc), which may be the residual itself; all float32, strides in elements.  K, lda and ldw are
// multiples of 4, a and w start on 16-byte boundaries.  form: 0 the rule's choice; 1 stream; 2, 3, 4 a tile of 128 x 128,
// 64 x 128, 64 x 64 in `splits` parts of k (1, 2, 4 or 8); 5 short (K up to 256).
SANDY_API int sandy_gemm_f32(const float* a, const float* w, const float* bias, const float* residual, float* out, int M, int N,
                             int K, int lda, int ldw, int ldr, int ldc, int act, int form, int splits, cudaStream_t stream) {
    if (M == 0 || N == 0) return SANDY_OK;
    if (!a || !w || !out || K <= 0 || M < 0 || N < 0) return SANDY_ERR_ARGUMENT;
    if (K % 4 || lda % 4 || ldw % 4 || ((uintptr_t)a & 15) || ((uintptr_t)w & 15)) return SANDY_ERR_UNSUPPORTED;
    const Product p = {a, w, bias, residual, out, M, N, K, lda, ldw, ldr, ldc, act};
    if (form == 0) {
        if (M <= STREAM_MAX_ROWS) form = 1;
        else form = 2 + choose(M, N, K, splits);
    } else if (form > 1 && form < 5 && (splits < 1 || splits > MAX_SPLITS || (splits & (splits - 1)))) {
        return SANDY_ERR_ARGUMENT;
    }
    if (form == 5) {
        if (K > SHORT_K || (M + SHORT_TILE - 1) / SHORT_TILE > 65535) return SANDY_ERR_UNSUPPORTED;
        return launch_short(p, stream);
    }
    if (form == 1) {
        if (M == 1) return launch_stream<1, 4, 2>(p, stream);
        if (M == 2) return launch_stream<2, 4, 2>(p, stream);
        if (M <= 4) return launch_stream<4, 3, 2>(p, stream);
        return launch_stream<8, 2, 2>(p, stream);
    }
    if (form == 2) return launch_tile<4, 2, 8>(p, splits, stream);
    if (form == 3) return launch_tile<2, 2, 8>(p, splits, stream);
    if (form == 4) return launch_tile<2, 2, 4>(p, splits, stream);
    return SANDY_ERR_ARGUMENT;
}
