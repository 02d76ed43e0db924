// Matrix product of float32 operands on the tensor cores, each operand in three bfloat16 pieces (split_f32.cuh), for weights
// stored [N, K] whose rows start on 16-byte boundaries, with bias / activation / residual folded into the write-back.
//
//   out[m, n] = act( sum_k a[m, k] * w[n, k] + bias[n] ) + residual[m, n]
//
// The same with one matrix per expert: rows of a and out in the routing's sorted order (as in grouped_gemm_tc.cu), 16 experts, 1,024 x
// 768, us, the fma tiles of grouped_gemm.cu -> this kernel: 80 slots 59 -> 23, 2,048 slots 105 -> 46.
//
// A block computes a tile of 128 x BN outputs, or a part of its k; the blocks of a tile's parts are a cluster.
//   warp 17       brings the float operands by TMA, a chunk of 64 k a stage of two
//   warps 0..15   split them: a's pieces go to tensor memory (a thread one row), w's to shared memory (128-byte swizzle); then add
//                 the accumulator of the chunk before into registers (a warp the lanes it may read, a quarter of the columns)
//   warp 16       allocates tensor memory (two accumulators, two stages of a's pieces); one lane issues a chunk's 24 tcgen05.mma
// Pieces and accumulators are written again two chunks later, when every warp has waited for the products that used them.
// Then the sums go through shared memory (and across the cluster, in the order of the parts), and all rows are written back.
// What bounds it: a chunk of 128 x 128 takes 1.1 us where its instructions take 0.8 (splitting 16 K floats costs the sixteen warps
// nearly as many issue slots), and a block 7 us beside its chunks.  a's pieces are in tensor memory because a product of two
// operands in shared memory reads 128 bytes a clock there, all there is (a chunk 1.8 us); the floats come by TMA, as loads through
// registers pass the same memory (1.4).  Alone, bias folded in, weights from HBM, us, the fma tiles of gemm_f32.cu -> this kernel:
// 2,048 rows, 2,304 x 768 167 -> 48 (151 TFLOP/s), 768 x 768 70 -> 20, 3,072 x 768 250 -> 71, 768 x 3,072 241 -> 55 (176 TFLOP/s
// of the 278 that a sixth of the measured bfloat16 rate is); 128 rows, 3,072 x 768 21 -> 11; 64 rows, 50,257 x 768 137 -> 76.
// Error against 64 bits (2-norm), fma kernels -> this one.  Operands of both signs, or one of them: 1.1e-7 -> 0.8e-7 (k 64),
// 1.4e-7 to 1.9e-7 -> 0.9e-7 (768), 2.6e-7 -> 1.1e-7 (3,072).  Operands all of one sign, which the additions towards zero shrink
// (split_f32.cuh): 0.7e-7 -> 0.8e-7 to 0.9e-7 (64), 0.5e-7 to 0.7e-7 -> 0.9e-7 (768 and 3,072), 0.8e-7 -> 0.9e-7 to 1.0e-7 (6,400).
// What is not finite, 2,048 x 2,304 x 768, us: finite 50; a NaN in one row of a 52, in every row 131, in one of w 62; infinities in every
// row of a 960 (the fma tiles 169 throughout).
// Every wait on an mbarrier is bounded: on expiry the kernel raises `*status`, stops issuing, frees its tensor memory and
// returns.
#include <cooperative_groups.h>

#include <algorithm>

#include "split_f32.cuh"

namespace cg = cooperative_groups;

namespace {

struct Product {
    const float* a;
    const float* w;
    const float* bias;
    const float* residual;
    float* out;
    int M, N, K, lda, ldw, ldr, ldc, act;
    int wide;               // rows of out and residual start on 16-byte boundaries
    const int* group_start; // a matrix per expert: where each expert's rows start, on the device
    int groups;
};

// PLAIN: one matrix.  EXPERTS: expert g has the rows g * N .. of w and the rows group_start[g] .. group_start[g + 1] - 1 of a and out;
// the grid covers the worst case of tiles, and blocks behind the step's last tile leave at once.  (A matrix per head, k 64 to 128, as a
// third kind was no faster than the fma tiles: a block's start is most of so short a sum.)
enum Kind { PLAIN, EXPERTS };

constexpr int WORKERS = 16, THREADS = (WORKERS + 2) * 32, MAX_PARTS = 8;

template <int BN>
struct Layout {
    static constexpr int A_HALF = BM * 128, W_HALF = BN * 128;          // 32 of a chunk's floats of every row, as TMA lays them down
    static constexpr int RAW = 2 * (A_HALF + W_HALF);
    static constexpr int W_PIECE = BN * 128, PIECES = N_PIECES * W_PIECE;
    static constexpr int PITCH = BN + 4;        // floats a row of the tile of sums: eight rows start in eight groups of banks
    static constexpr int SUMS = BM * PITCH * 4;
    static constexpr int BODY = 2 * (RAW + PIECES);
    static constexpr int SMEM = BODY + 1024 + 128;      // alignment, barriers
    static constexpr int A_COL = 2 * BN, A_COLS = N_PIECES * CHUNK / 2;         // in tensor memory, behind the accumulators
    static_assert(SUMS <= BODY && A_COL + 2 * A_COLS <= 512, "the sums reuse the stages; 512 columns there are");
};

template <int BN, Kind KIND>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const Product p,
                   int* __restrict__ status) {
    using L = Layout<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* pieces = smem + 2 * L::RAW;
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + L::BODY);   // [2] a stage's floats are there
    uint64_t* raw_empty = raw_full + 2;                                 // [2] ... have been read
    uint64_t* full = raw_empty + 2;                                     // [2] a stage's pieces are there
    uint64_t* done = full + 2;                                          // [2] the products of a stage are done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 2);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * BN;
    const int parts = gridDim.z, part = blockIdx.z;
    int group = 0, m0 = blockIdx.y * BM, m_end = p.M;
    if (KIND == EXPERTS) {
        pdl_wait();             // the groups' borders come from a kernel before
        int tile = blockIdx.y;
        m0 = p.group_start[0];
        for (; group < p.groups; group++) {
            m_end = p.group_start[group + 1];
            const int tiles = (m_end - m0 + BM - 1) / BM;
            if (tile < tiles) break;
            tile -= tiles;
            m0 = m_end;
        }
        if (group == p.groups) return;          // every thread of a cluster's blocks alike
        m0 += tile * BM;
    }
    const int w_row0 = group * p.N + n0;
    const int chunks_all = (p.K + CHUNK - 1) / CHUNK;
    const int first = (int)((long long)chunks_all * part / parts), chunks = (int)((long long)chunks_all * (part + 1) / parts) - first;

    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], WORKERS);
            mbar_init(&full[s], WORKERS);
            mbar_init(&done[s], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WORKERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();

    if (warp < WORKERS) {
        const int quarter = warp & 3, quad = warp >> 2;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        // a: a thread takes sixteen k (those of its warp's quad) of its row
        // w: an item is eight rows and the 32 k of a half, a thread eight k; lanes 0..3 and 4..7 take the rows r and r ^ 5, so that
        // eight lanes meet no bank twice, neither where they read floats (even or odd pieces of 16 bytes) nor where they write pieces
        constexpr int ITEMS = BN / 4, ROUNDS = (ITEMS + WORKERS - 1) / WORKERS;
        const int w_row = (lane & 4) ? (lane >> 3) ^ 5 : lane >> 3, w_k = lane & 3;
        uint32_t w_even[ROUNDS], w_piece[ROUNDS];           // where an item's first float4 and its first piece lie in their stages
#pragma unroll
        for (int i = 0; i < ROUNDS; i++) {
            const int item = warp + i * WORKERS, half = item & 1, row = (item >> 1) * 8 + w_row;
            w_even[i] = 2 * L::A_HALF + half * L::W_HALF + row * 128 + (((2 * w_k) ^ w_row) << 4);
            w_piece[i] = row * 128 + (((4 * half + w_k) ^ w_row) << 4);
        }
        uint32_t a_at[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            a_at[j] = (quad >> 1) * L::A_HALF + (quarter * 32 + lane) * 128 + ((((quad & 1) * 4 + j) ^ (lane & 7)) << 4);
        constexpr int COLS = BN / 4;
        float sum[COLS];
#pragma unroll
        for (int j = 0; j < COLS; j++) sum[j] = 0.0f;
        bool ok = true;
        auto split = [&](int c, int s) {
            ok = mbar_wait(&raw_full[s], (c >> 1) & 1);
            if (!ok) {
                if (lane == 0 && status) atomicOr(status, 1);
                return;
            }
            const uint8_t* raw = smem + s * L::RAW;
            uint8_t* to = pieces + s * L::PIECES;
#pragma unroll
            for (int i = 0; i < ROUNDS; i++) {
                if (ITEMS % WORKERS && i + 1 == ROUNDS && warp + i * WORKERS >= ITEMS) break;
                const float4 x = *reinterpret_cast<const float4*>(raw + w_even[i]);
                const float4 y = *reinterpret_cast<const float4*>(raw + (w_even[i] ^ 16));
                uint4 piece[N_PIECES];
                split_eight(x, y, piece);
#pragma unroll
                for (int j = 0; j < N_PIECES; j++) *reinterpret_cast<uint4*>(to + w_piece[i] + j * L::W_PIECE) = piece[j];
            }
            float4 x[4];
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] = *reinterpret_cast<const float4*>(raw + a_at[j]);
            uint4 low[N_PIECES], high[N_PIECES];
            split_eight(x[0], x[1], low);
            split_eight(x[2], x[3], high);
#pragma unroll
            for (int j = 0; j < N_PIECES; j++)
                tmem_st_32x8(tmem + lanes + L::A_COL + s * L::A_COLS + j * (CHUNK / 2) + quad * 8, low[j], high[j]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");        // my pieces, before the tensor core reads them
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[s]);
                mbar_arrive(&raw_empty[s]);
            }
        };
        auto add = [&](int c, int s) {
            ok = mbar_wait(&done[s], (c >> 1) & 1);
            if (!ok && lane == 0 && status) atomicOr(status, 4);
            tc_fence_after();
            uint32_t r[COLS];
#pragma unroll
            for (int j = 0; j < COLS; j += 8) tmem_ld_32x8(tmem + lanes + s * BN + quad * COLS + j, *reinterpret_cast<uint32_t (*)[8]>(r + j));
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < COLS; j++) sum[j] += __uint_as_float(r[j]);
            tc_fence_before();
        };
        split(0, 0);
        for (int c = 1; c < chunks && ok; c += 2) {
            split(c, 1);
            if (ok) add(c - 1, 0);
            if (c + 1 < chunks && ok) {
                split(c + 1, 0);
                if (ok) add(c, 1);
            }
        }
        if (ok) add(chunks - 1, (chunks - 1) & 1);
        // the last products are done, so nothing reads the stages any more (no copy is under way either: every chunk was waited for)
        float* mine = reinterpret_cast<float*>(smem) + (quarter * 32 + lane) * L::PITCH + quad * COLS;
        if (ok) {
#pragma unroll
            for (int j = 0; j < COLS; j += 4)
                *reinterpret_cast<float4*>(mine + j) = make_float4(UNSCALE * sum[j], UNSCALE * sum[j + 1], UNSCALE * sum[j + 2], UNSCALE * sum[j + 3]);
        }
        pdl_wait();         // for the write-back: out and residual may still be in use by the kernel before
    } else if (warp == WORKERS) {
        if (elect_one()) {
            constexpr uint32_t idesc = make_instr_desc(BN);
            for (int c = 0; c < chunks; c++) {
                const int s = c & 1;
                if (!mbar_wait(&full[s], (c >> 1) & 1)) {
                    if (status) atomicOr(status, 2);
                    break;
                }
                tc_fence_after();
                issue_chunk(tmem + s * BN, tmem + L::A_COL + s * L::A_COLS, smem_u32(pieces + s * L::PIECES), L::W_PIECE, idesc);
                umma_commit(&done[s]);
            }
        }
    } else if (elect_one()) {
        auto load_w = [&](int c) {
            uint8_t* raw = smem + (c & 1) * L::RAW + 2 * L::A_HALF;
            mbar_expect_tx(&raw_full[c & 1], L::RAW);
            for (int half = 0; half < 2; half++)
                tma_load_2d(raw + half * L::W_HALF, &map_w, (first + c) * CHUNK + 32 * half, w_row0, &raw_full[c & 1]);
        };
        auto load_a = [&](int c) {
            uint8_t* raw = smem + (c & 1) * L::RAW;
            for (int half = 0; half < 2; half++)
                tma_load_2d(raw + half * L::A_HALF, &map_a, (first + c) * CHUNK + 32 * half, m0, &raw_full[c & 1]);
        };
        for (int c = 0; c < min(chunks, 2); c++) load_w(c);         // weights are written by no kernel
        pdl_wait();
        for (int c = 0; c < chunks; c++) {
            if (c >= 2) {
                if (!mbar_wait(&raw_empty[c & 1], ((c >> 1) & 1) ^ 1)) {
                    if (status) atomicOr(status, 1);
                    break;
                }
                load_w(c);
            }
            load_a(c);
        }
    }
    __syncwarp();
    tc_fence_before();
    if (parts > 1) cg::this_cluster().sync();
    else __syncthreads();

    if (warp == WORKERS) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    } else if (warp < WORKERS) {
        // block r of a cluster adds up and writes every parts-th row
        constexpr int PER_ROW = BN / 4, WRITERS = WORKERS * 32;
        float* sums = reinterpret_cast<float*>(smem);
        const int total = BM / parts * PER_ROW;
        int nan_row = -1;           // the row of a in which this warp last found a NaN: all its sums are one
        for (int base = 0; base < total; base += WRITERS) {
            const int at = base + tid;
            const int row = at / PER_ROW * parts + part, col = at % PER_ROW * 4;
            const int m = m0 + row, n = n0 + col;
            const bool live = at < total && m < m_end && n < p.N;
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (live) {
                float* src = sums + row * L::PITCH + col;
                float4 s;
                if (parts == 1) {
                    s = *reinterpret_cast<const float4*>(src);
                } else {
                    cg::cluster_group cluster = cg::this_cluster();
                    float4 t[MAX_PARTS];            // all on their way before the first is needed
#pragma unroll
                    for (int r = 0; r < MAX_PARTS; r++)
                        if (r < parts) t[r] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(src, r));
                    s = t[0];
#pragma unroll
                    for (int r = 1; r < MAX_PARTS; r++)
                        if (r < parts) s = make_float4(s.x + t[r].x, s.y + t[r].y, s.z + t[r].z, s.w + t[r].w);
                }
                v[0] = s.x; v[1] = s.y; v[2] = s.z; v[3] = s.w;
            }
            bool odd = false;
#pragma unroll
            for (int e = 0; e < 4; e++) odd |= live && n + e < p.N && !is_finite(v[e]);
            for (unsigned again = __ballot_sync(0xffffffffu, odd); again; again &= again - 1) {
                const int who = __ffs(again) - 1, mm = __shfl_sync(0xffffffffu, m, who), nn = __shfl_sync(0xffffffffu, n, who);
                float plain[4] = {NAN, NAN, NAN, NAN};
                if (mm != nan_row && plain_sums(p.a + (size_t)mm * p.lda, p.w + (size_t)(w_row0 - n0 + nn) * p.ldw, p.ldw, min(4, p.N - nn), p.K, plain))
                    nan_row = mm;
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (lane == who && !is_finite(v[e])) v[e] = plain[e];
            }
            if (!live) continue;
            float* out = p.out + (size_t)m * p.ldc + n;
            const float* residual = p.residual ? p.residual + (size_t)m * p.ldr + n : nullptr;
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (n + e < p.N) v[e] = apply_act(p.bias ? v[e] + p.bias[n + e] : v[e], p.act);
            if (p.wide && n + 4 <= p.N) {
                if (residual) {
                    const float4 r = *reinterpret_cast<const float4*>(residual);
                    v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
                }
                *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (n + e < p.N) out[e] = residual ? v[e] + residual[e] : v[e];
            }
        }
    }
    if (parts > 1) cg::this_cluster().sync();         // nobody leaves while a peer may still read its shared memory
}

// row_tiles: the grid's tiles of 128 rows; w_rows: the rows of w.
template <int BN, Kind KIND>
int launch(const Product& p, int row_tiles, int parts, long long w_rows, int* status, cudaStream_t stream) {
    using L = Layout<BN>;
    const cudaError_t set = cudaFuncSetAttribute(gemm_f32_tc_kernel<BN, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (set != cudaSuccess) return (int)set;
    CUtensorMap map_a, map_w;
    if (!get_map(p.a, p.M, p.K, p.lda, BM, &map_a, 4) || !get_map(p.w, w_rows, p.K, p.ldw, BN, &map_w, 4)) return SANDY_ERR_ARGUMENT;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + BN - 1) / BN, row_tiles, parts);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = L::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (parts > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = parts;
        n++;
    }
    if (sandy_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel<BN, KIND>, map_a, map_w, p, status);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

template <Kind KIND>
int launch_tile(int tile, const Product& p, int row_tiles, int parts, long long w_rows, int* status, cudaStream_t stream) {
    if (row_tiles > 65535) return SANDY_ERR_UNSUPPORTED;
    if (tile == 64) return launch<64, KIND>(p, row_tiles, parts, w_rows, status, stream);
    if (tile == 96) return launch<96, KIND>(p, row_tiles, parts, w_rows, status, stream);
    if (tile == 128) return launch<128, KIND>(p, row_tiles, parts, w_rows, status, stream);
    return SANDY_ERR_ARGUMENT;
}

// SMs that clusters of `parts` blocks, one block an SM, can cover (groups of SMs that share a crossbar are not all multiples).
int coverable(int parts) {
    const int sms = sandy_sm_count();
    return parts <= 2 ? sms : parts == 4 ? sms * 9 / 10 : sms * 8 / 10;
}

// Which tile, in how many parts of k.  A block takes the SM to itself.  Its time is a start and a write-back, and a time for each
// chunk that grows with the tile's columns by less than they do (the splitting of a's 128 rows is the rest): fitted to 1,500
// measured (shape, tile, parts) of 26 to 2,048 rows, of which the choice meets the best within 0.4 % on average.
void choose(long long row_tiles, int N, int K, int& tile, int& parts) {
    struct Shape { int columns; float chunk_us, block_us; };
    const Shape shapes[3] = {{64, 0.92f, 4.8f}, {96, 1.05f, 6.0f}, {128, 1.21f, 6.9f}};
    const int chunks = (K + CHUNK - 1) / CHUNK;
    float best = 0.0f;
    for (const Shape& h : shapes) {
        const long long tiles = (long long)((N + h.columns - 1) / h.columns) * row_tiles;
        for (int p = 1; p <= MAX_PARTS && p <= chunks; p *= 2) {
            const long long rounds = (tiles * p + coverable(p) - 1) / coverable(p);
            const float cost = (float)rounds * ((float)((chunks + p - 1) / p) * h.chunk_us + h.block_us);
            if (best == 0.0f || cost < best) {
                best = cost;
                tile = h.columns;
                parts = p;
            }
        }
    }
}

}  // namespace

// a: [M, K] (row stride lda), w: [N, K] (row stride ldw), bias: [N] or null, residual: [M, N] (row stride ldr) or null,
// out: [M, N] (row stride ldc), which may be the residual itself; all float32, strides in elements.  K, lda and ldw are
// multiples of 4, a and w start on 16-byte boundaries.  tile: columns of a tile (64, 96, 128), its k in `parts` (1, 2, 4, 8);
// 0, 0: the rule's choice.
// status: a device int for expired waits, or null.
SANDY_API int sandy_gemm_f32_tc(const float* a, const float* w, const float* bias, const float* residual, float* out, int M, int N,
                                int K, int lda, int ldw, int ldr, int ldc, int act, int tile, int parts, int* status,
                                cudaStream_t stream) {
    if (M == 0 || N == 0) return SANDY_OK;
    if (!a || !w || !out || K <= 0 || M < 0 || N < 0) return SANDY_ERR_ARGUMENT;
    if (K % 4 || lda % 4 || ldw % 4 || ((uintptr_t)a & 15) || ((uintptr_t)w & 15)) return SANDY_ERR_UNSUPPORTED;
    if (tile == 0 && parts == 0) choose((M + BM - 1) / BM, N, K, tile, parts);
    if (parts < 1 || parts > MAX_PARTS || (parts & (parts - 1)) || parts > (K + CHUNK - 1) / CHUNK) return SANDY_ERR_ARGUMENT;
    const bool wide = !((uintptr_t)out & 15) && ldc % 4 == 0 && (!residual || (!((uintptr_t)residual & 15) && ldr % 4 == 0));
    const Product p = {a, w, bias, residual, out, M, N, K, lda, ldw, ldr, ldc, act, wide ? 1 : 0, nullptr, 1};
    return launch_tile<PLAIN>(tile, p, (M + BM - 1) / BM, parts, N, status, stream);
}

// Per expert: a [n_slots, K] with the rows of an expert one after another, w [G * N, K], group_start int32 [G + 1] on the device; act: 0
// none, 1 the square of relu.
SANDY_API int sandy_expert_product_f32_tc(const float* a, int lda, const float* w, int ldw, float* out, int ldo, int n_slots, int n_groups,
                                          int N, int K, const int* group_start, int act, int* status, cudaStream_t stream) {
    if (n_slots == 0 || n_groups == 0 || N == 0) return SANDY_OK;
    if (!a || !w || !out || !group_start || K <= 0 || n_slots < 0 || n_groups < 0 || N < 0) return SANDY_ERR_ARGUMENT;
    if (K % 4 || lda % 4 || ldw % 4 || ((uintptr_t)a & 15) || ((uintptr_t)w & 15)) return SANDY_ERR_UNSUPPORTED;
    const bool wide = !((uintptr_t)out & 15) && ldo % 4 == 0;
    const Product p = {a, w, nullptr, nullptr, out, n_slots, N, K, lda, ldw, 0, ldo, act == 1 ? SANDY_ACT_RELU_SQUARED : SANDY_ACT_NONE, wide ? 1 : 0,
                       group_start, n_groups};
    // as many tiles as evenly spread rows would have
    const long long spread = (long long)n_groups * (((n_slots + n_groups - 1) / n_groups + BM - 1) / BM);
    int tile, parts;
    choose(std::min<long long>(spread, n_slots), N, K, tile, parts);
    return launch_tile<EXPERTS>(tile, p, (n_slots + BM - 1) / BM + n_groups, parts, (long long)n_groups * N, status, stream);
}
