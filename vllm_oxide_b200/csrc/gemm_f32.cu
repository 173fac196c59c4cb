// True 32-bit matrix product: C[M, N] = A[M, K] * W[N, K]^T (+ bias), float32 in, float32 FMA, float32 out. No tensor cores, no
// TF32. This is the matrix product of the 32-bit engine; it exists to show faults that bfloat16 rounding would hide.
// Reference op: crates/engine/src/backend/cpu/mod.rs:199-229 (x * W^T with W [out, in]).
//
// The sum over k is the same in every kernel here, to the bit: K is cut into chunks of 128; a chunk is two chains of FMAs, over
// its even and its odd k in order, each starting from zero, and their sum; (number of chunks / 8, rounded up) chunks make a
// segment, whose chunks are added in order; the segments are added in order. An element therefore does not depend on M, on
// its row's place in the batch, on which kernel computes it or over how many blocks K is shared. (One chain over all of K
// rounds more often: relative error against 64 bits on normal values 8.1e-7 and 1.6e-6 at K = 2,048 and 8,192, here 1.6e-7 and 1.7e-7.)
//
// Two kernels:
//  * few rows (decode steps: M <= 8, M <= 16 while K is at most 4,096, eight at a time where `by_eights` says): bound by reading W once, 6.9 TB/s at
//    M = 1, 5.2 at 8 and 2.7 at 16 on 128,256 x 2,048, 5.5, 4.5 and 2.4 TB/s on 16,384 x 2,048 back to back (64 x 64 tiles, which served every M
//    before: 1.06 and 0.6 TB/s; 0.1 TB/s on 2,048 x 8,192, now 3.6 at eight rows). A thread has one or two weight rows and a chunk, all rows of A
//    in its registers' sums; weights arrive by cp.async into a ring per warp, so that no barrier of the block stands in the stream.
//  * tiles (everything else): bound by what two warps a scheduler can issue: the FMA units are busy 60 % of the cycles, shared memory
//    48 %, and a warp waits for the result in front or for a register's read most of the rest. 8 x 8 outputs a thread from
//    shared memory: 40 to 42 TFLOP/s on 16,384 x 2,048 at M = 1,250 and 2,048 (33 and 34 before), 33 TFLOP/s on 2,048 x 8,192 at M = 128 (6).
// Both multiply and add pairs of k in one instruction (fma.rn.f32x2, each half rounded as fmaf rounds it): single FMAs
// reach half the rate on this GPU (a tile kernel of 8 x 8 outputs a thread: 37 TFLOP/s with fmaf).
#include "common.cuh"
#include <cmath>
#include <cooperative_groups.h>
VOB_PDL_SWITCH(gemm_f32)

namespace cg = cooperative_groups;

namespace {

constexpr int CHUNK = 128;

// 16 bytes from global to shared memory, of which `bytes` are read and the rest is zero.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// (d0, d1) += (a0, a1) * (b0, b1): two float32 FMAs, each rounded as fmaf rounds it, in one instruction.
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(unsigned long long d) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
    return lo + hi;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Chunks of a segment.
__host__ __device__ constexpr int seg_chunks(int nc) { return (nc + 7) / 8; }

// ------------------------------------------------------------------------------------------------ few rows
// A block takes 64 weight rows and `q` chunks of K, four chunks at a time: a warp has one of the four and 32 of the rows (a lane
// one row, RN = 1, 8 warps) or all 64 (a lane two, RN = 2, 4 warps: from 5 rows of A on, where reading A from shared memory is
// what costs). A cluster of `c` blocks shares a row's K; each block leaves the sums of its chunks in its shared memory and the
// cluster adds them up, each block a part of the outputs. (Clusters that stay and take one set of 64 rows after another, the
// ring running on over them, are slower: 291 against 214 us at M = 1, 128,256 x 2,048. Their blocks meet twice a set.)
constexpr int FEW_N = 64, FEW_K = 32;                 // weight rows of a block, k of a ring stage

constexpr int few_rows_a_lane(int mb) { return mb <= 4 ? 1 : 2; }
// three blocks an SM (two from three rows of A on) for four chunks a block
__host__ __device__ constexpr int few_blocks(int mb) { return mb <= 2 ? 3 : 2; }
// Shared memory of a block that adds up `chunks` chunks: its warps' rings, x of four chunks, the chunks' sums.
constexpr size_t few_smem(int mb, int chunks, int stages) {
    return sizeof(float) * (size_t)(8 * stages * 32 * FEW_K + 4 * CHUNK * mb + chunks * mb * FEW_N);
}
constexpr size_t FEW_SMEM_MOST = 200 * 1024;
constexpr int few_registers(int rows) { return rows <= 2 ? rows : rows <= 4 ? 4 : rows <= 8 ? 8 : 16; }      // MB of `rows` rows

// Chunks of a block, a multiple of four: an eighth of K at least (a cluster holds eight blocks); all of it, half of it or, with one or two
// rows, a quarter, where 256 blocks are left and two of them find room on an SM. A block's start, its cluster's meeting and its end cost as much as
// four chunks of weights do. Cold, back to back, us with an eighth / now, 1, 4 and 8 rows: 16,384 x 2,048 26.5, 35, 38 / 23.7, 25.6, 29.5;
// 128,256 x 2,048 162, 233, 255 / 151, 164, 202; 28,672 x 4,096 91, 131, 142 / 82, 94, 111. Three blocks to a K of 32 chunks (6,144 x 4,096)
// lose from three rows on: 32.5 / 39 at eight. With one and two rows a last wave that is nearly empty takes back more than that: where the
// longer blocks would fill less than 0.7 of their waves K stays in eighths, or in the next smaller part (two rows, us, eighths / longer:
// 6,144 x 8,192, 1.3 waves, 39.3 / 46.5; 11,008 x 8,192, 1.2 waves of halves, 72.4 / 80.6; 22,016 x 2,560, 1.2 waves, 44.1 / 47.8; just above
// one wave, as at 0.7 to 0.8, they gain or are equal). From three rows on they gain there, too (11,008 x 4,096, 1.2 waves, at 4 and 8 rows 53, 60 / 44, 51).
//
// Stages of a warp's ring: two, and three for three and four rows whose blocks did not get longer, where that leaves two blocks an SM and at most two
// waves, or one block an SM and at most 120 blocks (clusters of eight one to an SM do not find the last places): there a warp's latency is
// not hidden by others. Three / two, us, 4 rows: 3,072 x 1,024 5.5 / 6.2, 1,024 x 8,960 16.1 / 19.6, 896 x 14,336 22 / 27; beyond, 49,152 x 1,280
// 67.3 / 65.1, 1,024 x 11,008 32.9 / 20.8, 4,100 x 14,336 109 / 60. One and two rows have three blocks an SM, five and more a lane's two rows:
// two stages there.
struct FewPlan { int chunks, stages; };
inline int few_resident(int mb, int chunks, int stages) {
    const int room = (int)(227 * 1024 / (few_smem(mb, chunks, stages) + 1024));
    return room < few_blocks(mb) ? room : few_blocks(mb);
}
inline FewPlan few_plan(int rows, long long row_blocks, int nc) {
    const int least = ((nc + 7) / 8 + 3) / 4 * 4, mb = few_registers(rows);
    if (mb > 8) return {least, 2};
    for (int c = 1; c <= (rows <= 2 ? 4 : 2); c *= 2) {
        const int q = (nc + c - 1) / c;
        if (q <= least || q % 4 != 0 || nc % q != 0 || row_blocks * c < 256 || few_smem(mb, q, 2) > 112 * 1024) continue;
        const double waves = (double)(row_blocks * c) / (148.0 * few_resident(mb, q, 2));
        if (rows > 2 || waves <= 1.05 || waves >= 0.7 * std::ceil(waves)) return {q, 2};
    }
    if (mb != 4) return {least, 2};
    const int chunks = least < nc ? least : nc;
    const long long blocks = row_blocks * ((nc + least - 1) / least);
    const bool deep = few_smem(mb, chunks, 3) <= FEW_SMEM_MOST && blocks <= (few_resident(mb, chunks, 3) >= 2 ? 2 * 2 * 148 : 120);
    return {least, deep ? 3 : 2};
}
// Whether a block finds room for its chunks' sums: it does up to K = 61,440 at 5 to 8 rows, 131,072 at 3 and 4, 548,864 at one.
inline bool few_fits(int rows, long long row_blocks, int nc) {
    const FewPlan p = few_plan(rows, row_blocks, nc);
    return few_smem(few_registers(rows), p.chunks < nc ? p.chunks : nc, p.stages) <= FEW_SMEM_MOST;
}

// GLU: W is [gate; up] ([2N, K]); the block's 64 weight rows are 32 of each half, of the same features, and C[m, n] =
// silu(gate) * up. The sums and the activation are those of the product and the activation kernel behind one another, to the bit; a
// launch and the way of gate and up through memory are saved. A decode step at 1B sizes (16 layers), us: five requests 1,973 -> 1,876, one
// 1,337 -> 1,339 (there the activation kernel was hidden by its neighbours). With one thread adding up a feature's gate and then its up
// value, one request took 1,380.
template <int MB, int RN, int NS, bool GLU>
__global__ void __launch_bounds__(256 / RN, few_blocks(MB))
gemm_f32_few_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw, float* __restrict__ C,
                    long long ldc, int M, int N, int K, const float* __restrict__ bias, int nc, int q, int c, int early) {
    constexpr int THREADS = 256 / RN, STAGE = 32 * RN * FEW_K;        // floats of a warp's stage: its rows, 16-byte pieces at (piece ^ row & 7)
    extern __shared__ __align__(16) float smem[];
    float* ring = smem;                               // [8 / RN warps][NS][STAGE]
    float* xs = ring + 8 / RN * NS * STAGE;           // [MB][4 chunks * CHUNK]
    float* part = xs + 4 * CHUNK * MB;                // [q][MB][FEW_N]
    pdl_launch_dependents();
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int FEATS = GLU ? FEW_N / 2 : FEW_N;    // output features of a block
    int rank = blockIdx.x % c, n0 = (blockIdx.x / c) * FEATS;
    int half = RN == 1 ? warp & 1 : 0, slot = RN == 1 ? warp >> 1 : warp;
    int first = rank * q, mine = min(q, nc - first);  // this block's chunks
    float* wring = ring + warp * NS * STAGE;
    int lrow = lane >> 3, lpiece = lane & 7;          // loads: 8 lanes take 128 bytes of a row
    // the next stage to ask for: of the warp's chunk `lchunk` (slot, slot + 4, ...), its `lu`-th
    int lchunk = slot, lu = 0, lput = 0;
    auto load = [&]() {
        if (lchunk < mine) {
            int k = (first + lchunk) * CHUNK + lu * FEW_K + lpiece * 4;
            float* dst = wring + lput * STAGE;
#pragma unroll
            for (int i = 0; i < 8 * RN; ++i) {
                int r = i * 4 + lrow, row = half * 32 + r, n = n0 + (GLU ? row & 31 : row);
                bool in = n < N && k < K;             // K is a multiple of 4
                size_t wr = GLU && row >= 32 ? (size_t)N + n : (size_t)n;
                cp_async16(dst + r * FEW_K + ((lpiece ^ (r & 7)) << 2), in ? W + wr * ldw + k : W, in ? 16 : 0);
            }
            lput = lput + 1 == NS ? 0 : lput + 1;
            if (++lu == CHUNK / FEW_K) { lu = 0; lchunk += 4; }
        }
        cp_async_commit();
    };
    // `early`: no kernel writes W, so its first stages are asked for before the wait
    if (!early) pdl_wait(11);
#pragma unroll
    for (int s = 0; s < NS; ++s) load();
    if (early) pdl_wait(11);

    int get = 0, seg = seg_chunks(nc);
    for (int t = 0; t * 4 < mine; ++t) {
        if (t > 0) __syncthreads();                   // everyone has read the chunks in front
        int kbase = (first + t * 4) * CHUNK;
        // x of four chunks; what lies beyond K or M is zero
        for (int i = threadIdx.x; i < CHUNK * MB; i += THREADS) {
            int m = i / CHUNK, k4 = (i % CHUNK) * 4;  // 4 * CHUNK / 4 pieces of every row
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (m < M && kbase + k4 < K) v = *reinterpret_cast<const float4*>(A + (size_t)m * lda + kbase + k4);
            *reinterpret_cast<float4*>(xs + m * 4 * CHUNK + k4) = v;
        }
        __syncthreads();
        if (t * 4 + slot < mine) {
            unsigned long long acc[RN][MB];
#pragma unroll
            for (int r = 0; r < RN; ++r)
#pragma unroll
                for (int m = 0; m < MB; ++m) acc[r][m] = 0;
            const float* xc = xs + slot * CHUNK;
#pragma unroll 1
            for (int u = 0; u < CHUNK / FEW_K; ++u) {
                cp_async_wait<NS - 1>();
                __syncwarp();
                const float* row = wring + get * STAGE + lane * FEW_K;
                const float* xk = xc + u * FEW_K;
#pragma unroll
                for (int p = 0; p < FEW_K / 4; ++p) {
                    ulonglong2 w[RN];
#pragma unroll
                    for (int r = 0; r < RN; ++r) w[r] = *reinterpret_cast<const ulonglong2*>(row + r * 32 * FEW_K + ((p ^ (lane & 7)) << 2));
#pragma unroll
                    for (int m = 0; m < MB; ++m) {
                        ulonglong2 x = *reinterpret_cast<const ulonglong2*>(xk + m * 4 * CHUNK + p * 4);
#pragma unroll
                        for (int r = 0; r < RN; ++r) { fma2(acc[r][m], w[r].x, x.x); fma2(acc[r][m], w[r].y, x.y); }
                    }
                }
                get = get + 1 == NS ? 0 : get + 1;
                __syncwarp();                     // the warp has read this stage
                load();
            }
            float* dst = part + (size_t)(t * 4 + slot) * MB * FEW_N + half * 32 + lane;
#pragma unroll
            for (int r = 0; r < RN; ++r)
#pragma unroll
                for (int m = 0; m < MB; ++m) dst[m * FEW_N + r * 32] = sum2(acc[r][m]);
        }
    }
    if (c > 1) { cluster_arrive(); cluster_wait(); }
    else __syncthreads();
    // this block's share of the outputs: the chunks' sums, segment by segment, from the blocks that hold them
    int total = M * FEW_N, share = ((total + c - 1) / c + 1) & ~1;
    auto sum_of = [&](int m, int col) {
        float sum = 0.f, run = 0.f;
        int in_seg = 0;
        bool begun = false;
        for (int b = 0; b < c; ++b) {
            const float* p = (c > 1 ? cg::this_cluster().map_shared_rank(part, b) : part) + m * FEW_N + col;
            int have = min(q, nc - b * q);
            for (int i0 = 0; i0 < have; i0 += 4) {            // q is a multiple of 4: four reads on their way at once
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = i0 + i < have ? p[(size_t)(i0 + i) * MB * FEW_N] : 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i0 + i >= have) break;
                    run = in_seg == 0 ? v[i] : run + v[i];
                    if (++in_seg == seg) { sum = begun ? sum + run : run; begun = true; in_seg = 0; }
                }
            }
        }
        if (in_seg) sum = begun ? sum + run : run;
        return sum;
    };
    // GLU: neighbouring threads add up a feature's gate and its up value, and the even one of the two finishes
    for (int base = rank * share, end = min(total, base + share); base < end; base += THREADS) {
        int e = base + threadIdx.x, m = e / FEW_N, col = e % FEW_N;
        if (GLU) col = (col >> 1) + (col & 1) * 32;
        int n = n0 + (GLU ? col & 31 : col);
        float sum = e < end && n < N ? sum_of(m, col) : 0.f;
        if (GLU) {
            float up = __shfl_down_sync(0xffffffffu, sum, 1);
            sum = sum / (1.0f + expf(-sum)) * up;
        }
        if (e < end && n < N && !(GLU && (e & 1))) C[(size_t)m * ldc + n] = !GLU && bias ? sum + bias[n] : sum;
    }
    cp_async_wait<0>();
    __syncwarp();
    if (c > 1) { cluster_arrive(); cluster_wait(); }  // peers have read this block's sums
}

template <int MB, int NS, bool GLU>
int launch_few(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc, int M, int N, int K,
               const float* bias, int q, int early, cudaStream_t stream) {
    constexpr int RN = few_rows_a_lane(MB), FEATS = GLU ? FEW_N / 2 : FEW_N;
    const int nc = (K + CHUNK - 1) / CHUNK, c = (nc + q - 1) / q;
    size_t smem = few_smem(MB, min(q, nc), NS);
    if (smem > FEW_SMEM_MOST) return VOB_ERR_UNSUPPORTED;
    auto kernel = gemm_f32_few_kernel<MB, RN, NS, GLU>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    long long blocks = (long long)((N + FEATS - 1) / FEATS) * c;
    if (blocks > 0x7fffffffLL) return VOB_ERR_UNSUPPORTED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(256 / RN);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_vob_pdl ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kernel, A, lda, W, ldw, C, ldc, M, N, K, bias, nc, q, c, early);
    return e != cudaSuccess ? (int)e : vob_launch_status();
}

// ------------------------------------------------------------------------------------------------ tiles
// A block of 128 threads computes 16 * TR rows by 64 columns (TR 2, 4 to 8), a thread TR x 8 of them (rows tm + 16 i, columns tn + 8 j). K
// comes in slabs of 16 through a ring of three stages, [row][k] as it lies in memory, rows 20 floats apart: the 16-byte reads
// of different rows that a warp makes at once fall into different banks. The sums of the chunks so far wait in shared
// memory: the segment's, and (CL == 1) the finished segments'. Or a cluster of CL = 8 blocks shares K, a segment each, and
// adds the segments' sums: eight times the blocks, for few tiles or a last wave that would be nearly empty.
constexpr int TN = 64, TK = 16, TLD = TK + 4, TSTAGES = 3, GRID_Y = 32768;
__host__ __device__ constexpr int tile_blocks(int tr) { return tr >= 5 ? 2 : tr == 4 ? 3 : 4; }   // resident on an SM

template <int TR, bool VEC, int CL>
__global__ void __launch_bounds__(128, tile_blocks(TR))
gemm_f32_tile_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw, float* __restrict__ C,
                     long long ldc, int M, int N, int K, const float* __restrict__ bias, int seg) {
    constexpr int TM = 16 * TR, QUADS = TR * 2;
    extern __shared__ __align__(16) float smem[];
    float* stage = smem;                                        // [TSTAGES][(TM + TN)][TLD]
    float4* sums = reinterpret_cast<float4*>(smem + TSTAGES * (TM + TN) * TLD);    // [CL == 1 ? 2 : 1][QUADS][128]
    pdl_launch_dependents();
    pdl_wait(11);
    int tid = threadIdx.x, lane = tid & 31;
    int tn = (lane & 3) | ((lane >> 4) << 2), tm = ((tid >> 5) << 2) | ((lane >> 2) & 3);
    int rank = blockIdx.x % CL, m0 = blockIdx.x / CL * TM, n0 = (blockIdx.z * GRID_Y + blockIdx.y) * TN;
    int kb = min(K, rank * seg * CHUNK), ke = CL > 1 ? min(K, kb + seg * CHUNK) : K;
    int slabs = (ke - kb + TK - 1) / TK;
    int put_at = 0;
    const int lk = (tid & 3) * 4;
    auto load = [&](int s) {
        if (s < slabs) {
            float* st = stage + put_at * (TM + TN) * TLD;
            put_at = put_at + 1 == TSTAGES ? 0 : put_at + 1;
            int k = kb + s * TK + lk;
#pragma unroll
            for (int i = 0; i < (TM + TN + 31) / 32; ++i) {
                int r = i * 32 + (tid >> 2);
                if ((TM + TN) % 32 != 0 && r >= TM + TN) break;
                bool isA = TM % 32 == 0 ? i < TM / 32 : r < TM;
                int g = isA ? m0 + r : n0 + r - TM;
                const float* p = isA ? A + (size_t)g * lda : W + (size_t)g * ldw;
                bool row = g < (isA ? M : N);
                float* d = st + r * TLD + (tid & 3) * 4;
                if constexpr (VEC) {                                      // K is a multiple of 4
                    bool in = row && k < ke;
                    cp_async16(d, in ? p + k : A, in ? 16 : 0);
                } else {
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        bool in = row && k + x < ke;
                        cp_async4(d + x, in ? p + k + x : A, in ? 4 : 0);
                    }
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < TSTAGES - 1; ++s) load(s);
    unsigned long long acc[TR][8];                              // even and odd k
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0;
    int chunk = 0;                                              // of the segment
    int at = 0;
    for (int s = 0; s < slabs; ++s) {
        cp_async_wait<TSTAGES - 2>();
        __syncthreads();                                        // slab s is here, and slab s - 1 has been read by all
        load(s + TSTAGES - 1);
        const float* as = stage + at * (TM + TN) * TLD + tm * TLD;
        const float* bs = stage + at * (TM + TN) * TLD + (TM + tn) * TLD;
#pragma unroll
        for (int k = 0; k < TK; k += 4) {
            ulonglong2 b[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(bs + j * 8 * TLD + k);
#pragma unroll
            for (int i = 0; i < TR; ++i) {
                ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + i * 16 * TLD + k);
#pragma unroll
                for (int j = 0; j < 8; ++j) fma2(acc[i][j], a.x, b[j].x);
#pragma unroll
                for (int j = 0; j < 8; ++j) fma2(acc[i][j], a.y, b[j].y);
            }
        }
        at = at + 1 == TSTAGES ? 0 : at + 1;
        bool last = s == slabs - 1;
        if ((s & (CHUNK / TK - 1)) == CHUNK / TK - 1 || last) {                 // the chunk ends
            bool seg_ends = chunk == seg - 1 || last, first_seg = s < seg * (CHUNK / TK);
            float4* d = sums + tid;
#pragma unroll
            for (int e = 0; e < QUADS; ++e) {
                const unsigned long long* x = &acc[e >> 1][(e & 1) * 4];
                float4 v = make_float4(sum2(x[0]), sum2(x[1]), sum2(x[2]), sum2(x[3]));
                if (chunk > 0) {
                    float4 o = d[e * 128];
                    v.x = o.x + v.x; v.y = o.y + v.y; v.z = o.z + v.z; v.w = o.w + v.w;
                }
                if (CL > 1 || !seg_ends) d[e * 128] = v;
                else {
                    if (!first_seg) {
                        float4 o = d[(QUADS + e) * 128];
                        v.x = o.x + v.x; v.y = o.y + v.y; v.z = o.z + v.z; v.w = o.w + v.w;
                    }
                    d[(QUADS + e) * 128] = v;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[e >> 1][(e & 1) * 4 + j] = 0;
            }
            chunk = seg_ends ? 0 : chunk + 1;
        }
    }
    cp_async_wait<0>();
    auto put = [&](int e, float4 v) {                           // quad e of this thread
        int m = m0 + tm + 16 * (e >> 1), n = n0 + tn + 32 * (e & 1);
        if (m >= M) return;
        float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n + 8 * j < N) C[(size_t)m * ldc + n + 8 * j] = bias ? o[j] + bias[n + 8 * j] : o[j];
    };
    if constexpr (CL == 1) {                                               // a thread's own sums: no barrier
#pragma unroll
        for (int e = 0; e < QUADS; ++e) put(e, sums[(QUADS + e) * 128 + tid]);
        return;
    }
    cluster_arrive();
    cluster_wait();
    int have = (K + seg * CHUNK - 1) / (seg * CHUNK);           // segments that are not empty
    for (int e = rank; e < QUADS; e += CL) {
        float4 o[8];
#pragma unroll
        for (int b = 0; b < 8; ++b)
            if (b < have) o[b] = cg::this_cluster().map_shared_rank(sums, b)[e * 128 + tid];
        float4 v = o[0];
#pragma unroll
        for (int b = 1; b < 8; ++b)
            if (b < have) { v.x += o[b].x; v.y += o[b].y; v.z += o[b].z; v.w += o[b].w; }
        put(e, v);
    }
    cluster_arrive();
    cluster_wait();                                             // peers have read this block's sums
}

template <int TR>
int launch_tile(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc, int M, int N, int K,
                const float* bias, int nc, int c, int vec, cudaStream_t stream) {
    int mtiles = (M + 16 * TR - 1) / (16 * TR), ntiles = (N + TN - 1) / TN;
    auto kernel = c == 1 ? (vec ? gemm_f32_tile_kernel<TR, true, 1> : gemm_f32_tile_kernel<TR, false, 1>)
                         : (vec ? gemm_f32_tile_kernel<TR, true, 8> : gemm_f32_tile_kernel<TR, false, 8>);
    size_t smem = sizeof(float) * (size_t)(TSTAGES * (16 * TR + TN) * TLD + (c == 1 ? 2 : 1) * TR * 8 * 128);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(mtiles * c), (unsigned)min(ntiles, GRID_Y), (unsigned)((ntiles + GRID_Y - 1) / GRID_Y));
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_vob_pdl ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kernel, A, lda, W, ldw, C, ldc, M, N, K, bias, seg_chunks(nc));
    return e != cudaSuccess ? (int)e : vob_launch_status();
}

// Tiles of 128, 112, 96, 80, 64 or 32 rows, a block or eight to a tile: the choice whose estimated time is least. The table holds us per chunk of K.
// One block to a tile: for grids of at most 48 and 74 blocks, which find an SM each beside their neighbours', for 1, 2, 3 and 4 blocks on the fullest of
// 148 SMs, and per block beyond. Eight to a tile, a segment of K each: for at most 4, 6, 8, 10, 12, 15, 23, 32, 42, 48 and 64 clusters, and per 16
// clusters beyond. `by4`: how much longer both take where operands come by 4 bytes. What is added is a block's start and the cluster's sums. In
// the long run a row costs alike at 64 rows and more (0.93 to 1.01 us a chunk, 16 rows and SM), 1.37 at 32: rows that are not there, waves and
// idle SMs decide.
// The numbers are fitted to 3,125 sizes (N 64 to 32,000, K 96 to 14,336, 17 to 4,096 rows), where every height with and without a shared K was timed
// twice: back to back, and with another kernel in between, which places small grids otherwise. Over both the choice takes 1.014 and 1.033 of the
// best one's time on average; 128, 64 and 32 rows by rows and waves took 1.10 and 1.13, all six by rows and waves 1.09 and 1.10. Against those three
// heights 20 and 18 sizes lose more than 2 %, all but a few of small grids. us, those three / now: 64 x 516 at 160 rows 17.5 / 17.5, 3,072 x 516 at 81
// 32.4 / 32.4, 16,384 x 2,048 at 72, 300, 450 and 2,048 rows 242, 563, 941, 3,262 / 170, 563, 799, 3,262; 2,048 x 8,192 at 97 and 450 126, 494 /
// 115, 494; 8,192 x 4,096 at 300 610 / 610; 2,048 x 2,050 at 260 159 / 140.
struct TilePick { int tr, c; };
TilePick pick_tile(int M, int N, int K, bool vec) {
    static const struct { int tr; float one[7], shared[12], by4[2]; } times[] = {
        {2, {3.27f, 4.51f, 7.15f, 7.67f, 10.0f, 10.5f, 2.73f}, {4.66f, 4.08f, 4.91f, 5.17f, 5.54f, 6.25f, 9.21f, 11.4f, 9.7f, 12.3f, 12.2f, 2.38f}, {1.44f, 1.4f}},
        {4, {5.23f, 5.53f, 10.3f, 10.6f, 12.2f, 15.8f, 3.87f}, {5.4f, 5.16f, 5.68f, 9.46f, 7.72f, 9.58f, 12.6f, 12.2f, 10.3f, 12.6f, 16.9f, 3.69f}, {1.41f, 1.3f}},
        {5, {7.91f, 7.85f, 7.85f, 10.1f, 15.1f, 19.5f, 5.07f}, {6.0f, 7.22f, 7.23f, 7.29f, 7.77f, 7.01f, 8.95f, 8.63f, 15.8f, 17.2f, 20.4f, 4.78f}, {1.27f, 1.25f}},
        {6, {8.39f, 9.84f, 10.1f, 11.9f, 16.5f, 21.5f, 5.65f}, {7.05f, 9.26f, 8.11f, 8.95f, 9.24f, 11.1f, 12.9f, 12.5f, 17.5f, 20.9f, 25.4f, 5.67f}, {1.27f, 1.13f}},
        {7, {8.07f, 9.7f, 11.4f, 13.6f, 20.7f, 26.4f, 6.7f}, {7.22f, 9.38f, 8.67f, 9.78f, 11.2f, 11.0f, 15.7f, 15.5f, 20.0f, 25.3f, 27.8f, 6.24f}, {1.32f, 1.15f}},
        {8, {8.64f, 10.5f, 14.9f, 14.9f, 23.5f, 29.7f, 7.44f}, {8.76f, 9.88f, 8.78f, 12.6f, 11.8f, 13.1f, 15.9f, 16.3f, 23.3f, 27.9f, 30.2f, 6.76f}, {1.33f, 1.14f}}};
    static const int clusters[] = {4, 6, 8, 10, 12, 15, 23, 32, 42, 48, 64};
    const int nc = (K + CHUNK - 1) / CHUNK;
    TilePick best = {8, 1};
    double least = 1e300;
    for (const auto& t : times) {
        if (t.tr > 4 && t.tr < 8 && M <= 64) continue;
        const long long tiles = ((long long)M + 16 * t.tr - 1) / (16 * t.tr) * ((N + TN - 1) / TN);
        const long long per_sm = (tiles + 147) / 148;
        const double chunk = tiles <= 48 ? t.one[0] : tiles <= 74 ? t.one[1] : per_sm <= 4 ? t.one[per_sm + 1] : t.one[6] * (double)per_sm;
        const double one = chunk * (K / (double)CHUNK) * (vec ? 1.0 : t.by4[0]) + 1.5 + 0.13 * t.tr * (double)per_sm;
        if (one < least) { least = one; best = {t.tr, 1}; }
        if (nc < 8) continue;
        int i = 0;
        while (i < 11 && tiles > clusters[i]) ++i;
        const double segment = i < 11 ? t.shared[i] : t.shared[11] * ((double)tiles / 16.0 + 0.7);
        const double shared = segment * seg_chunks(nc) * (vec ? 1.0 : t.by4[1]) + 2.0 + 0.1 * t.tr * ((double)tiles / 16.0);
        if (shared < least) { least = shared; best = {t.tr, 8}; }
    }
    return best;
}

// Whether the kernel for few rows is the faster one (see vob_gemm_f32).
bool few_rows(int M, int K) {
    int nc = (K + CHUNK - 1) / CHUNK, q = ((nc + 7) / 8 + 3) / 4 * 4;
    return M <= (K <= 64 ? 4 : 8) || (M <= 16 && q == 4 && nc > 1);
}

// More than 32 chunks and 9 to 24 rows: whether eight rows at a time are faster than the tiles. (A block of 16 rows would have its SM to itself
// there.) Cold, back to back, us in eights / in tiles of 32 rows with K shared, at 9, 16, 17 and 24 rows: 2,048 x 8,192 33, 36, 50, 53 / 86 to 87;
// 8,192 x 8,192, whose weights come from memory every time, 116, 146, 189, 218 / 184; 500 x 5,120 19, 23, 30, 33 / 23. Three eights gain only
// where the tiles are at their worst, with 24 to 50 clusters of eight blocks, and where L2 keeps the weights: 1,024 x 6,144 at 17 and 24 rows 42, 46 /
// 46 (39 with the weights in L2), 3,072 x 6,144 70, 85 / 71. Under 40 chunks the last block of a K has little to do, and a narrow N goes to
// the tiles (500 x 4,612 at 16 rows 24.6 / 23.0, 896 x 4,864 24.6 / 29.2); beyond 128 a block of eight rows has its SM to itself (3,584 x 18,944 at 16 rows 245 / 218,
// 2,560 x 18,944 0.86 of the tiles' time). A decode step of 12 requests at 1B sizes 3,590 -> 2,660 us.
bool by_eights(int M, int N, int K) {
    const int nc = (K + CHUNK - 1) / CHUNK;
    const double w_bytes = 4.0 * N * K;
    if (M <= 8 || M > 24 || nc <= 32 || !few_fits(8, (N + FEW_N - 1) / FEW_N, nc)) return false;
    if (M <= 16) return w_bytes <= 320e6 && (nc >= 40 || N >= 768) && (nc <= 128 || N <= 3072);
    return N >= 1536 && N <= 3200 && w_bytes > 33e6 && w_bytes <= 70e6;
}

template <bool GLU>
int few(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc, int M, int N, int K, const float* bias,
        int early, cudaStream_t stream) {
    constexpr int FEATS = GLU ? FEW_N / 2 : FEW_N;
    const FewPlan p = few_plan(M, (N + FEATS - 1) / FEATS, (K + CHUNK - 1) / CHUNK);
    const int q = p.chunks;
    if constexpr (!GLU)
        if (M > 8) return launch_few<16, 2, GLU>(A, lda, W, ldw, C, ldc, M, N, K, bias, q, early, stream);
    return M == 1          ? launch_few<1, 2, GLU>(A, lda, W, ldw, C, ldc, M, N, K, bias, q, early, stream)
           : M == 2        ? launch_few<2, 2, GLU>(A, lda, W, ldw, C, ldc, M, N, K, bias, q, early, stream)
           : M > 4         ? launch_few<8, 2, GLU>(A, lda, W, ldw, C, ldc, M, N, K, bias, q, early, stream)
           : p.stages == 3 ? launch_few<4, 3, GLU>(A, lda, W, ldw, C, ldc, M, N, K, bias, q, early, stream)
                           : launch_few<4, 2, GLU>(A, lda, W, ldw, C, ldc, M, N, K, bias, q, early, stream);
}

}  // namespace

// Whether vob_gemm_f32_swiglu takes a product of these sizes (then it is also the faster way).
VOB_EXPORT int vob_gemm_f32_swiglu_supported(int M, int I, int K) {
    if (M <= 0 || I <= 0 || K <= 0 || K % 4 != 0 || M > 8 || !few_rows(M, K)) return 0;      // 12 rows: 1 % slower in a whole step
    return few_fits(M, (I + FEW_N / 2 - 1) / (FEW_N / 2), (K + CHUNK - 1) / CHUNK);
}

// C[M, I] = silu(A Wg^T) * (A Wu^T), W = [Wg; Wu] of shape [2I, K], few rows; the bits of vob_gemm_f32 and vob_swiglu one behind the other.
VOB_EXPORT int vob_gemm_f32_swiglu(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc, int M, int I,
                                   int K, int early, cudaStream_t stream) {
    if (M <= 0 || I <= 0) return 0;
    if (K <= 0 || lda < K || ldw < K || ldc < I) return VOB_ERR_BAD_ARG;
    if (!vob_gemm_f32_swiglu_supported(M, I, K) || lda % 4 || ldw % 4 || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return VOB_ERR_UNSUPPORTED;
    return few<true>(A, lda, W, ldw, C, ldc, M, I, K, nullptr, early, stream);
}

// For tests: 8 * chunks of a block + stages of a ring of the few-row kernel (`features`: 64 a block, 32 with the activation in the epilogue).
VOB_EXPORT int vob_gemm_f32_few_plan(int rows, int N, int K, int features) {
    if (rows < 1 || rows > 16 || N < 1 || K < 1 || (features != FEW_N && features != FEW_N / 2)) return 0;
    const FewPlan p = few_plan(rows, (N + features - 1) / features, (K + CHUNK - 1) / CHUNK);
    return 8 * p.chunks + p.stages;
}

// For tests: 16 * a tile's rows / 16 + blocks that share its K.
VOB_EXPORT int vob_gemm_f32_tile(int M, int N, int K, int vec) {
    if (M < 1 || N < 1 || K < 1) return 0;
    const TilePick t = pick_tile(M, N, K, vec != 0);
    return 16 * t.tr + t.c;
}

// Kernels that a product of these sizes takes (operands that come by 16 bytes).
VOB_EXPORT int vob_gemm_f32_launches(int M, int N, int K) { return M > 0 && N > 0 && K > 0 && K % 4 == 0 && by_eights(M, N, K) ? (M + 7) / 8 : 1; }

// `bias` (N entries, may be null) is added to every row after the sum over k. `early`: W holds weights, which no kernel writes, and
// may be read while the kernels in front still run.
VOB_EXPORT int vob_gemm_f32(const float* A, long long lda, const float* W, long long ldw, float* C,
                            long long ldc, int M, int N, int K, const float* bias, int early, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || lda < K || ldw < K || ldc < N) return VOB_ERR_BAD_ARG;
    if ((M + 63) / 64 > 65535) return VOB_ERR_UNSUPPORTED;
    int nc = (K + CHUNK - 1) / CHUNK;
    int vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    // 16 rows: what a lane's registers hold. Cold, 9 to 16 rows, us here / in tiles (32 rows at least): 2,048 x 512 16 / 23, 2,048 x 2,048
    // 19 / 21, 4,096 x 4,096 41 / 55, 16,384 x 2,048 68 / 94, 128,256 x 2,048 391 / 644; where K has more than 32 chunks see
    // `by_eights`. Up to 8 rows the tiles never win: 2,048 x 8,192 in 32 rows of a tile 86, here 18 at eight rows. A single chunk is too short for what a block of 5 rows and more sets
    // up (back to back, 16 rows: 64 x 64 7.3 / 2.9, 2,048 x 64 7.7 / 3.1, 128 x 128 7.5 / 4.7; 8 rows 4.4 / 2.9, 4.6 / 3.1, 4.5 / 4.7).
    if (vec && few_rows(M, K)) {
        int e = few<false>(A, lda, W, ldw, C, ldc, M, N, K, bias, early, stream);
        if (e != VOB_ERR_UNSUPPORTED) return e;       // a K whose sums find no room in shared memory: tiles
    }
    if (vec && by_eights(M, N, K)) {
        for (int m = 0; m < M; m += 8) {
            int e = few<false>(A + (size_t)m * lda, lda, W, ldw, C + (size_t)m * ldc, ldc, min(8, M - m), N, K, bias, early, stream);
            if (e) return e;
        }
        return 0;
    }
    const TilePick t = pick_tile(M, N, K, vec);
    switch (t.tr) {
        case 2: return launch_tile<2>(A, lda, W, ldw, C, ldc, M, N, K, bias, nc, t.c, vec, stream);
        case 4: return launch_tile<4>(A, lda, W, ldw, C, ldc, M, N, K, bias, nc, t.c, vec, stream);
        case 5: return launch_tile<5>(A, lda, W, ldw, C, ldc, M, N, K, bias, nc, t.c, vec, stream);
        case 6: return launch_tile<6>(A, lda, W, ldw, C, ldc, M, N, K, bias, nc, t.c, vec, stream);
        case 7: return launch_tile<7>(A, lda, W, ldw, C, ldc, M, N, K, bias, nc, t.c, vec, stream);
        default: return launch_tile<8>(A, lda, W, ldw, C, ldc, M, N, K, bias, nc, t.c, vec, stream);
    }
}
