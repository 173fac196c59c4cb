// Causal grouped-query attention over the paged cache, for portions of prompts and for single
// decoded tokens alike.
//
// Math per (row, head a), the row at position p of its request, kvh = a / (H / KV):
//   s_j = (q_a . K[j, kvh]) * scale         for keys j in [first, p],  first = max(0, p+1-window)
//   out_a = sum_j softmax(s)_j * V[j, kvh]   softmax in float32 (running max and sum)
// Causality is "visit keys 0..p only", with the step's own keys already in the cache; there is
// no mask tensor. Reference: crates/engine/src/backend/cpu/attention.rs:76-128 (two passes
// there, one pass with a running maximum here; same value up to rounding), called for prefill
// and decode alike (crates/engine/src/backend/cpu/mod.rs:310,337).
// Cache layout per layer: K and V are [num_pages][KV][page_size][hd]; key j of a request lives
// in page block_table[seq][j / page_size] at offset j % page_size.
#include "common.cuh"
#include <cfloat>
#include <cooperative_groups.h>
#include <type_traits>
VOB_PDL_SWITCH(attention)

// ---------------------------------------------------------------------------------------------
// General kernel: one warp per (row, head). Keys are visited in chunks of 32: each lane scores
// one key (its K row read in 16-byte pieces against q held in shared memory), the warp agrees
// on the running maximum, then the 32 weighted V rows are summed with lanes spread over the
// head's dimensions. Any head_dim that is a multiple of 8 up to 256, any H, KV, page size.
// Launch: ceil(T*H / 4) blocks of 128 threads; 4*hd floats of shared memory.
// Bound: L2/L1 bandwidth (every head of a group re-reads its K/V); this is the kernel of the
// 32-bit engine for sizes the kernels below refuse, and the fallback of the bfloat16 engine for sizes its tuned kernels refuse.
// A row's result depends only on its own q and keys, never on the batch around it.
// ---------------------------------------------------------------------------------------------
template <typename T> struct Vec16;
template <> struct Vec16<float> {
    static constexpr int N = 4;
    __device__ static inline void load(const float* p, float* o) {
        float4 v = *reinterpret_cast<const float4*>(p);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
};
template <> struct Vec16<__nv_bfloat16> {
    static constexpr int N = 8;
    __device__ static inline void load(const __nv_bfloat16* p, float* o) {
        uint4 v = *reinterpret_cast<const uint4*>(p);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 f = __bfloat1622float2(h[i]);
            o[2 * i] = f.x; o[2 * i + 1] = f.y;
        }
    }
};

template <typename T>
__global__ void __launch_bounds__(128, 8)
paged_attention_warp_kernel(const T* __restrict__ q, long long q_stride, T* __restrict__ out, long long out_stride,
                            const T* __restrict__ kcache, const T* __restrict__ vcache,
                            const int* __restrict__ block_tables, int max_pages,
                            const int* __restrict__ row_seq, const int* __restrict__ positions,
                            int T_rows, int H, int KV, int hd, int page_size, int window, float scale) {
    pdl_launch_dependents();
    pdl_wait(6);
    extern __shared__ float qs_all[];
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long long w = (long long)blockIdx.x * 4 + warp;
    if (w >= (long long)T_rows * H) return;          // whole warp leaves together
    int row = (int)(w / H), head = (int)(w % H);
    int kvh = head / (H / KV);
    float* qs = qs_all + warp * hd;
    const T* qp = q + (size_t)row * q_stride + (size_t)head * hd;
    for (int d = lane; d < hd; d += 32) qs[d] = ld_f(qp + d);
    __syncwarp();

    int pos = positions[row];
    if (pos < 0) {                                   // a padding row: no keys, zero output
        T* op0 = out + (size_t)row * out_stride + (size_t)head * hd;
        for (int d = lane; d < hd; d += 32) st_f(op0 + d, 0.f);
        return;
    }
    int seq = row_seq[row];
    const int* bt = block_tables + (size_t)seq * max_pages;
    int first = window > 0 ? max(0, pos + 1 - window) : 0;

    constexpr int VN = Vec16<T>::N;
    float m = -INFINITY, l = 0.f;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;

    for (int c0 = first; c0 <= pos; c0 += 32) {
        int j = c0 + lane;
        bool valid = j <= pos;
        int slot_row = 0;          // row index of key j in the [.., hd] view of the layer's cache
        float s = -INFINITY;
        if (valid) {
            int page = bt[j / page_size];
            slot_row = (page * KV + kvh) * page_size + (j % page_size);
            const T* kp = kcache + (size_t)slot_row * hd;
            float dot = 0.f;
            for (int d = 0; d < hd; d += VN) {
                float kv[VN];
                Vec16<T>::load(kp + d, kv);
#pragma unroll
                for (int i = 0; i < VN; ++i) dot = fmaf(qs[d + i], kv[i], dot);
            }
            s = dot * scale;
        }
        float m_new = fmaxf(m, warp_max(s));
        float p = valid ? expf(s - m_new) : 0.f;
        float alpha = expf(m - m_new);               // 0 on the first chunk (m = -inf)
        l = l * alpha + warp_sum(p);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] *= alpha;
        m = m_new;
        int nk = min(32, pos - c0 + 1);
        for (int jj = 0; jj < nk; ++jj) {
            float pj = __shfl_sync(0xffffffffu, p, jj);
            int sr = __shfl_sync(0xffffffffu, slot_row, jj);
            const T* vp = vcache + (size_t)sr * hd;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                int d = 2 * lane + 64 * i;
                if (d < hd) {
                    acc[2 * i] = fmaf(pj, ld_f(vp + d), acc[2 * i]);
                    acc[2 * i + 1] = fmaf(pj, ld_f(vp + d + 1), acc[2 * i + 1]);
                }
            }
        }
    }
    float inv_l = 1.0f / l;
    T* op = out + (size_t)row * out_stride + (size_t)head * hd;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int d = 2 * lane + 64 * i;
        if (d < hd) {
            st_f(op + d, acc[2 * i] * inv_l);
            st_f(op + d + 1, acc[2 * i + 1] * inv_l);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The 32-bit engine at head sizes 64 and 128 with at most 8 heads a kv head: two kernels, one for portions of prompts and one
// for single tokens. Both form a row's result in the same steps, so that a row's bits depend neither on the batch nor on which
// of the two computed it. Keys are taken in tiles of 32 (key 32 t .. 32 t + 31 of the request, t ascending); of a tile
//   s_j = scale * (q . k_j)      two chains of FMAs, over even and odd d, and their sum
//   m_t = max(max s_j, -FLT_MAX),  p_j = expf(s_j - m_t),  l_t = sum p_j,  o_t[d] = sum p_j v_j[d]     chains over the keys in order
// and the tile joins what is behind it: M' = max(M, m_t), acc = acc expf(M - M') + o_t expf(m_t - M'), l likewise. Keys that a
// row may not see take no part (what they hold, infinities too, does not reach the row). A tile whose scores are all minus infinity
// weighs nothing: with -FLT_MAX for its maximum expf gives zeros, and not the NaN of minus infinity less itself.
// (The general kernel above sums over all keys in one chain: relative error against 64 bits at 4,000 keys 1.2e-6, here 3.4e-7.)
// ---------------------------------------------------------------------------------------------
namespace cg = cooperative_groups;

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long d) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(d));
    return f;
}
__device__ __forceinline__ float sum2(unsigned long long d) {
    float2 f = unpack2(d);
    return __fadd_rn(f.x, f.y);
}
// 16 bytes from global to shared memory, zeros where `in` is false.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}

constexpr int KT = 32;            // keys of a tile

// Portions of prompts. A block takes 64 / G rows (64 queries) of one kv head, and two tiles of keys at a time. Rows of several
// requests may meet in a block: it goes through the requests one after another, the rows of the others sitting out.
// Bound: at 700 rows the walk of the longest block (352 blocks are one wave; while they run the FMA units are busy 39 % of the cycles
// and waits for the result in front lead), with more rows the FMA units and shared-memory reads. 32 heads of 64 on 8, 700 / 2,048
// rows: 175 / 837 us (general kernel 1,009 / 7,738).
template <int HD>
__global__ void __launch_bounds__(128)
attn_f32_rows_kernel(const float* __restrict__ q, long long q_stride, float* __restrict__ out, long long out_stride,
                     const float* __restrict__ kcache, const float* __restrict__ vcache, const int* __restrict__ block_tables,
                     int max_pages, const int* __restrict__ row_seq, const int* __restrict__ positions, int T, int G, int KV,
                     int page_size, int window, float scale) {
    constexpr int LD = HD + 4, DP = HD / 32;         // DP: pairs of features a thread has in the second product
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                // [64][LD]
    float* ks = qs + 64 * LD;                        // [64][LD]
    float* vs = ks + 64 * LD;                        // [64][HD]
    float* ps = vs + 64 * HD;                        // [64 keys][68]
    float2* ab = reinterpret_cast<float2*>(ps + 64 * 68);      // [2 tiles][64]: the factors of a tile's joining
    __shared__ float run_max[64];
    __shared__ int last[64], first[64];              // the keys a query sees in the current request: first .. last (-1: none)
    __shared__ int slot[2][64];
    pdl_launch_dependents();
    pdl_wait(6);
    int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int rows = 64 / G, kvh = blockIdx.y;
    int r0 = (gridDim.x - 1 - blockIdx.x) * rows;    // late rows have the most keys: they go first
    int rn = min(rows, T - r0), nq = rn * G;
#pragma unroll 8
    for (int x = tid / HD; x < 64; x += 128 / HD)
        qs[x * LD + tid % HD] = x < nq ? q[(size_t)(r0 + x / G) * q_stride + (size_t)(kvh * G + x % G) * HD + tid % HD] : 0.f;
    if (tid < 64) run_max[tid] = -INFINITY;
    // first product: queries sq + 8 i, keys sk + 16 j (j / 2 = tile); second: queries 8 og + i, features 4 od .. (+ 64)
    int sq = warp * 2 + (lane >> 4), sk = lane & 15;
    int og = sq, od = sk;
    unsigned long long acc[8][DP];
    float l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        l[i] = 0.f;
#pragma unroll
        for (int d = 0; d < DP; ++d) acc[i][d] = 0;
    }
    for (int a = r0; a < r0 + rn;) {
        int seq = row_seq[a], e = a + 1;
        bool pad = positions[a] < 0;
        while (e < r0 + rn && row_seq[e] == seq && (positions[e] < 0) == pad) ++e;
        int ra = a - r0, rb = e - r0;
        a = e;
        if (pad) continue;
        __syncthreads();
        if (tid < 64) {
            int r = tid / G;
            bool in = r >= ra && r < rb;
            int p = in ? positions[r0 + r] : -1;
            last[tid] = p;
            first[tid] = in && window > 0 ? max(0, p + 1 - window) : 0;
        }
        __syncthreads();
        // (rows of a request ascend, but nothing here rests on it)
        int lo = 0x7fffffff, hi = -1, lo_last = 0x7fffffff, hi_first = 0;
        for (int x = ra * G; x < rb * G; x += G) {
            lo = min(lo, first[x]); hi = max(hi, last[x]);
            lo_last = min(lo_last, last[x]); hi_first = max(hi_first, first[x]);
        }
        const int* bt = block_tables + (size_t)seq * max_pages;
        // where the keys of two tiles lie (-1: no key of this request's), looked up one step ahead
        auto find = [&](int k0) {
            int j = k0 + tid;
            if (tid < 64) slot[k0 >> 6 & 1][tid] = j >= lo && j <= hi ? (bt[j / page_size] * KV + kvh) * page_size + j % page_size : -1;
        };
        find(lo / 64 * 64);
        __syncthreads();
        for (int k0 = lo / 64 * 64; k0 <= hi; k0 += 64) {
            for (int i = tid; i < 64 * (HD / 4); i += 128) {
                int r = i / (HD / 4), d = i % (HD / 4) * 4, at = slot[k0 >> 6 & 1][r];
                cp_async16(ks + r * LD + d, kcache + (size_t)max(at, 0) * HD + d, at >= 0);
                cp_async16(vs + r * HD + d, vcache + (size_t)max(at, 0) * HD + d, at >= 0);
            }
            find(k0 + 64);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // every query of the block sees every key
            bool whole = rb - ra == rows && k0 + 63 <= lo_last && k0 >= hi_first;
            {
                unsigned long long s2[8][4];
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s2[i][j] = 0;
#pragma unroll 2
                for (int d = 0; d < HD; d += 4) {
                    ulonglong2 kf[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) kf[j] = *reinterpret_cast<const ulonglong2*>(ks + (sk + 16 * j) * LD + d);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        ulonglong2 qf = *reinterpret_cast<const ulonglong2*>(qs + (sq + 8 * i) * LD + d);
#pragma unroll
                        for (int j = 0; j < 4; ++j) { fma2(s2[i][j], qf.x, kf[j].x); fma2(s2[i][j], qf.y, kf[j].y); }
                    }
                }
                float mine[2] = {0.f, 0.f};           // the maxima of query sq + 8 (lane & 7)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    int x = sq + 8 * i, xf = first[x], xl = last[x];
                    float s[4], m[2];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        int key = k0 + sk + 16 * j;
                        s[j] = key >= xf && key <= xl ? __fmul_rn(sum2(s2[i][j]), scale) : -INFINITY;
                    }
                    m[0] = fmaxf(s[0], s[1]); m[1] = fmaxf(s[2], s[3]);
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) {
                        m[0] = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], o));
                        m[1] = fmaxf(m[1], __shfl_xor_sync(0xffffffffu, m[1], o));
                    }
                    m[0] = fmaxf(m[0], -FLT_MAX); m[1] = fmaxf(m[1], -FLT_MAX);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        int key = k0 + sk + 16 * j;
                        ps[(sk + 16 * j) * 68 + x] = key >= xf && key <= xl ? expf(s[j] - m[j >> 1]) : 0.f;
                    }
                    if ((lane & 7) == i) { mine[0] = m[0]; mine[1] = m[1]; }
                }
                // lane: query sq + 8 (lane & 7), tile (lane >> 3) & 1; a tile without a key of the query's leaves it alone
                int x = sq + 8 * (lane & 7), xf = first[x], xl = last[x];
                float m = run_max[x];
                bool on0 = xl >= k0 && xf <= k0 + 31 && xf <= xl, on1 = xl >= k0 + 32 && xf <= k0 + 63;
                float m0 = on0 ? fmaxf(m, mine[0]) : m, m1 = on1 ? fmaxf(m0, mine[1]) : m0;
                bool second = lane & 8;
                bool on = second ? on1 : on0;
                float from = second ? m0 : m, to = second ? m1 : m0, mt = second ? mine[1] : mine[0];
                ab[(second ? 64 : 0) + x] = on ? make_float2(expf(from - to), expf(mt - to)) : make_float2(1.f, 0.f);
                __syncwarp();
                if (!second) run_max[x] = m1;
            }
            __syncthreads();
#pragma unroll 1
            for (int t = 0; t < 2; ++t) {
                unsigned long long o[8][DP], lt[4] = {0, 0, 0, 0};
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int d = 0; d < DP; ++d) o[i][d] = 0;
                const float* pr = ps + t * KT * 68 + og * 8;
                const float* vr = vs + t * KT * HD + od * 4;
                int from[8], to[8];                  // a query's keys of the tile, where not every query sees every key
                if (!whole) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) { from[i] = first[og * 8 + i] - k0 - t * KT; to[i] = last[og * 8 + i] - k0 - t * KT; }
                }
                auto key_step = [&](int k, auto masked) {
                    ulonglong2 pa = *reinterpret_cast<const ulonglong2*>(pr + k * 68), pb = *reinterpret_cast<const ulonglong2*>(pr + k * 68 + 4);
                    unsigned long long pp[4] = {pa.x, pa.y, pb.x, pb.y}, vf[DP];
#pragma unroll
                    for (int d = 0; d < DP; d += 2) {
                        ulonglong2 v2 = *reinterpret_cast<const ulonglong2*>(vr + k * HD + d * 32);
                        vf[d] = v2.x; vf[d + 1] = v2.y;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        float2 f = unpack2(pp[i >> 1]);
                        float p = i & 1 ? f.y : f.x;
                        if constexpr (decltype(masked)::value) {
                            if (k < from[i] || k > to[i]) continue;
                        }
                        unsigned long long p2 = pack2(p, p);
#pragma unroll
                        for (int d = 0; d < DP; ++d) fma2(o[i][d], p2, vf[d]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(lt[i]) : "l"(pp[i]));     // a key not seen adds 0
                };
                if (whole) {
#pragma unroll 4
                    for (int k = 0; k < KT; ++k) key_step(k, std::false_type{});
                } else {
#pragma unroll 4
                    for (int k = 0; k < KT; ++k) key_step(k, std::true_type{});
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float2 f = ab[t * 64 + og * 8 + i], x = unpack2(lt[i >> 1]);
                    l[i] = fmaf(l[i], f.x, __fmul_rn(i & 1 ? x.y : x.x, f.y));
#pragma unroll
                    for (int d = 0; d < DP; ++d) {
                        float2 ov = unpack2(o[i][d]), av = unpack2(acc[i][d]);
                        acc[i][d] = pack2(fmaf(av.x, f.x, __fmul_rn(ov.x, f.y)), fmaf(av.y, f.x, __fmul_rn(ov.y, f.y)));
                    }
                }
            }
            __syncthreads();                         // the tiles and the weights have been read
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int x = og * 8 + i;
        if (x >= nq) break;
        bool pad = positions[r0 + x / G] < 0;        // a padding row: no keys, zero output
        float inv = 1.0f / l[i];
        float* op = out + (size_t)(r0 + x / G) * out_stride + (size_t)(kvh * G + x % G) * HD + od * 4;
#pragma unroll
        for (int d = 0; d < DP; ++d) {
            float2 av = unpack2(acc[i][d]);
            op[(d >> 1) * 64 + (d & 1) * 2] = pad ? 0.f : __fmul_rn(av.x, inv);
            op[(d >> 1) * 64 + (d & 1) * 2 + 1] = pad ? 0.f : __fmul_rn(av.y, inv);
        }
    }
}

// Single tokens. A cluster of `c` blocks takes one row of one kv head, 8 c tiles at a time, a tile to a warp; the tiles' sums
// are joined in order, each block a part of the (head, feature) pairs. With more rows than blocks fit at once a block takes
// `rows` of them (c = 1), whose tiles its warps take one after another. Bound: the latency of a tile (its keys and values are
// asked for at once) and of the barriers around the joining, so the blocks are as many as the GPU holds. Back to back, 32 heads of 64
// on 8: one row with 40 / 300 / 4,000 keys 6.3 / 10.5 / 26.5 us (general kernel 13 / 78 / 1,000), 64 rows with 1,000 keys 104 (722), 600 with
// 30 keys 40 (91; a row a block 109).
template <int G, int HD>
__global__ void __launch_bounds__(256, 2)
attn_f32_single_kernel(const float* __restrict__ q, long long q_stride, float* __restrict__ out, long long out_stride,
                       const float* __restrict__ kcache, const float* __restrict__ vcache, const int* __restrict__ block_tables,
                       int max_pages, const int* __restrict__ row_seq, const int* __restrict__ positions, int T, int heads, int KV,
                       int page_size, int window, float scale, int rows, int c) {
    constexpr int DL = HD / 32;                      // features of a lane
    constexpr int PER = HD + 4;                      // floats of a tile's sums for a head: o, m, l
    extern __shared__ __align__(16) float smem[];
    float (*ps)[G][KT] = reinterpret_cast<float (*)[G][KT]>(smem);                              // [8]
    float (*part)[G][PER] = reinterpret_cast<float (*)[G][PER]>(smem + 8 * G * KT);             // [8]
    float* qs = smem + 8 * G * (KT + PER);           // [rows][G * HD]
    // the block's rows; tiles first_of[r] .. first_of[r + 1] - 1 of the block are row r's
    __shared__ int pos_of[8], key_of[8], tile_of[8], seq_of[8], first_of[9];
    pdl_launch_dependents();
    pdl_wait(6);
    int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int rank = blockIdx.x % c, row0 = blockIdx.x / c, apart = gridDim.x / c, kvh = blockIdx.y;
    if (warp == 0) {
        int row = row0 + lane * apart, pos = lane < rows && row < T ? positions[row] : -1;
        int first = window > 0 ? max(0, pos + 1 - window) : 0, upto = pos < 0 ? 0 : pos / KT + 1 - first / KT;
        if (lane < 8) { pos_of[lane] = pos; key_of[lane] = first; tile_of[lane] = first / KT; seq_of[lane] = pos < 0 ? 0 : row_seq[row]; }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        if (lane < 8) first_of[lane + 1] = upto;
        if (lane == 0) first_of[0] = 0;
    }
    for (int i = tid; i < rows * G * HD; i += 256) {
        int row = row0 + i / (G * HD) * apart, e = i % (G * HD);
        qs[i] = row < T && e < heads * HD ? q[(size_t)row * q_stride + (size_t)kvh * heads * HD + e] : 0.f;
    }
    __syncthreads();
    const int tiles = first_of[rows];
    auto out_of = [&](int r) { return out + (size_t)(row0 + r * apart) * out_stride + (size_t)kvh * heads * HD; };
    for (int r = 0; r < rows && rank == 0; ++r)      // a padding row: no keys, zero output
        if (pos_of[r] < 0 && row0 + r * apart < T)
            for (int i = tid; i < heads * HD; i += 256) out_of(r)[i] = 0.f;
    if (c > 1 && tiles <= 8) {                       // a block's worth of tiles: the others leave (and no block of the cluster waits)
        if (rank) return;
        c = 1;
    }
    // this block's (head, feature) pairs of the joining: at most four a thread
    constexpr int MOST = (G * HD + 255) / 256;
    int total = heads * HD, share = (total + c - 1) / c;
    float acc[MOST], l[MOST], m[MOST];
#pragma unroll
    for (int i = 0; i < MOST; ++i) { acc[i] = 0.f; l[i] = 0.f; m[i] = -INFINITY; }
    for (int tr = 0; tr < tiles; tr += 8 * c) {
        int p = tr + rank * 8 + warp;
        if (p < tiles) {
            int r = 0;
            while (p >= first_of[r + 1]) ++r;
            int k0 = (tile_of[r] + p - first_of[r]) * KT, k_lo = max(key_of[r] - k0, 0), k_hi = min(pos_of[r] - k0, KT - 1);    // the tile's keys
            const int* bt = block_tables + (size_t)seq_of[r] * max_pages;
            const float* qr = qs + r * G * HD;
            int j = k0 + lane;
            bool valid = lane >= k_lo && lane <= k_hi;
            int slot = valid ? (bt[j / page_size] * KV + kvh) * page_size + j % page_size : 0;
            float s[G];
            {
                unsigned long long s2[G];
#pragma unroll
                for (int g = 0; g < G; ++g) s2[g] = 0;
                const ulonglong2* kp = reinterpret_cast<const ulonglong2*>(kcache + (size_t)slot * HD);
#pragma unroll(G == 8 ? 4 : 8)
                for (int d = 0; d < HD / 4; ++d) {
                    ulonglong2 kf = valid ? kp[d] : make_ulonglong2(0, 0);
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        ulonglong2 qf = *reinterpret_cast<const ulonglong2*>(qr + g * HD + d * 4);
                        fma2(s2[g], qf.x, kf.x); fma2(s2[g], qf.y, kf.y);
                    }
                }
#pragma unroll
                for (int g = 0; g < G; ++g) s[g] = valid ? __fmul_rn(sum2(s2[g]), scale) : -INFINITY;
            }
            float mt[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                mt[g] = fmaxf(warp_max(s[g]), -FLT_MAX);
                ps[warp][g][lane] = valid ? expf(s[g] - mt[g]) : 0.f;
            }
            __syncwarp();
            unsigned long long o[G][DL / 2];
            float lt[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                lt[g] = 0.f;
#pragma unroll
                for (int d = 0; d < DL / 2; ++d) o[g][d] = 0;
            }
#pragma unroll 1
            for (int kb = k_lo & ~7; kb <= k_hi; kb += 8) {     // eight values' rows on their way at once
                unsigned long long vf[8][DL / 2];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    int sr = __shfl_sync(0xffffffffu, slot, kb + k);
                    const unsigned long long* vp = reinterpret_cast<const unsigned long long*>(vcache + (size_t)sr * HD + lane * DL);
                    bool in = kb + k >= k_lo && kb + k <= k_hi;
#pragma unroll
                    for (int d = 0; d < DL / 2; ++d) vf[k][d] = in ? vp[d] : 0;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (kb + k < k_lo || kb + k > k_hi) continue;
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        float p = ps[warp][g][kb + k];
                        unsigned long long p2 = pack2(p, p);
                        lt[g] = __fadd_rn(lt[g], p);
#pragma unroll
                        for (int d = 0; d < DL / 2; ++d) fma2(o[g][d], p2, vf[k][d]);
                    }
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float* pg = part[warp][g];
#pragma unroll
                for (int d = 0; d < DL / 2; ++d) *reinterpret_cast<unsigned long long*>(pg + lane * DL + 2 * d) = o[g][d];
                if (lane == 0) { pg[HD] = mt[g]; pg[HD + 1] = lt[g]; }
            }
        }
        if (c > 1) cg::this_cluster().sync();
        else __syncthreads();
        for (int b = 0; b < c; ++b) {
            const float* pb = c > 1 ? cg::this_cluster().map_shared_rank(&part[0][0][0], b) : &part[0][0][0];
            int n = min(8, tiles - tr - b * 8);
            if (rows > 1) {                          // tiles of several rows: a row begins, goes on or ends with each
                for (int w = 0; w < n; ++w) {
                    int p = tr + w, r = 0;
                    while (p >= first_of[r + 1]) ++r;
                    bool begins = p == first_of[r], ends = p + 1 == first_of[r + 1];
#pragma unroll
                    for (int i = 0; i < MOST; ++i) {
                        int e = tid + i * 256;
                        if (e >= total) continue;
                        if (begins) { acc[i] = 0.f; l[i] = 0.f; m[i] = -INFINITY; }
                        const float* pw = pb + (w * G + e / HD) * PER;
                        float mt = pw[HD], to = fmaxf(m[i], mt), fa = expf(m[i] - to), fb = expf(mt - to);
                        l[i] = fmaf(l[i], fa, __fmul_rn(pw[HD + 1], fb));
                        acc[i] = fmaf(acc[i], fa, __fmul_rn(pw[e % HD], fb));
                        m[i] = to;
                        if (ends) out_of(r)[e] = __fmul_rn(acc[i], 1.0f / l[i]);
                    }
                }
                continue;
            }
#pragma unroll
            for (int i = 0; i < MOST; ++i) {
                int e = rank * share + tid + i * 256;
                if (e >= min(total, (rank + 1) * share)) continue;
                const float* pe = pb + (e / HD) * PER;
#pragma unroll 4
                for (int w = 0; w < n; ++w) {
                    const float* pw = pe + w * G * PER;
                    float mt = pw[HD], to = fmaxf(m[i], mt), fa = expf(m[i] - to), fb = expf(mt - to);
                    l[i] = fmaf(l[i], fa, __fmul_rn(pw[HD + 1], fb));
                    acc[i] = fmaf(acc[i], fa, __fmul_rn(pw[e % HD], fb));
                    m[i] = to;
                }
            }
        }
        if (c > 1) cg::this_cluster().sync();        // the sums have been read
        else __syncthreads();
    }
    if (rows > 1 || tiles == 0) return;
#pragma unroll
    for (int i = 0; i < MOST; ++i) {
        int e = rank * share + tid + i * 256;
        if (e < min(total, (rank + 1) * share)) out_of(0)[e] = __fmul_rn(acc[i], 1.0f / l[i]);
    }
}

template <int HD>
static int attn_f32_rows(const float* q, long long q_stride, float* out, long long out_stride, const float* kcache, const float* vcache,
                         const int* block_tables, int max_pages, const int* row_seq, const int* positions, int T, int G, int KV,
                         int page_size, int window, float scale, cudaStream_t stream) {
    size_t smem = sizeof(float) * (size_t)(2 * 64 * (HD + 4) + 64 * HD + 64 * 68 + 2 * 2 * 64);
    cudaError_t e = cudaFuncSetAttribute(attn_f32_rows_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    int rows = 64 / G;
    return vob_launch(attn_f32_rows_kernel<HD>, dim3((unsigned)((T + rows - 1) / rows), (unsigned)KV), dim3(128), smem, stream, q, q_stride, out,
                      out_stride, kcache, vcache, block_tables, max_pages, row_seq, positions, T, G, KV, page_size, window, scale);
}

template <int G, int HD>
static int attn_f32_single(const float* q, long long q_stride, float* out, long long out_stride, const float* kcache, const float* vcache,
                           const int* block_tables, int max_pages, const int* row_seq, const int* positions, int T, int heads, int KV,
                           int page_size, int window, float scale, cudaStream_t stream) {
    // a cluster as wide as the GPU has room for with two blocks an SM
    int c = 8;
    while (c > 1 && (long long)T * KV * c > 296) c /= 2;
    // Rows that do not fit at once share blocks: the number whose waves of blocks cost least, a block's start counted as one row. Rows
    // of a block are far apart, so that neighbours with long contexts meet in none.
    int rows = 1;
    long long best = 1LL << 60;
    for (int r = 1; r <= 8 && (long long)T * KV > 296; ++r) {
        long long cost = ((long long)((T + r - 1) / r) * KV + 295) / 296 * (r + 1);
        if (cost <= best) { best = cost; rows = r; }
    }
    const size_t smem = sizeof(float) * (size_t)(8 * G * (KT + HD + 4) + rows * G * HD);
    cudaError_t e = cudaFuncSetAttribute(attn_f32_single_kernel<G, HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((T + rows - 1) / rows * c), (unsigned)KV);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_vob_pdl ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, attn_f32_single_kernel<G, HD>, q, q_stride, out, out_stride, kcache, vcache, block_tables, max_pages, row_seq,
                           positions, T, heads, KV, page_size, window, scale, rows, c);
    return e != cudaSuccess ? (int)e : vob_launch_status();
}

template <int HD>
static int attn_f32(const float* q, long long q_stride, float* out, long long out_stride, const float* kcache, const float* vcache,
                    const int* block_tables, int max_pages, const int* row_seq, const int* positions, int T, int G, int KV,
                    int page_size, int window, float scale, int singles, int portions, cudaStream_t stream) {
    // Few rows make too few blocks for the rows' kernel, and a block of it goes through its requests one after another. What a row costs
    // here grows with the kv heads and, half as fast, with their group; there a step's time hardly depends on either while the blocks
    // fit at once. us here / there, no context and behind 500 to 1,500 keys: 32 heads of 64 on 8, 128 rows of one request 27 / 33 and
    // 174 / 166 (1,000 keys), three requests of 128 rows 58 / 45 and 836 / 334, six of 64 39 / 32 and 821 / 307, ten of 32 19 / 31 and 671 / 317,
    // 64 of 4 9 / 76 and 172 / 440; 4 heads of 64 on 2, one of 300 27 / 53, two of 300 134 / 201 (500 keys); 8 of 64 on one 30 / 50, 130 / 190;
    // 8 heads of 128 on 8, one of 300 106 / 90, two 706 / 328. Short prompts are the usual case of many portions.
    const int rest = T - singles;
    if (portions >= 0 && ((long long)rest * KV * (4 + G) <= 10800 || rest < portions * 64LL)) singles = T;
    if (singles > 0) {
        auto f = G == 1 ? attn_f32_single<1, HD> : G == 2 ? attn_f32_single<2, HD> : G <= 4 ? attn_f32_single<4, HD> : attn_f32_single<8, HD>;
        int e = f(q, q_stride, out, out_stride, kcache, vcache, block_tables, max_pages, row_seq, positions, singles, G, KV, page_size,
                  window, scale, stream);
        if (e || singles == T) return e;
    }
    return attn_f32_rows<HD>(q + singles * q_stride, q_stride, out + singles * out_stride, out_stride, kcache, vcache, block_tables, max_pages,
                             row_seq + singles, positions + singles, T - singles, G, KV, page_size, window, scale, stream);
}

// `singles`: so many of the leading rows are single tokens of requests of their own; `portions`: so many requests bring the rows behind
// them (0: not known; -1: they all go to the portions' kernel). Which kernel computes a row of the 32-bit engine changes its speed,
// not its bits.
VOB_EXPORT int vob_paged_attention(const void* q, long long q_stride, void* out, long long out_stride,
                                   const void* kcache, const void* vcache, int code,
                                   const int* block_tables, int max_pages, const int* row_seq,
                                   const int* positions, int T_rows, int H, int KV, int hd, int page_size,
                                   int window, float scale, int singles, int portions, cudaStream_t stream) {
    if (T_rows <= 0) return 0;
    if (H <= 0 || KV <= 0 || H % KV != 0 || page_size <= 0 || max_pages <= 0) return VOB_ERR_BAD_ARG;
    if (hd <= 0 || hd % 8 != 0 || hd > 256) return VOB_ERR_UNSUPPORTED;
    if (singles < 0 || singles > T_rows || portions < -1) return VOB_ERR_BAD_ARG;
    int G = H / KV;
    // wider groups would not leave a lane of the single-token kernel its registers; KV and T bound the grids
    if (code == VOB_F32 && (hd == 64 || hd == 128) && G <= 8 && KV <= 65535 && T_rows <= (1 << 27) &&
        (((uintptr_t)kcache | (uintptr_t)vcache) & 15) == 0) {
        auto f = hd == 64 ? attn_f32<64> : attn_f32<128>;
        return f((const float*)q, q_stride, (float*)out, out_stride, (const float*)kcache, (const float*)vcache, block_tables, max_pages, row_seq,
                 positions, T_rows, G, KV, page_size, window, scale, singles, portions, stream);
    }
    long long warps = (long long)T_rows * H;
    long long blocks = (warps + 3) / 4;
    if (blocks > 0x7fffffffLL) return VOB_ERR_UNSUPPORTED;
    size_t smem = 4 * (size_t)hd * sizeof(float);
    VOB_DISPATCH_ELEM(code, return vob_launch(paged_attention_warp_kernel<ElemT>, dim3((unsigned)blocks), dim3(128), smem, stream,
        (const ElemT*)q, q_stride, (ElemT*)out, out_stride, (const ElemT*)kcache, (const ElemT*)vcache, block_tables,
        max_pages, row_seq, positions, T_rows, H, KV, hd, page_size, window, scale));
    return 0;
}
