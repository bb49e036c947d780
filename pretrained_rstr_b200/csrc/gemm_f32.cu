// The true 32-bit matrix product: C = epilogue(A[M,K] . W[N,K]^T + bias), plain FMA on
// CUDA cores, no tensor cores and no reduced-precision mode.
//
// ONE order of summation for every size, so that a row's result does not depend on how many
// other rows are in the batch nor on which of the two kernels below computes it: K is cut into
// chunks of 32; a thread accumulates a chunk's even and its odd k's, each in ascending order, and
// adds the two (a pair is what fma.rn.f32x2 takes: half the instructions); the chunks are cut into
// four runs of ceil(chunks / 4), a run's chunk sums are added in ascending order, and the result is
// (run 0 + run 1) + (run 2 + run 3).  (Closer to the 64-bit product than one chain over all of K:
// 1.0e-7 against 4.9e-7 relative at K = 768, 1.3e-7 against 1.0e-6 at 3,072, normal numbers.)
//
// gemm_f32_stream_kernel: up to eight rows a CTA (9 to 16 rows are two groups of CTAs, which read the
// weights each), bound by the weights' way from memory.  Every CTA owns a run of weight rows and
// requests them through a ring of shared-memory stages (TMA where K is a multiple of 32, else
// cp.async; the first of them, where the caller says that the weights are settled, before the kernel
// ahead has ended); a thread keeps its chunk of up to four rows of A in registers and walks the
// weight rows of a stage, so an FMA costs a quarter of a shared-memory operand; chunk sums meet in
// shared memory.  The rows of A come by asynchronous copies, all at once, and what the sums are finished
// with (quotients of run-time counts, bias, residual) is there before them: 8 rows, 2,304 x 768 7.0 -> 6.6 us,
// 768 x 768 4.6 -> 4.2, 3,072 x 768 8.8 -> 8.4, 768 x 3,072 10.4 -> 8.1, 50,257 x 768 81 -> 78 us = 2.0 TB/s; one
// CTA a tile of 64 x 64 (12 CTAs for 768 columns) takes 177 us on average over a model's products.
//
// gemm_f32_tile_kernel: more rows.  Tiles of BM x BN, the four runs of K by the CTAs of a cluster, one or
// two each (a prompt of a few hundred tokens has too few tiles for 148 SMs otherwise), partial tiles added
// through distributed shared memory, a part of the rows a CTA.  Stages come by TMA where the rows allow
// it; a chunk's row is 128 bytes, its 16-byte pieces swizzled.  690 rows: 2,304 x 768 77 -> 76 us, 3,072 x 768
// 101 -> 97, 768 x 768 31 -> 28, 768 x 3,072 109 -> 91, 50,257 x 768 1.50 -> 1.34 ms = 40 TFLOP/s; one CTA a tile
// over all of K 14 TFLOP/s.  What bounds it: the FMA loop.  fma.rn.f32x2 of operands in three registers
// runs at 57 TFLOP/s (72 with two); 255 registers leave two warps a scheduler, which cover neither its
// latency nor that of shared memory whole (counters at 690 x 3,072 x 768: issue slots 38 %, shared memory 59 %).
#include "common.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace {
constexpr int CH = 32;              // k's of a chunk
constexpr int CHP = 36;             // its floats in shared memory: 16-byte reads of neighbouring
                                    // chunks (or rows) by a quarter of a warp hit all banks once

struct Args {
    float* c;
    const float* a;
    const float* w;
    const float* bias;
    const float* resid;
    int m, n, k;
    long lda, ldw, ldc;
    int act;
    bool settled;                   // w may be read before the kernel ahead has ended
    int* status;
    // The stream kernel only: columns of a fused QKV product that also go to the paged cache ([q_width,
    // q_width + kv_width) are keys, the next kv_width values); kv_width == 0: none.
    float* k_pages;                 // [pages][kv heads][page_size][head_dim]
    float* v_pages;
    const int* slots;               // cache slot of each row, -1 = none
    int q_width, kv_width, head_dim, page_size, num_pages;
};

// Where (row, col) also goes in the cache, or null.
__device__ __forceinline__ float* cache_place(const Args& p, int row, int col) {
    if (p.kv_width == 0 || col < p.q_width) return nullptr;
    const int slot = p.slots[row];
    if (slot < 0) return nullptr;
    const unsigned page = (unsigned)slot / (unsigned)p.page_size, off = (unsigned)slot - page * p.page_size;
    if ((int)page >= p.num_pages) {
        prb_set_status(p.status, PRB_S_SLOT_RANGE, row, slot, p.num_pages);
        return nullptr;
    }
    unsigned c = (unsigned)(col - p.q_width);
    float* pages = c < (unsigned)p.kv_width ? p.k_pages : p.v_pages;
    if (c >= (unsigned)p.kv_width) c -= p.kv_width;
    const unsigned h = c / (unsigned)p.head_dim, d = c - h * p.head_dim;
    return pages + (size_t)page * p.kv_width * p.page_size + ((size_t)h * p.page_size + off) * p.head_dim + d;
}

using tc5::mbar_expect_tx;
using tc5::mbar_init;
using tc5::mbar_wait;
using tc5::mbar_try_wait;
using tc5::smem_u32;

// copies `bytes` (0..16) and fills the rest of the 16 bytes with zeros
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One row of `k` floats into padded chunks of shared memory by one warp (zeros beyond K;
// a row outside the matrix, `valid` false, is left alone and `src` only has to be an address).
template <bool VEC>
__device__ __forceinline__ void copy_row(float* dst, const float* src, int k, int nc, int lane) {
    const uint32_t d = smem_u32(dst);
    if (VEC) {
        for (int q = lane; q < nc * (CH / 4); q += 32) {
            const int left = k - q * 4;                       // (a multiple of 4)
            cp16(d + (uint32_t)((q >> 3) * CHP + (q & 7) * 4) * 4u, left > 0 ? src + q * 4 : src,
                 left > 0 ? 16 : 0);
        }
    } else {
        for (int i = lane; i < nc * CH; i += 32)
            cp4(d + (uint32_t)((i >> 5) * CHP + (i & 31)) * 4u, i < k ? src + i : src, i < k ? 4 : 0);
    }
}

// acc += a * b, both halves (each rounded once, as fmaf)
__device__ __forceinline__ void fma2(float2& acc, float ax, float ay, float bx, float by) {
    asm("{\n\t.reg .b64 a, b, c;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(acc.x), "+f"(acc.y) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}

__device__ __forceinline__ float finish(const Args& p, float v, int row, int col) {
    if (p.bias) v += p.bias[col];
    v = prb_activate(v, p.act);
    if (p.resid) v += p.resid[(size_t)row * p.ldc + col];
    return v;
}

// ------------------------------------------------------------------------- a few rows
constexpr int STREAM_THREADS = 256;
constexpr int STREAM_STAGES_MAX = 6;

struct StreamGeo {
    int rows_per_cta;               // weight rows a CTA owns
    int rows;                       // of them in a stage
    int stages;
    int stage_len;                  // floats of a stage
    int nc;                         // chunks of K
    int items, slots;               // (chunk, group of rows of A) pairs; weight rows walked side by side
};

// How the weights come: single floats or 16 bytes by cp.async (chunks padded to CHP floats), or a
// stage at a time by TMA (K a multiple of 32; chunks of 128 bytes, their 16-byte pieces swizzled).
enum { COPY_4 = 0, COPY_16 = 1, COPY_TMA = 2 };

// {32 floats, chunks, rows} of a row-major [n, k] matrix: a copy brings `rows` whole rows, chunk
// after chunk, 128-byte swizzle; x is always 0, so the 16-byte rule on it holds.
int chunk_map(const float* w, int n, int k, long ldw, int rows, CUtensorMap* out) {
    static std::unordered_map<tmap::MapKey, CUtensorMap, tmap::MapKeyHash> cache;
    static std::mutex mu;
    const tmap::MapKey key{w, n, k, ldw, rows};
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return 0;
    }
    auto fn = tmap::encode_fn();
    if (!fn) return -6;
    cuuint64_t dims[3] = {CH, (cuuint64_t)(k / CH), (cuuint64_t)n};
    cuuint64_t strides[2] = {CH * 4, (cuuint64_t)ldw * 4};
    cuuint32_t box[3] = {CH, (cuuint32_t)(k / CH), (cuuint32_t)rows};
    cuuint32_t estr[3] = {1, 1, 1};
    CUtensorMap map;
    if (fn(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(w), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return -5;
    if (cache.size() > 8192) cache.clear();
    cache.emplace(key, map);
    *out = map;
    return 0;
}

template <int MB, int COPY>
__global__ void __launch_bounds__(STREAM_THREADS, 1)
gemm_f32_stream_kernel(Args p, StreamGeo g, const __grid_constant__ CUtensorMap map_w) {
    constexpr int MT = MB < 4 ? MB : 4;                       // rows of A a thread holds
    constexpr bool VEC = COPY != COPY_4;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint64_t bars[STREAM_STAGES_MAX];
    __shared__ int failed_word;
    volatile int* failed = &failed_word;
    // (the swizzle is a function of the address: stages start on 1,024 bytes)
    float* ws = reinterpret_cast<float*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row_len = g.nc * CHP;
    float* as = ws + (size_t)g.stages * g.stage_len;          // [MB][row_len]
    float* part = as + MB * row_len;                          // [2][rows * MB][nc + 1]
    const int part_len = g.rows * MB * (g.nc + 1);
    const int n0 = blockIdx.x * g.rows_per_cta;
    const int n1 = min(p.n, n0 + g.rows_per_cta);
    const int m0 = blockIdx.y * MB;
    const int n_stages = (n1 - n0 + g.rows - 1) / g.rows;
    bool alive = true;
    int issued = 0;                                           // stages thread 0 has asked for
    if (COPY == COPY_TMA) {
        if (tid == 0) {
            for (int s = 0; s < g.stages; ++s) mbar_init(smem_u32(&bars[s]), 1);
            *failed = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads();
    }

    auto load_stage = [&](int s) {
        if constexpr (COPY == COPY_TMA) {
            if (tid == 0 && s < n_stages && alive) {
                const uint32_t bar = smem_u32(&bars[s % g.stages]);
                mbar_expect_tx(bar, (uint32_t)g.rows * g.nc * CH * 4);
                asm volatile(
                    "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                    "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(ws + (size_t)(s % g.stages) * g.stage_len)),
                    "l"(&map_w), "r"(bar), "r"(0), "r"(0), "r"(n0 + s * g.rows)
                    : "memory");
                ++issued;
            }
        } else {
            if (s < n_stages) {
                float* dst = ws + (size_t)(s % g.stages) * g.stage_len;
                for (int r = warp; r < g.rows; r += STREAM_THREADS / 32) {
                    const int n = n0 + s * g.rows + r;
                    if (n < n1) copy_row<VEC>(dst + r * row_len, p.w + (size_t)n * p.ldw, p.k, g.nc, lane);
                }
            }
            cp_commit();
        }
    };
    // weights never depend on the kernel before this one; A does
    for (int s = 0; s < g.stages; ++s) load_stage(s);
    const bool resident = g.items <= STREAM_THREADS;          // a thread keeps one item for good
    const int my_slot = resident ? tid / g.items : 0;
    const int first_item = resident ? tid - my_slot * g.items : tid;
    // the sum this thread finishes in the first round of a stage: a run of output (row of A, weight row)
    const int fin_q = tid & 3, fin_i = (tid >> 2) / g.rows, fin_r = (tid >> 2) - fin_i * g.rows;
    prb_grid_wait();
    prb_grid_launch_dependents();
    for (int r = warp; r < MB; r += STREAM_THREADS / 32) {
        float* dst = as + r * row_len;
        if (COPY == COPY_TMA && m0 + r < p.m) {
            // (all of the row at once: loaded and stored a few pieces at a time, 3,072 columns took
            // six round trips to the L2)
            copy_row<true>(dst, p.a + (size_t)(m0 + r) * p.lda, p.k, g.nc, lane);
        } else if (m0 + r < p.m) {
            const float* src = p.a + (size_t)(m0 + r) * p.lda;
            for (int i = lane * 4; i < g.nc * CH; i += 128) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (VEC) {
                    if (i < p.k) v = *reinterpret_cast<const float4*>(src + i);
                } else {
                    if (i < p.k) v.x = src[i];
                    if (i + 1 < p.k) v.y = src[i + 1];
                    if (i + 2 < p.k) v.z = src[i + 2];
                    if (i + 3 < p.k) v.w = src[i + 3];
                }
                *reinterpret_cast<float4*>(dst + (i >> 5) * CHP + (i & 31)) = v;
            }
        } else {
            for (int i = lane * 4; i < row_len; i += 128)
                *reinterpret_cast<float4*>(dst + i) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    if (COPY == COPY_TMA) {
        cp_commit();
        cp_wait<0>();
    }
    __syncthreads();

    float4 av[MT][CH / 4];
    auto load_a = [&](int item) {
        const int c = item % g.nc, group = item / g.nc;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < CH / 4; ++j)
                av[i][j] = *reinterpret_cast<const float4*>(as + (group * MT + i) * row_len + c * CHP + j * 4);
    };
    if (resident && my_slot < g.slots) load_a(first_item);

    const int run = (g.nc + 3) / 4;
    for (int s = 0; s < n_stages; ++s) {
        // what the first round's sums are finished with is asked for before the stage is waited for
        const int fin_row = m0 + fin_i, fin_col = n0 + s * g.rows + fin_r;
        const bool fin = fin_q == 0 && fin_i < MB && fin_row < p.m && fin_r < min(g.rows, n1 - (n0 + s * g.rows));
        const float fin_bias = fin && p.bias ? p.bias[fin_col] : 0.0f;
        const float fin_resid = fin && p.resid ? p.resid[(size_t)fin_row * p.ldc + fin_col] : 0.0f;
        float* const fin_cache = fin ? cache_place(p, fin_row, fin_col) : nullptr;
        if constexpr (COPY == COPY_TMA) {
            alive = alive && mbar_wait(smem_u32(&bars[s % g.stages]), (uint32_t)(s / g.stages) & 1u, failed);
        } else {
            // all groups but the (stages - 1) newest have landed: stage s among them
            switch (g.stages) {
                case 1: cp_wait<0>(); break;
                case 2: cp_wait<1>(); break;
                case 3: cp_wait<2>(); break;
                case 4: cp_wait<3>(); break;
                case 5: cp_wait<4>(); break;
                default: cp_wait<5>(); break;
            }
            __syncthreads();
        }
        const float* wst = ws + (size_t)(s % g.stages) * g.stage_len;
        float* pt = part + (s & 1) * part_len;
        const int rows = min(g.rows, n1 - (n0 + s * g.rows));
        for (int item = first_item; item < g.items; item += STREAM_THREADS) {
            if (my_slot >= g.slots) break;
            if (!resident) load_a(item);
            const int c = item % g.nc, group = item / g.nc;
            for (int r = my_slot; r < rows; r += g.slots) {
                const float* wr = COPY == COPY_TMA ? wst + (r * g.nc + c) * CH : wst + r * row_len + c * CHP;
                const int swz = COPY == COPY_TMA ? (r * g.nc + c) & 7 : 0;
                float2 acc[MT];
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int j = 0; j < CH / 4; ++j) {
                    const float4 wv = *reinterpret_cast<const float4*>(wr + (j ^ swz) * 4);
#pragma unroll
                    for (int i = 0; i < MT; ++i) {
                        fma2(acc[i], av[i][j].x, av[i][j].y, wv.x, wv.y);
                        fma2(acc[i], av[i][j].z, av[i][j].w, wv.z, wv.w);
                    }
                }
#pragma unroll
                for (int i = 0; i < MT; ++i)
                    pt[((group * MT + i) * g.rows + r) * (g.nc + 1) + c] = acc[i].x + acc[i].y;
            }
        }
        __syncthreads();
        if (COPY == COPY_TMA) alive = alive && !*failed;      // one thread that gave up is enough
        load_stage(s + g.stages);
        // four threads an output, a run of chunk sums each
        for (int t0 = 0; t0 < g.rows * MB * 4; t0 += STREAM_THREADS) {
            const int t = t0 + tid;
            const int q = t & 3, o = t >> 2;
            const int i = t0 == 0 ? fin_i : o / g.rows, r = t0 == 0 ? fin_r : o - i * g.rows;
            float sum = 0.0f;
            const bool live = o < g.rows * MB && r < rows && m0 + i < p.m && alive;
            if (live) {
                const float* src = pt + o * (g.nc + 1);
                for (int c = q * run; c < min(g.nc, (q + 1) * run); ++c) sum += src[c];
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if (live && q == 0) {
                const int row = m0 + i, col = n0 + s * g.rows + r;
                float v;
                if (t0 == 0) {
                    v = sum;
                    if (p.bias) v += fin_bias;
                    v = prb_activate(v, p.act);
                    if (p.resid) v += fin_resid;
                } else {
                    v = finish(p, sum, row, col);
                }
                p.c[(size_t)row * p.ldc + col] = v;
                float* const cached = t0 == 0 ? fin_cache : cache_place(p, row, col);
                if (cached != nullptr) *cached = v;
            }
        }
    }
    if constexpr (COPY == COPY_TMA) {
        if (tid == 0 && !alive) {
            prb_set_status(p.status, PRB_S_WAIT_TIMEOUT, 40, blockIdx.x, blockIdx.y);
            for (int s = max(0, issued - g.stages); s < issued; ++s)       // copies in flight, bounded
                for (uint32_t i = 0; i < tc5::WAIT_LIMIT; ++i)
                    if (mbar_try_wait(smem_u32(&bars[s % g.stages]), (uint32_t)(s / g.stages) & 1u)) break;
        }
    } else {
        cp_wait<0>();
    }
}

// ------------------------------------------------------------------------- many rows
// {32 floats, rows} of a row-major [rows, k] matrix, 128-byte swizzle, zeros beyond both; x is a
// multiple of 32 floats, so the 16-byte rule on it holds.
int tile_map(const float* t, int rows, int k, long ld, int box_rows, CUtensorMap* out) {
    static std::unordered_map<tmap::SlabKey, CUtensorMap, tmap::SlabKeyHash> cache;
    static std::mutex mu;
    const tmap::SlabKey key{t, rows, k, ld, box_rows, 1};
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return 0;
    }
    auto fn = tmap::encode_fn();
    if (!fn) return -6;
    cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {CH, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUtensorMap map;
    if (fn(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(t), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return -5;
    if (cache.size() > 8192) cache.clear();
    cache.emplace(key, map);
    *out = map;
    return 0;
}

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr, uint32_t rank) {
    uint32_t r;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r));
    return v;
}
__device__ __forceinline__ int ld_cluster1(uint32_t addr, uint32_t rank) {
    uint32_t r;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(r) : "memory");
    return v;
}
// two neighbouring floats as fma.rn.f32x2 takes them, four of them by one read of shared memory
typedef unsigned long long pair_t;
__device__ __forceinline__ void fma_pairs(pair_t& acc, pair_t a, pair_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float add_pair(pair_t v) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    return x + y;
}

// RUNS: runs of K a CTA takes (the others of the four are its cluster's)
template <int BM, int BN, int TM, int TN, int RUNS> struct TileCfg {
    static constexpr int THREADS = (BM / TM) * (BN / TN);
    static constexpr int STAGE = (BM + BN) * CH;              // floats
    static constexpr int STAGES = BN > 64 ? 2 : 4;            // (of 24 KB: a chunk's FMAs take several times its copies' way)
    static constexpr int HELD = RUNS - 1;                     // runs' sums set aside
    static constexpr int OUT_LD = BN + 4;
    static constexpr int RING = STAGES * STAGE > BM * OUT_LD ? STAGES * STAGE : BM * OUT_LD;
    static constexpr size_t SMEM = 1024 + sizeof(float) * ((size_t)RING + (size_t)HELD * BM * BN);
};

// grid (cluster x column tiles, row tiles), clusters of 4 / RUNS along x: CTA q sums runs RUNS * q ..
template <int BM, int BN, int TM, int TN, int COPY, int RUNS>
__global__ void __cluster_dims__(4 / RUNS, 1, 1) __launch_bounds__((BM / TM) * (BN / TN), TM * TN <= 32 ? 3 : 2)
gemm_f32_tile_kernel(Args p, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w) {
    using Cfg = TileCfg<BM, BN, TM, TN, RUNS>;
    constexpr int NT = Cfg::THREADS, CL = 4 / RUNS, TILE_STAGES = Cfg::STAGES;
    static_assert(RUNS == 1 || RUNS == 2, "one run or two");
    constexpr int TY = BM / TM, TX = BN / TN;
    static_assert(TX % 8 == 0 && TY % 8 == 0, "a warp is 8 columns by 4 rows of threads; a thread's rows share a swizzle");
    extern __shared__ __align__(16) uint8_t tile_raw[];
    __shared__ uint64_t bars[TILE_STAGES];
    __shared__ int failed_word;
    volatile int* failed = &failed_word;
    float* smem = reinterpret_cast<float*>(((uintptr_t)tile_raw + 1023) & ~(uintptr_t)1023);
    float* held = smem + Cfg::RING;                           // [TM * TN][NT]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % (TX / 8)) * 8 + (lane & 7);
    const int ty = (warp / (TX / 8)) * 4 + (lane >> 3);
    const int part = blockIdx.x % CL;
    const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / CL) * BN;
    const int nc = (p.k + CH - 1) / CH, run = (nc + 3) / 4;
    const int c0 = min(nc, part * RUNS * run), c1 = min(nc, c0 + RUNS * run);
    if (COPY == COPY_TMA && tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        for (int s = 0; s < TILE_STAGES; ++s) mbar_init(smem_u32(&bars[s]), 1);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }

    bool alive = true;
    // rows [0, BM) of a stage are A's, the next BN W's; rows outside the matrices are zeros.  A row is
    // a chunk of 128 bytes, its 16-byte pieces swizzled with the row.
    auto load_rows = [&](int c, bool weights) {
        if (c >= c1) return;
        const int s = (c - c0) % TILE_STAGES;
        float* st = smem + s * Cfg::STAGE + (weights ? BM * CH : 0);
        if constexpr (COPY == COPY_TMA) {
            // (only after its own wait for the stage's last copy, which may else still be on its way)
            if (tid == 0 && alive) {
                const uint32_t bar = smem_u32(&bars[s]);
                if (weights) mbar_expect_tx(bar, Cfg::STAGE * 4);
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                    "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(st)),
                    "l"(weights ? &map_w : &map_a), "r"(bar), "r"(c * CH), "r"(weights ? n0 : m0)
                    : "memory");
            }
        } else {
            const float* base = weights ? p.w : p.a;
            const long ld = weights ? p.ldw : p.lda;
            const int first = weights ? n0 : m0, end = weights ? p.n : p.m;
            constexpr int PER = COPY == COPY_16 ? CH / 4 : CH;
            const int rows = weights ? BN : BM;
            for (int i = tid; i < rows * PER; i += NT) {
                const int r = i / PER, e = (i % PER) * (CH / PER);
                const bool in = first + r < end && c * CH + e < p.k;
                const float* src = in ? base + (size_t)(first + r) * ld + c * CH + e : base;
                const uint32_t dst = smem_u32(st + r * CH + (((e >> 2) ^ (r & 7)) << 2) + (e & 3));
                if (COPY == COPY_16) cp16(dst, src, in ? 16 : 0);
                else cp4(dst, src, in ? 4 : 0);
            }
        }
    };
    if (COPY == COPY_TMA) __syncthreads();
    for (int s = 0; s < TILE_STAGES; ++s) load_rows(c0 + s, true);
    prb_grid_wait();
    prb_grid_launch_dependents();
    for (int s = 0; s < TILE_STAGES; ++s) {
        load_rows(c0 + s, false);
        if (COPY != COPY_TMA) cp_commit();
    }

    float sum[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sum[i][j] = 0.0f;
    const uint32_t sw_a = (uint32_t)(ty & 7), sw_w = (uint32_t)(tx & 7);
    int c = c0;
#pragma unroll 1
    for (int r = 0; r < RUNS; ++r) {
        const int end = min(c1, c0 + (r + 1) * run);
#pragma unroll 1
        for (; c < end; ++c) {
            const int s = (c - c0) % TILE_STAGES;
            if constexpr (COPY == COPY_TMA) {
                if (alive && !mbar_wait(smem_u32(&bars[s]), (uint32_t)((c - c0) / TILE_STAGES) & 1u, failed)) {
                    alive = false;
                    for (int i = c; tid == 0 && i < min(c1, c + TILE_STAGES); ++i)       // copies in flight, bounded
                        for (uint32_t w = 0; w < tc5::WAIT_LIMIT; ++w)
                            if (mbar_try_wait(smem_u32(&bars[(i - c0) % TILE_STAGES]), (uint32_t)((i - c0) / TILE_STAGES) & 1u)) break;
                }
            } else {
                cp_wait<TILE_STAGES - 1>();
                __syncthreads();
            }
            const float* ap = smem + s * Cfg::STAGE + ty * CH;
            const float* wp = smem + s * Cfg::STAGE + (BM + tx) * CH;
            pair_t acc[TM][TN];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = 0;
#pragma unroll
            for (uint32_t e = 0; e < CH / 4; ++e) {
                const float *ea = ap + ((e ^ sw_a) << 2), *ew = wp + ((e ^ sw_w) << 2);
                ulonglong2 wv[TN];
#pragma unroll
                for (int j = 0; j < TN; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(ew + j * TX * CH);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(ea + i * TY * CH);
#pragma unroll
                    for (int j = 0; j < TN; ++j) fma_pairs(acc[i][j], av.x, wv[j].x);
#pragma unroll
                    for (int j = 0; j < TN; ++j) fma_pairs(acc[i][j], av.y, wv[j].y);
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) sum[i][j] += add_pair(acc[i][j]);
            __syncthreads();                                  // the stage has been read
            load_rows(c + TILE_STAGES, true);
            load_rows(c + TILE_STAGES, false);
            if (COPY != COPY_TMA) cp_commit();
        }
        // two runs are added, then the two sums of two
        if constexpr (RUNS == 2) {
            float* mine = held + tid;
#pragma unroll
            for (int i = 0; i < TM * TN; ++i) {
                if (r == 0) {
                    mine[i * NT] = sum[i / TN][i % TN];
                    sum[i / TN][i % TN] = 0.0f;
                } else {
                    sum[i / TN][i % TN] = mine[i * NT] + sum[i / TN][i % TN];
                }
            }
        }
    }
    if (COPY != COPY_TMA) {
        cp_wait<0>();
    } else if (tid == 0 && *failed) {                         // (the last chunk's barrier is behind every wait)
        prb_set_status(p.status, PRB_S_WAIT_TIMEOUT, 41, blockIdx.x, blockIdx.y);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) smem[(ty + i * TY) * Cfg::OUT_LD + tx + j * TX] = sum[i][j];
    cluster_sync_all();
    // a part of the rows, four columns at a time; all remote reads are asked for at once (one
    // after the other they cost 25 us a 128 x 128 tile, twice the tile's FMAs)
    constexpr int ROWS = BM / CL, PER = ROWS * (BN / 4) / NT, AT_ONCE = PER < 4 ? PER : 4;
    static_assert(ROWS * (BN / 4) % NT == 0 && PER % AT_ONCE == 0, "whole rounds");
    const int r0 = part * ROWS;
    const bool whole = p.ldc % 4 == 0 && ((uintptr_t)p.c) % 16 == 0;
#pragma unroll
    for (int i0 = 0; i0 < PER; i0 += AT_ONCE) {
        float4 v[AT_ONCE][CL];
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            const int e = tid + (i0 + i) * NT;
            const uint32_t at = smem_u32(smem + (r0 + e / (BN / 4)) * Cfg::OUT_LD + (e % (BN / 4)) * 4);
#pragma unroll
            for (int q = 0; q < CL; ++q) v[i][q] = ld_cluster4(at, q);
        }
        // a partial tile that a CTA of the cluster gave up on is in nobody's sums
        if (COPY == COPY_TMA && i0 == 0) {
            int any = 0;
#pragma unroll
            for (int q = 0; q < CL; ++q) any |= ld_cluster1(smem_u32(&failed_word), q);
            alive = any == 0;
        }
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            const int e = tid + (i0 + i) * NT;
            const int row = m0 + r0 + e / (BN / 4), col = n0 + (e % (BN / 4)) * 4;
            if (row >= p.m || !alive) continue;
            float4 x = v[i][0];
            if constexpr (CL == 2) {
                x = make_float4(x.x + v[i][1].x, x.y + v[i][1].y, x.z + v[i][1].z, x.w + v[i][1].w);
            } else {
                const float4 y = v[i][1], z = v[i][2], w = v[i][3];
                x = make_float4((x.x + y.x) + (z.x + w.x), (x.y + y.y) + (z.y + w.y),
                                (x.z + y.z) + (z.z + w.z), (x.w + y.w) + (z.w + w.w));
            }
            const float t[4] = {x.x, x.y, x.z, x.w};
            float y[4];
#pragma unroll
            for (int d = 0; d < 4; ++d) y[d] = col + d < p.n ? finish(p, t[d], row, col + d) : 0.0f;
            float* out = p.c + (size_t)row * p.ldc + col;
            if (whole && col + 4 <= p.n) {
                *reinterpret_cast<float4*>(out) = make_float4(y[0], y[1], y[2], y[3]);
            } else {
                for (int d = 0; d < 4; ++d)
                    if (col + d < p.n) out[d] = y[d];
            }
        }
    }
    __syncwarp();
    cluster_sync_all();                                       // nobody leaves while its tile is read
}

template <int BM, int BN, int TM, int TN, int COPY, int RUNS>
int launch_tile_by(const Args& p, cudaStream_t stream) {
    using Cfg = TileCfg<BM, BN, TM, TN, RUNS>;
    CUtensorMap map_a = {}, map_w = {};
    if (COPY == COPY_TMA) {
        int rc = tile_map(p.a, p.m, p.k, p.lda, BM, &map_a);
        if (rc == 0) rc = tile_map(p.w, p.n, p.k, p.ldw, BN, &map_w);
        if (rc) return rc;
    }
    constexpr auto kernel = gemm_f32_tile_kernel<BM, BN, TM, TN, COPY, RUNS>;
    cudaError_t e = prb_allow_shared<kernel>((int)Cfg::SMEM);
    if (e != cudaSuccess) return (int)e;
    dim3 grid((4 / RUNS) * ((p.n + BN - 1) / BN), (p.m + BM - 1) / BM);
    if (grid.y > 65535) return PRB_E_SIZE;
    e = prb_launch_maybe_early(p.settled, kernel, grid, dim3(Cfg::THREADS), Cfg::SMEM, stream, p, map_a, map_w);
    return e == cudaSuccess ? 0 : (int)e;
}

template <int BM, int BN, int TM, int TN, int RUNS>
int launch_tile(const Args& p, int copy, cudaStream_t stream) {
    return copy == COPY_TMA  ? launch_tile_by<BM, BN, TM, TN, COPY_TMA, RUNS>(p, stream)
           : copy == COPY_16 ? launch_tile_by<BM, BN, TM, TN, COPY_16, 1>(p, stream)
                             : launch_tile_by<BM, BN, TM, TN, COPY_4, 1>(p, stream);
}
// Clusters of an instance that run side by side, as the device says (asked once per device).
template <int BM, int BN, int TM, int TN, int RUNS>
int active_clusters() {
    using Cfg = TileCfg<BM, BN, TM, TN, RUNS>;
    constexpr auto kernel = gemm_f32_tile_kernel<BM, BN, TM, TN, COPY_TMA, RUNS>;
    static std::atomic<int> known[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    int n = known[dev].load(std::memory_order_relaxed);
    if (n > 0) return n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(4 / RUNS);
    cfg.blockDim = dim3(Cfg::THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 4 / RUNS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (prb_allow_shared<kernel>((int)Cfg::SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess)
        cudaGetLastError();
    n = n > 0 ? n : 1;
    known[dev].store(n, std::memory_order_relaxed);
    return n;
}
// Which tiles a product takes: 3 (64 x 64), 4 or 5 (64 x 128, one run or two a CTA).  What a launch costs is
// counted in rounds of the clusters that the device runs side by side, a round in chunks of K: those of a CTA
// and one and a half for its first copies and its part of the cluster's sums.  A last round that leaves the SMs
// fewer CTAs than they hold (2 of 64 x 128, 3 of 64 x 64) is shorter; not where it is the only one, since a launch
// that is placed early fills the SMs that the kernel ahead leaves first (logits of three texts, whose 768 columns
// are 72 tiles: 8.19 ms with two runs there, a CTA an SM, 7.45 as it is).  A chunk of 64 x 64 takes 0.82 of one of
// 64 x 128.  us of 3 / 4 / 5 by tiles of 64 x 128 at K = 768 (104 / 71 / 148 clusters side by side): 48 22.0 / 27.3 /
// 32.8, 54 29.4 / 27.6 / 32.9, 70 35.9 / 27.7 / 33.1, 75 37.0 / 40.4 / 49.9, 90 41.6 / 41.0 / 50.3, 132 54.7 / 54.0 /
// 50.7, 264 101 / 98.3 / 97.0, 4,323 1,517 / 1,474 / 1,344; at K = 3,072 90 145 / 138 / 179, 198 282 / 261 / 268.  It
// is off most at 108 tiles (48.5 / 51.9 / 50.3: it takes 5).  (All four runs in a CTA leave room for one an SM: 1,831
// at 4,323.)
int tile_rule(long m, long n, int k, bool two_runs, bool only_wide) {
    const long rows = (m + 63) / 64, big = rows * ((n + 127) / 128), small = rows * ((n + 63) / 64);
    const int run = ((k + CH - 1) / CH + 3) / 4;
    auto cost = [](long clusters, int active, int held, const double* last, double chunks) {
        const long full = clusters / active, rest = clusters % active;
        if (full == 0) return chunks;
        return chunks * ((double)full + (rest == 0 ? 0.0 : last[(rest * held + active - 1) / active - 1]));
    };
    static const double last2[] = {0.6, 1.0}, last3[] = {0.48, 0.71, 1.0};
    const double of3 = cost(small, active_clusters<64, 64, 8, 4, 1>(), 3, last3, 0.82 * (run + 1.5));
    const double of4 = cost(big, active_clusters<64, 128, 8, 8, 1>(), 2, last2, run + 1.5);
    const double of5 = two_runs ? cost(big, active_clusters<64, 128, 8, 8, 2>(), 2, last2, 2 * run + 1.5) : of4;
    return !only_wide && of3 < of4 && of3 < of5 ? 3 : of5 < of4 ? 5 : 4;
}

constexpr size_t STREAM_SMEM = 220 * 1024;                    // the most a launch of the stream kernel takes

template <int MB, int COPY>
int launch_stream_by(const Args& p, StreamGeo g, size_t smem, cudaStream_t stream) {
    CUtensorMap map = {};
    if (COPY == COPY_TMA) {
        const int rc = chunk_map(p.w, p.n, p.k, p.ldw, g.rows, &map);
        if (rc) return rc;
    }
    constexpr auto kernel = gemm_f32_stream_kernel<MB, COPY>;
    cudaError_t e = prb_allow_shared<kernel>((int)STREAM_SMEM);
    if (e != cudaSuccess) return (int)e;
    dim3 grid((p.n + g.rows_per_cta - 1) / g.rows_per_cta, (p.m + MB - 1) / MB);
    e = prb_launch_maybe_early(p.settled, kernel, grid, dim3(STREAM_THREADS), smem, stream, p, g, map);
    return e == cudaSuccess ? 0 : (int)e;
}

template <int MB>
int launch_stream(const Args& p, StreamGeo g, int copy, size_t smem, cudaStream_t stream) {
    return copy == COPY_TMA  ? launch_stream_by<MB, COPY_TMA>(p, g, smem, stream)
           : copy == COPY_16 ? launch_stream_by<MB, COPY_16>(p, g, smem, stream)
                             : launch_stream_by<MB, COPY_4>(p, g, smem, stream);
}

// The stream kernel's geometry for `mb` rows of A a CTA; false if it does not fit.
bool stream_geometry(const Args& p, int mb, int copy, StreamGeo* g, size_t* smem) {
    const size_t budget = STREAM_SMEM;
    const int sms = prb_sm_count();
    const int mt = mb < 4 ? mb : 4;
    g->nc = (p.k + CH - 1) / CH;
    g->items = g->nc * (mb / mt);
    g->slots = g->items <= STREAM_THREADS ? STREAM_THREADS / g->items : 1;
    const int groups = (p.m + mb - 1) / mb;
    const int ctas = sms / groups > 0 ? sms / groups : 1;     // one to an SM
    g->rows_per_cta = (p.n + ctas - 1) / ctas;
    const size_t row = (size_t)g->nc * CHP * 4, w_row = (size_t)g->nc * (copy == COPY_TMA ? CH : CHP) * 4;
    auto stage_bytes = [&](int rows) { return (rows * w_row + 1023) / 1024 * 1024; };
    auto bytes = [&](int rows, int stages) {
        return 1024 + (size_t)mb * row + stages * stage_bytes(rows) + 2ull * rows * mb * (g->nc + 1) * 4;
    };
    // about ten weight rows a stage (a stage costs two block barriers), at least two stages
    // unless one holds all the CTA has; slots that have no row in a round stand idle
    int best = 0;
    for (int rows = 1; rows <= 12 && rows <= g->rows_per_cta; ++rows) {
        const bool whole = rows >= g->rows_per_cta;
        if (bytes(rows, whole ? 1 : 2) > budget) break;
        if (rows % g->slots == 0 || best == 0 || whole || rows < g->slots) best = rows;
    }
    if (best == 0) return false;
    const int wanted = (g->rows_per_cta + best - 1) / best;
    best = (g->rows_per_cta + wanted - 1) / wanted;           // (stages of equal size)
    g->rows = best;
    g->stage_len = (int)(stage_bytes(best) / 4);
    g->stages = 1;
    while (g->stages < wanted && g->stages < STREAM_STAGES_MAX && bytes(best, g->stages + 1) <= budget)
        ++g->stages;
    *smem = bytes(best, g->stages);
    return true;
}
// The same for the most rows of A a CTA can hold; returns them, 0 where even one does not fit.
int stream_rows(const Args& p, int copy, StreamGeo* g, size_t* smem) {
    for (int mb = p.m == 1 ? 1 : p.m == 2 ? 2 : p.m <= 4 ? 4 : 8; mb >= 1; mb /= 2)
        if (stream_geometry(p, mb, copy, g, smem)) return (p.m + mb - 1) / mb <= 65535 ? mb : 0;
    return 0;
}
constexpr int STREAM_ROWS = 16;                               // most rows that take the stream kernel by themselves
}  // namespace

// which: 0 the rule below; 1 the stream kernel where it fits, 2 / 3 tiles of 64 x 128, 64 x 64, 4 / 5 tiles of
// 64 x 128 of one run and of two runs a CTA (the same bits from all of them).  settled: w was written long before (by no kernel of the step), so the
// launch may be placed, and w read, before the kernel ahead in the stream has ended.
// kv_width > 0 (where prb_gemm_f32_scatters says so, else refused): the product is a fused QKV
// projection, whose key and value columns also go to the paged cache (float32, contiguous) at slots[row]: 8
// requests generating 24 tokens 19.2 -> 19.0 ms.  (In the tiles' epilogue it cost more than the append
// behind them: three prompts of 301 tokens 7.36 -> 7.49 ms.)
PRB_API int prb_gemm_f32(float* c, const float* a, const float* w, const float* bias,
                         const float* resid, int m, int n, int k, long lda, long ldw, long ldc,
                         int act, int which, int settled, float* k_pages, float* v_pages,
                         const int* slots, int q_width, int kv_width, int head_dim, int page_size,
                         int num_pages, int* status, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0) return PRB_E_SIZE;
    if (kv_width != 0 && (kv_width < 0 || head_dim <= 0 || kv_width % head_dim != 0 || page_size <= 0 || q_width < 0 ||
                          q_width + 2 * kv_width != n || k_pages == nullptr || v_pages == nullptr || slots == nullptr))
        return PRB_E_ARG;
    const Args p{c, a, w, bias, resid, m, n, k, lda, ldw, ldc, act, settled != 0, status,
                 k_pages, v_pages, slots, q_width, kv_width, head_dim, page_size, num_pages};
    // 16-byte copies where every row starts on 16 bytes and K ends on them, else single floats
    const bool vec = k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)a) % 16 == 0 &&
                     ((uintptr_t)w) % 16 == 0;
    // Up to 16 rows the stream kernel.  us as a stream / as tiles: 8 rows, 768 x 768 4.2 / 10.8, 2,304 x 768 6.7 / 15.0,
    // 50,257 x 768 78 / 137; 16 rows 4.9 / 11.0, 10.2 / 15.3, 148 / 139; 32 rows 7.4 / 11.1, 18.1 / 15.3, 292 / 144.
    if (which == 1 || (which == 0 && m <= STREAM_ROWS)) {
        StreamGeo g;
        size_t smem;
        // (rows that overlap, an expanded row for one, are no tensor that a copy engine's map describes)
        const int copy = !vec ? COPY_4 : k % CH == 0 && k / CH <= 256 && ldw >= k ? COPY_TMA : COPY_16;
        switch (stream_rows(p, copy, &g, &smem)) {
            case 1: return launch_stream<1>(p, g, copy, smem, stream);
            case 2: return launch_stream<2>(p, g, copy, smem, stream);
            case 4: return launch_stream<4>(p, g, copy, smem, stream);
            case 8: return launch_stream<8>(p, g, copy, smem, stream);
        }
    }
    if (kv_width != 0) return PRB_E_SIZE;
    // (rows that overlap are no tensor that a copy engine's map describes)
    const int tiled = !vec ? COPY_4 : ldw >= k && lda >= k ? COPY_TMA : COPY_16;
    const int kind = which >= 3 && which <= 5 ? which : tile_rule(m, n, k, tiled == COPY_TMA, which == 2);
    if (kind == 3) return launch_tile<64, 64, 8, 4, 1>(p, tiled, stream);
    return kind == 5 ? launch_tile<64, 128, 8, 8, 2>(p, tiled, stream)
                     : launch_tile<64, 128, 8, 8, 1>(p, tiled, stream);
}
// Whether prb_gemm_f32 brings key and value columns to the cache: whether the stream kernel takes the sizes,
// however the rows are aligned.
PRB_API int prb_gemm_f32_scatters(int m, int n, int k) {
    if (m <= 0 || n <= 0 || k <= 0 || m > STREAM_ROWS) return 0;
    Args p{};
    p.m = m; p.n = n; p.k = k;
    StreamGeo g;
    size_t smem;
    return stream_rows(p, COPY_4, &g, &smem) > 0 && stream_rows(p, COPY_TMA, &g, &smem) > 0;
}
// The tiles that a product of more than 16 rows takes (3, 4 or 5, as above), and how many clusters of each kind
// run side by side.
PRB_API int prb_gemm_f32_tiles(int m, int n, int k, int* side_by_side) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    side_by_side[0] = active_clusters<64, 64, 8, 4, 1>();
    side_by_side[1] = active_clusters<64, 128, 8, 8, 1>();
    side_by_side[2] = active_clusters<64, 128, 8, 8, 2>();
    return tile_rule(m, n, k, true, false);
}
