// Matrix product for a few dozen rows (17..64 tokens: decoding a large batch) with the
// reduction dimension split over a thread-block cluster:
//
//     C[M,N] = act(A[M,K] . W[N,K]^T + bias[N]) (+ resid[M,N]),   M <= 64, K % 64 == 0
//
// With so few rows a product has too few output tiles to fill the GPU when every tile walks
// all of K (N = 768: 12 tiles of 64 columns), and what bounds a tile is the bytes its SM
// takes in.  Here a cluster of S CTAs shares one tile of NB output columns: CTA r multiplies
// the r-th part of K (A and W slices come by TMA through a ring of shared-memory stages,
// 128-byte swizzle, mma.sync m16n8k16 with ldmatrix) and writes row i of its partial tile to
// the shared memory of CTA i mod S, which after one cluster barrier sums its rows' parts in rank
// order and runs the epilogue for them (bias, activation, residual, store).  (Parts that their owner
// reads after the barrier cost a remote round trip and a second barrier more: 768 x 3,072 at 64 rows
// 8.4 us in a step without dependent launch, 7.2 so.)  S depends on K, N and how many clusters the
// device runs at a time, and a row's sum is taken in a fixed order, so a row's result does not depend
// on the batch.
// No TMA load uses cluster multicast.  Every mbarrier wait is bounded: on a timeout the
// kernel records PRB_S_WAIT_TIMEOUT, stores nothing, waits (bounded) for its copies in
// flight and leaves through the same cluster barriers as its peers.
#include <mutex>

#include "common.cuh"
#include "tensor_map.cuh"

#ifdef PRB_TRACE
__device__ unsigned long long g_midm_trace[512 * 8];
#define MT_TRACE(slot)                                                                \
    do {                                                                              \
        const int cta__ = blockIdx.z * gridDim.x + blockIdx.x;                        \
        if (threadIdx.x == 0 && cta__ < 512) {                                        \
            unsigned long long t__;                                                   \
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t__));                   \
            g_midm_trace[cta__ * 8 + (slot)] = t__;                                   \
        }                                                                             \
    } while (0)
PRB_API int prb_gemm_midm_trace(unsigned long long* host, int n) {
    return (int)cudaMemcpyFromSymbol(host, g_midm_trace, sizeof(unsigned long long) * n);
}
#else
#define MT_TRACE(slot)
#endif

namespace {
constexpr int THREADS = 256;
constexpr int WARPS = 8;
constexpr int MROWS = 64;           // token rows of a tile (rows beyond M are zero)
constexpr int KC = 2;               // 64-column slabs per stage
constexpr int STAGES = 4;
constexpr int PART_ROWS = 72;       // S * ceil(64 / S) for S up to 8, at most
constexpr uint32_t WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* failed) {
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && *failed) return false;
    }
    *failed = 1;
    return false;
}
// x is always 0 (a slab is 64 elements wide), so the 16-byte rule on x holds.
__device__ __forceinline__ void tma_load_slabs(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                               int row, int slab) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
        "l"(map), "r"(bar), "r"(0), "r"(row), "r"(slab)
        : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local_addr, int rank) {
    uint32_t raddr;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(local_addr), "r"(rank));
    return raddr;
}
__device__ __forceinline__ void st_cluster_f32x2(uint32_t addr, float x, float y) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

struct Args {
    void* c;
    const float* bias;
    const float* resid;
    int m, n, k;
    long ldc;
    int act;
    int splits;                     // CTAs of a cluster (grid z)
    int* status;
    // columns [q_width, q_width + kv_width) are keys, the next kv_width values of token row r: they
    // also (only_cache: only) go to the paged cache at slots[r] (-1: none); kv_width 0: off
    void* k_pages;
    void* v_pages;
    const int* slots;
    int q_width, kv_width, head_dim, page_size, num_pages, only_cache;
};

// Address of the 16-byte piece `piece` (0..7) of row `row` in a slab of [rows][64] bfloat16
// written by TMA with the 128-byte swizzle (slab base 1024-byte aligned).
__device__ __forceinline__ uint32_t swz(uint32_t slab, int row, int piece) {
    return slab + (uint32_t)row * 128 + (uint32_t)((piece ^ (row & 7)) << 4);
}

template <int NB, typename O>
__global__ void __launch_bounds__(THREADS)
gemm_midm_kernel(Args a, const __grid_constant__ CUtensorMap map_a,
                 const __grid_constant__ CUtensorMap map_w) {
    constexpr int NT = NB / 16;                       // 8-column MMA tiles per warp: 2 or 4
    constexpr uint32_t A_BYTES = KC * MROWS * 128, W_BYTES = KC * NB * 128;
    constexpr uint32_t STAGE_BYTES = A_BYTES + W_BYTES;
    constexpr int PP = NB + 8;                        // pitch of a row's part (floats): rows a warp
                                                      // writes together start 8 banks apart
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t ring = smem_u32(smem);
    // parts of this CTA's rows, [rank of the sender][row / S][PP]; 64 / S rows, rounded up
    float* part = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(part + PART_ROWS * PP);
    volatile uint32_t* missing = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES);   // [8]
    volatile int* failed = reinterpret_cast<volatile int*>(bars + 2 * STAGES + 4);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * NB;
    const int rank = blockIdx.z, S = a.splits;
    // this CTA's part of K, in slabs of 64
    const int slabs = a.k / 64;
    const int slab_lo = (int)((unsigned)(slabs * rank) / (unsigned)S);
    const int slab_hi = (int)((unsigned)(slabs * (rank + 1)) / (unsigned)S);
    const int items = (slab_hi - slab_lo + KC - 1) / KC;

    MT_TRACE(0);
    prb_grid_launch_dependents();
    cluster_arrive();                                 // (the peers exist: waited for before the first store to them)
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, WARPS);
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto issue_w = [&](int i) {
        const int st = i % STAGES;
        mbar_expect_tx(full0 + 8 * st, STAGE_BYTES);
        tma_load_slabs(ring + st * STAGE_BYTES + A_BYTES, &map_w, full0 + 8 * st, n0,
                       slab_lo + i * KC);
    };
    auto issue_a = [&](int i) {
        const int st = i % STAGES;
        tma_load_slabs(ring + st * STAGE_BYTES, &map_a, full0 + 8 * st, 0, slab_lo + i * KC);
    };
    // The weights do not depend on the previous kernel; the activations do.
    const int first = min(STAGES, items);
    if (threadIdx.x == 0)
        for (int i = 0; i < first; ++i) issue_w(i);
    // What takes quotients of run-time counts is worked out before the wait, not between the last
    // multiplication and the store: where this warp's rows go, and where a column lies in the cache.
    // (23 rows: 1,024 x 4,096 7.8 -> 7.05 us, 3,072 x 1,024 7.0 -> 6.3; 64 rows: 768 x 3,072 6.4 -> 5.9.)
    const int per = (int)((unsigned)(MROWS + S - 1) / (unsigned)S);      // rows of a CTA
    uint32_t part_dst[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const unsigned row = (warp & 3) * 16 + (lane >> 2) + 8 * half, to = row / (unsigned)S;
        part_dst[half] = cluster_addr(
            smem_u32(part + (size_t)(rank * per + (int)to) * PP + (warp >> 2) * (NB / 2) + (lane & 3) * 2),
            row - to * S);
    }
    const int col = threadIdx.x % NB, rsub = threadIdx.x / NB;
    const int gcol = n0 + col;
    const bool to_cache = a.kv_width != 0 && gcol >= a.q_width && gcol < a.n;
    O* column = nullptr;                              // this column in page 0, place 0
    long page_len = 0;                                // elements of a page
    if (to_cache) {
        unsigned cc = (unsigned)(gcol - a.q_width);
        column = reinterpret_cast<O*>(cc < (unsigned)a.kv_width ? a.k_pages : a.v_pages);
        if (cc >= (unsigned)a.kv_width) cc -= a.kv_width;
        const unsigned head = cc / (unsigned)a.head_dim, dim = cc - head * a.head_dim;
        page_len = (long)a.kv_width * a.page_size;
        column += (long)head * a.page_size * a.head_dim + dim;
    }
    prb_grid_wait();
    if (threadIdx.x == 0)
        for (int i = 0; i < first; ++i) issue_a(i);

    // warp -> 16 token rows (mt) and NB/2 columns (nh)
    const int mt = warp & 3, nh = warp >> 2;
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
    int issued = first;
    bool alive = true;
    for (int i = 0; i < items; ++i) {
        const int st = i % STAGES;
        if (alive && threadIdx.x == 0 && i >= 1 && i - 1 + STAGES < items) {
            const int pi = i - 1;
            if (mbar_wait(empty0 + 8 * (pi % STAGES), (uint32_t)(pi / STAGES) & 1u, failed)) {
                issue_w(pi + STAGES);
                issue_a(pi + STAGES);
                issued = pi + STAGES + 1;
            }
        }
        // (one answer for the warp: what follows are its instructions, not its lanes')
        if (alive) alive = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * st, (uint32_t)(i / STAGES) & 1u, failed));
        if (i == 0) MT_TRACE(1);
        if (i == items - 1) MT_TRACE(2);
        if (alive) {
            const uint32_t abase = ring + st * STAGE_BYTES, wbase = abase + A_BYTES;
            // slabs of this stage that lie inside this CTA's part of K (a copy may have run
            // past it into the next CTA's slabs; those are simply not multiplied)
            const int valid = min(KC, slab_hi - (slab_lo + i * KC));
            for (int sl = 0; sl < valid; ++sl) {
                const uint32_t aslab = abase + sl * (MROWS * 128), wslab = wbase + sl * (NB * 128);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {          // four k-steps of 16 in a slab
                    uint32_t af[4];
                    ldmatrix_x4(af, swz(aslab, mt * 16 + (lane & 15), kk * 2 + (lane >> 4)));
#pragma unroll
                    for (int np = 0; np < NT / 2; ++np) {     // two 8-column tiles per ldmatrix
                        uint32_t bf[4];
                        const int nrow = nh * (NB / 2) + np * 16 + ((lane >> 4) << 3) + (lane & 7);
                        ldmatrix_x4(bf, swz(wslab, nrow, kk * 2 + ((lane >> 3) & 1)));
                        mma16816(acc[2 * np], af, bf[0], bf[1]);
                        mma16816(acc[2 * np + 1], af, bf[2], bf[3]);
                    }
                }
            }
            if (i + STAGES < items) {
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * st);
            }
        }
    }
    MT_TRACE(3);
    // ---- the rows of this CTA's partial tile to the CTAs that finish them
    __syncwarp();
    cluster_wait();
    {
        const int g = lane >> 2;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int row = mt * 16 + g + 8 * half;
            if (row < a.m) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                    st_cluster_f32x2(part_dst[half] + nt * 32, acc[nt][2 * half], acc[nt][2 * half + 1]);
            }
        }
    }
    // bias and residual of the outputs this thread finishes, asked for before the barrier
    constexpr int RPP = THREADS / NB;                     // rows per pass
    constexpr int PASSES = MROWS / RPP;                   // (S = 1; a split has 1 / S of them)
    constexpr int AHEAD = PASSES < 4 ? PASSES : 4;
    const float bias = (a.bias && gcol < a.n) ? a.bias[gcol] : 0.0f;
    float res[AHEAD];
    O* place[AHEAD];                                      // in the cache, or null
    auto cache_place = [&](int row) -> O* {
        const int at = to_cache && row < a.m ? a.slots[row] : -1;
        if (at < 0) return nullptr;
        const int page = (int)((unsigned)at / (unsigned)a.page_size);
        if (page >= a.num_pages) {
            prb_set_status(a.status, PRB_S_SLOT_RANGE, row, at, a.num_pages);
            return nullptr;
        }
        return column + page * page_len + (long)(at - page * a.page_size) * a.head_dim;
    };
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
        const int row = rank + (rsub + i * RPP) * S;
        place[i] = rsub + i * RPP < per ? cache_place(row) : nullptr;
        res[i] = (a.resid && gcol < a.n && row < a.m) ? a.resid[(size_t)row * a.ldc + gcol] : 0.0f;
    }
    __syncthreads();
    const bool bad_here = *failed != 0;
    if (bad_here && threadIdx.x == 0) {
        prb_set_status(a.status, PRB_S_WAIT_TIMEOUT, blockIdx.x, rank, 0);
        for (int i = max(0, issued - STAGES); i < issued; ++i) {
            const uint32_t bar = full0 + 8 * (i % STAGES);
            const uint32_t parity = (uint32_t)(i / STAGES) & 1u;
            for (uint32_t w = 0; w < WAIT_LIMIT; ++w)
                if (mbar_try_wait(bar, parity)) break;
        }
    }
    if (threadIdx.x < S)                                  // peers see whether this part is missing
        st_cluster_u32(cluster_addr(smem_u32((const void*)(missing + rank)), threadIdx.x), bad_here ? 1u : 0u);
    __syncwarp();
    MT_TRACE(4);
    cluster_arrive();
    cluster_wait();                                       // every part is in place
    MT_TRACE(5);
    // ---- rows rank, rank + S, ...: sum over the cluster in rank order, epilogue, store
    bool any_bad = false;
    for (int r = 0; r < S; ++r) any_bad |= missing[r] != 0;
    if (!any_bad && gcol < a.n) {
        O* out = reinterpret_cast<O*>(a.c);
#pragma unroll
        for (int i = 0; i < PASSES; ++i) {
            const int local = rsub + i * RPP, row = rank + local * S;
            if (local >= per || row >= a.m) break;
            const float* src = part + (size_t)local * PP + col;
            float pv[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) pv[r] = r < S ? src[(size_t)r * per * PP] : 0.0f;
            float v = 0.0f;
#pragma unroll
            for (int r = 0; r < 8; ++r) v += pv[r];
            v = prb_activate(v + bias, a.act);
            if (a.resid) v += i < AHEAD ? res[i < AHEAD ? i : 0] : a.resid[(size_t)row * a.ldc + gcol];
            if (!to_cache || !a.only_cache) out[(size_t)row * a.ldc + gcol] = prb_from_float<O>(v);
            if (to_cache) {
                O* at = i < AHEAD ? place[i < AHEAD ? i : 0] : cache_place(row);
                if (at != nullptr) *at = prb_from_float<O>(v);
            }
        }
    }
    MT_TRACE(6);
    MT_TRACE(7);
}

template <int NB> constexpr size_t midm_smem() {
    return 1024 + (size_t)STAGES * KC * (MROWS + NB) * 128 + (size_t)PART_ROWS * (NB + 8) * 4 +
           2 * STAGES * 8 + 32 + 16;
}

template <int NB, typename O> int configure_midm() {
    static int rc = [] {
        cudaFuncSetAttribute(gemm_midm_kernel<NB, O>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
        return (int)cudaFuncSetAttribute(gemm_midm_kernel<NB, O>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)midm_smem<NB>());
    }();
    return rc;
}

template <int NB> void midm_launch(const Args& a, cudaStream_t stream, cudaLaunchConfig_t* cfg,
                                   cudaLaunchAttribute* attr) {
    cfg->gridDim = dim3((a.n + NB - 1) / NB, 1, a.splits);
    cfg->blockDim = dim3(THREADS);
    cfg->dynamicSmemBytes = midm_smem<NB>();
    cfg->stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)a.splits;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = prb_pdl_enabled() ? 1 : 0;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

template <int NB, typename O>
int launch_midm(const Args& a, const CUtensorMap& ma, const CUtensorMap& mw, cudaStream_t stream) {
    const int rc = configure_midm<NB, O>();
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    midm_launch<NB>(a, stream, &cfg, attr);
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_midm_kernel<NB, O>, a, ma, mw);
    return e == cudaSuccess ? 0 : (int)e;
}

// How many clusters of `splits` CTAs run at a time (asked once per device).
template <int NB> int active_clusters(int splits) {
    static int known[64][9] = {};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || configure_midm<NB, float>() != 0) return 1;
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev][splits] == 0) {
        Args a{};
        a.n = NB;
        a.splits = splits;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        midm_launch<NB>(a, nullptr, &cfg, attr);
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_midm_kernel<NB, float>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        known[dev][splits] = n > 0 ? n : 1;
    }
    return known[dev][splits];
}
}  // namespace

// 1 when the kernel takes these sizes (else the caller uses another product kernel).
PRB_API int prb_gemm_midm_supports(int m, int n, int k) {
    return m >= 1 && m <= MROWS && n >= 1 && k >= 64 && k % 64 == 0 ? 1 : 0;
}

// a: bfloat16 [M,K]; w: bfloat16 [N,K]; c: bfloat16 or float32 [M,N] (resid float32, may
// alias c).  M <= 64, K a multiple of 64, pitches multiples of 8 elements.
// k_pages / v_pages / slots: the cache of the output's element type that key and value columns of a
// fused QKV product also (only_cache: only) go to; null: none.
PRB_API int prb_gemm_midm(void* c, const void* a, const void* w, const float* bias,
                          const float* resid, int m, int n, int k, long lda, long ldw, long ldc,
                          int act, int out_dtype, void* k_pages, void* v_pages, const int* slots,
                          int q_width, int kv_width, int head_dim, int page_size, int num_pages,
                          int only_cache, int* status, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (!prb_gemm_midm_supports(m, n, k)) return PRB_E_SIZE;
    if (lda % 8 != 0 || ldw % 8 != 0 || ((uintptr_t)a) % 16 != 0 || ((uintptr_t)w) % 16 != 0)
        return PRB_E_ALIGN;
    if (out_dtype != PRB_F32 && out_dtype != PRB_BF16) return PRB_E_DTYPE;
    if (k_pages != nullptr &&
        (v_pages == nullptr || slots == nullptr || resid != nullptr || head_dim <= 0 || kv_width <= 0 ||
         kv_width % head_dim != 0 || page_size <= 0 || q_width < 0 || q_width + 2 * kv_width != n))
        return PRB_E_ARG;
    // Tile width and cluster size from N and K (and the device) only.  All CTAs should run at once (one per
    // SM with 64-column tiles, two with 32-column tiles); within that, the split that gives
    // an SM the fewest bytes to take in (its CTAs' slices of A and W) wins.
    const int slabs = k / 64;
    const int sms = prb_sm_count();
    int nb = 32, splits = 1;
    long best = -1;
    for (int cand = 64; cand >= 32; cand /= 2) {
        const int tiles = (n + cand - 1) / cand;
        const int slots = sms * (cand == 64 ? 1 : 2);
        int s = slots / tiles;
        if (s > 8) s = 8;
        if (s > slabs / 2) s = slabs / 2;
        if (s < 1) s = 1;
        // (clusters are placed inside groups of SMs whose sizes differ: 16 clusters of eight do not
        // all run at once on 148 SMs, and a second round costs as much as the first)
        while (s > 1 && tiles > (cand == 64 ? active_clusters<64>(s) : active_clusters<32>(s))) --s;
        const long per_cta = (long)(MROWS + cand) * 2 * ((long)k / s);
        const long ctas = (long)tiles * s;
        const long per_sm = per_cta * ((ctas + sms - 1) / sms);
        if (best < 0 || per_sm < best) { best = per_sm; nb = cand; splits = s; }
    }
    CUtensorMap ma, mw;
    int rc = tmap::slab_map(a, m, k, lda, MROWS, KC, &ma);
    if (rc) return rc;
    if ((rc = tmap::slab_map(w, n, k, ldw, nb, KC, &mw)) != 0) return rc;
    Args args{c, bias, resid, m, n, k, ldc, act, splits, status, k_pages, v_pages, slots, q_width,
              k_pages != nullptr ? kv_width : 0, head_dim, page_size, num_pages, only_cache};
    if (nb == 64)
        return out_dtype == PRB_F32 ? launch_midm<64, float>(args, ma, mw, stream)
                                    : launch_midm<64, __nv_bfloat16>(args, ma, mw, stream);
    return out_dtype == PRB_F32 ? launch_midm<32, float>(args, ma, mw, stream)
                                : launch_midm<32, __nv_bfloat16>(args, ma, mw, stream);
}
