// Causal attention over the paged cache in true 32-bit arithmetic: the kernels of the float32
// path for head sizes that are multiples of 4 up to 128 (`attention_generic.cu` takes the rest).
//
// ONE order of operations for every query, whatever else is in the batch, however a prompt was
// cut and whichever kernel runs.  Keys are cut by their absolute positions into chunks of 64 and
// groups of four chunks.  A chunk by itself: scores (one chain over the head's even dimensions, one
// over the odd ones, added: what fma.rn.f32x2 takes as a pair), its maximum m, weights exp(s - m), their sum l (keys i, i + 16, i + 32, i + 48 first, then a
// tree over i), rows o = sum w v in ascending order.  Chunks are merged into their group in
// ascending order, groups likewise:  m' = max(m, mc), l' = l e^(m-m') + lc e^(mc-m'), o likewise;
// a chunk of which a query sees nothing is passed over.  Result: o / l.
//
// One CTA per (queries, head, group), the CTAs of a (queries, head) as a cluster along z (up to
// eight; further groups in turn), merged through distributed shared memory:
//   attention_f32_tile_kernel    32 consecutive queries of a request; a chunk's keys and values in
//                                shared memory (cp.async: the next keys come while the values are
//                                multiplied, the next values during the next scores); a thread has
//                                4 queries x 4 keys, then 4 queries x 4 dimensions, since what
//                                bounds it is shared-memory reads per FMA
//   attention_f32_single_kernel  one query; four teams of 64 threads take a chunk each, straight
//                                from memory (a thread a key, then a thread a dimension): what
//                                counts is that a group's 128 KB are requested at once
// With one thread block a (token, head) that walks all keys (attention_generic.cu) 8 requests leave
// most SMs idle, and a prompt reads every key again for each query.  8 requests of about 100 tokens,
// 12 heads: 8.5 us a launch (a chain of look-ups: list, place of the token, page, keys, values), 44
// that way; prompts of 650 tokens together 94 us, 376 that way.  Contexts or prompts of some 20
// tokens are where that way is the faster one (12 heads: 64 requests of 10 tokens 7.6 us, here 19.0; a
// prompt of 17 8.3 and 18.3): a group's CTA takes its rounds whatever it holds, and the order of sums
// has to be the same for all of a model's steps.
#include "common.cuh"

namespace {
constexpr int THREADS = 256;
constexpr int CHUNK = 64, GROUP = 256;
constexpr int TQ = 32;              // queries of a tile CTA
constexpr int TILE_THREADS = 128;
constexpr int TQP = TQ + 4;
constexpr int MAX_CLUSTER = 8;

struct Args {
    float* out;
    const float* q;
    const float* k_pages;
    const float* v_pages;
    const int* block_table;
    const int* seq_of_token;
    const int* positions;
    const int* tile_row0;           // tiles: first token and number of tokens
    const int* tile_rows;
    const int* list;                // singles: token indices
    const int* count;               // tiles or singles on the device
    int n_list;                     // most of them
    long out_stride, q_stride;
    int n_heads, kv_heads, head_dim, page_size, max_pages, num_pages, max_context, window;
    float scale;
    int slots;                      // groups a CTA may hold
    int* status;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t addr, uint32_t rank) {
    uint32_t r;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
    return v;
}

// What a query may see: keys lo..pos; pos = -1 for a row that is not there or out of range.
__device__ __forceinline__ int visible(const Args& p, int t, int* lo) {
    const int pos = p.positions[t];
    *lo = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
    if (pos < 0 || pos - *lo + 1 > p.max_context || pos >= p.max_pages * p.page_size) {
        prb_set_status(p.status, PRB_S_POSITION_RANGE, t, pos, p.max_context);
        return -1;
    }
    return pos;
}
// Row of key position j in the pools (in rows of head_dim), -1 (and the status word) if its page
// is not there.
__device__ __forceinline__ long key_row(const Args& p, const int* table, int hk, int j, int t) {
    const int page = table[j / p.page_size];
    if (page < 0 || page >= p.num_pages) {
        prb_set_status(p.status, PRB_S_PAGE_RANGE, t, j, page);
        return -1;
    }
    return ((long)page * p.kv_heads + hk) * p.page_size + j % p.page_size;
}

// acc += a * b, both halves (each rounded once, as fmaf)
__device__ __forceinline__ void fma2(float& accx, float& accy, float ax, float ay, float bx, float by) {
    asm("{\n\t.reg .b64 a, b, c;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(accx), "+f"(accy) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}

// (m, l, o) joined by a later part (mc, lc, oc).  A part without a visible key (no weight) changes
// nothing; a part of keys whose scores are no numbers has no maximum either, but no sum: it makes
// the sum none (and the result zero, as one walk over all keys does).  A part whose weight vanishes
// beside the other contributes nothing, whatever its values are.
template <int N>
__device__ __forceinline__ void join(float& m, float& l, float (&o)[N], float mc, float lc, const float (&oc)[N]) {
    if (mc == -INFINITY && lc == 0.0f) return;
    const float mn = fmaxf(m, mc);
    const float sa = expf(m - mn), sb = expf(mc - mn);
    l = l * sa + lc * sb;
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = (sa == 0.0f ? 0.0f : o[i] * sa) + (sb == 0.0f ? 0.0f : oc[i] * sb);
    m = mn;
}

// The groups of a cluster's queries joined in order and written: `parts` [slot][pitch][hd + 2] of
// every CTA holds (m, l, o...) of the first `queries` of `pitch` queries.  CTA `rank` finishes
// queries rank, rank + size, ...
__device__ __forceinline__ void finish(const Args& p, const float* parts, int pitch, int queries,
                                       int n_groups, int first_row, int rank, int size, int h) {
    const int len = p.head_dim + 2;
    const int mine = queries > rank ? (queries - rank + size - 1) / size : 0;
    for (int i = threadIdx.x; i < mine * p.head_dim; i += blockDim.x) {
        const int qi = rank + (i / p.head_dim) * size, d = i % p.head_dim;
        float m = -INFINITY, l = 0.0f, o[1] = {0.0f};
        for (int g = 0; g < n_groups; ++g) {
            const uint32_t at = smem_u32(parts + ((g / size) * pitch + qi) * len);
            const float oc[1] = {ld_cluster(at + 4u * (2 + d), g % size)};
            join(m, l, o, ld_cluster(at, g % size), ld_cluster(at + 4u, g % size), oc);
        }
        p.out[(size_t)(first_row + qi) * p.out_stride + (size_t)h * p.head_dim + d] =
            l > 0.0f ? o[0] / l : 0.0f;
    }
    __syncwarp();
}

template <int ND>                   // float4s of a row a thread accumulates (head size up to 64 ND)
__global__ void __launch_bounds__(TILE_THREADS)
attention_f32_tile_kernel(Args p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int s_pos[TQ], s_lo[TQ], s_ok[2][CHUNK];
    prb_grid_wait();
    prb_grid_launch_dependents();
    const int tile = blockIdx.x >> 2, sub = blockIdx.x & 3, h = blockIdx.y;
    if (tile >= min(p.n_list, *p.count)) return;              // (the whole cluster leaves)
    const int rows = min(TQ, p.tile_rows[tile] - sub * TQ);
    if (rows <= 0) return;
    const int row0 = p.tile_row0[tile] + sub * TQ;
    const int rank = blockIdx.z, size = gridDim.z;
    const int hd = p.head_dim, ld = hd + 4;
    float* sq = smem;                                         // [TQ][ld]
    float* sk = sq + TQ * ld;                                 // [CHUNK][ld]
    float* sv = sk + CHUNK * ld;                              // [CHUNK][ld]
    float* sw = sv + CHUNK * ld;                              // [CHUNK][TQP]
    float* parts = sw + CHUNK * TQP;                          // [slots][TQ][hd + 2]
    const int tid = threadIdx.x, q0 = (tid >> 4) * 4, x = tid & 15;
    const int b = p.seq_of_token[row0];
    const int hk = h / (p.n_heads / p.kv_heads);
    const int* table = p.block_table + (size_t)b * p.max_pages;
    if (tid < TQ) {
        int lo = 0;
        s_pos[tid] = tid < rows && b >= 0 ? visible(p, row0 + tid, &lo) : -1;
        s_lo[tid] = lo;
    }
    for (int i = tid; i < TQ * hd; i += TILE_THREADS) {
        const int r = i / hd, d = i % hd;
        sq[r * ld + d] = r < rows ? p.q[(size_t)(row0 + r) * p.q_stride + (size_t)h * hd + d] : 0.0f;
    }
    __syncthreads();
    int last = -1, first = 0x7fffffff;
    for (int i = 0; i < TQ; ++i)
        if (s_pos[i] >= 0) { last = max(last, s_pos[i]); first = min(first, s_lo[i]); }
    const int g0 = last < 0 ? 0 : first / GROUP;
    int n_groups = last < 0 ? 0 : last / GROUP - g0 + 1;
    if (n_groups > p.slots * size) {                          // not consecutive tokens: no room for their keys
        if (tid == 0 && rank == 0) prb_set_status(p.status, PRB_S_POSITION_RANGE, row0, last, p.max_context);
        n_groups = 0;                                         // (the same for the whole cluster; zeros are written)
    }
    const int c_first = first / CHUNK, c_last = last / CHUNK;  // chunks anyone sees

    // this CTA's chunks in order: step i is chunk i % 4 of its group i / 4
    const int my_groups = n_groups > rank ? (n_groups - rank + size - 1) / size : 0;
    const int steps = my_groups * 4;
    auto chunk_of = [&](int i) { return (g0 + rank + (i >> 2) * size) * 4 + (i & 3); };
    auto load = [&](int i, float* dst, const float* pages, bool note) {
        if (i < steps) {
            const int c = chunk_of(i);
            if (c >= c_first && c <= c_last) {
                const int per = hd / 4;
                for (int e = tid; e < CHUNK * per; e += TILE_THREADS) {
                    const int r = e / per, d = (e % per) * 4, j = c * CHUNK + r;
                    // (rows after the last position hold what a page's earlier owner left)
                    const long row = j <= last && j >= first ? key_row(p, table, hk, j, row0) : -1;
                    cp16(smem_u32(dst + r * ld + d), pages + (row < 0 ? 0 : (size_t)row * hd + d), row < 0 ? 0 : 16);
                    if (note && d == 0) s_ok[i & 1][r] = row >= 0;
                }
            }
        }
        cp_commit();
    };
    load(0, sk, p.k_pages, true);
    load(0, sv, p.v_pages, false);
    float gm[4], gl[4], go[4][4 * ND];
    for (int i = 0; i < steps; ++i) {
        if ((i & 3) == 0) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                gm[r] = -INFINITY;
                gl[r] = 0.0f;
#pragma unroll
                for (int e = 0; e < 4 * ND; ++e) go[r][e] = 0.0f;
            }
        }
        const int c = chunk_of(i);
        const bool live = c >= c_first && c <= c_last;        // (the same for the whole CTA)
        cp_wait<1>();                                         // this step's keys are here
        __syncthreads();
        float mc[4], lc[4];
        if (live) {
            float s[4][4];                                    // [query][key x + 16 j]
            {
                float2 acc[4][4];
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[r][j] = make_float2(0.0f, 0.0f);
#pragma unroll 2
                for (int d = 0; d < hd; d += 4) {
                    float4 kv[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        kv[j] = *reinterpret_cast<const float4*>(sk + (x + 16 * j) * ld + d);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float4 qv = *reinterpret_cast<const float4*>(sq + (q0 + r) * ld + d);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            fma2(acc[r][j].x, acc[r][j].y, qv.x, qv.y, kv[j].x, kv[j].y);
                            fma2(acc[r][j].x, acc[r][j].y, qv.z, qv.w, kv[j].z, kv[j].w);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[r][j] = acc[r][j].x + acc[r][j].y;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int pos = s_pos[q0 + r], lo = s_lo[q0 + r];
                mc[r] = -INFINITY;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = c * CHUNK + x + 16 * j;
                    s[r][j] = key <= pos && key >= lo && s_ok[i & 1][x + 16 * j] ? s[r][j] * p.scale : -INFINITY;
                    mc[r] = fmaxf(mc[r], s[r][j]);
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) mc[r] = fmaxf(mc[r], __shfl_xor_sync(0xffffffffu, mc[r], o));
                lc[r] = 0.0f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[r][j] = s[r][j] == -INFINITY ? 0.0f : expf(s[r][j] - mc[r]);
                    lc[r] += s[r][j];
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) lc[r] += __shfl_xor_sync(0xffffffffu, lc[r], o);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(sw + (x + 16 * j) * TQP + q0) =
                    make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
        }
        __syncthreads();                                      // the keys' buffer is free
        load(i + 1, sk, p.k_pages, true);
        cp_wait<1>();                                         // this step's values are here
        __syncthreads();
        if (live) {
            float oc[4][4 * ND];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int e = 0; e < 4 * ND; ++e) oc[r][e] = 0.0f;
#pragma unroll 4
            for (int j = 0; j < CHUNK; ++j) {
                const float4 w4 = *reinterpret_cast<const float4*>(sw + j * TQP + q0);
                const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int e = 0; e < ND; ++e) {
                    const int d = (x + 16 * e) * 4;
                    if (d < hd) {
                        const float4 v = *reinterpret_cast<const float4*>(sv + j * ld + d);
#pragma unroll
                        for (int r = 0; r < 4; ++r)
                            if (w[r] != 0.0f) {               // (a value nobody sees may be infinite)
                                fma2(oc[r][4 * e], oc[r][4 * e + 1], w[r], w[r], v.x, v.y);
                                fma2(oc[r][4 * e + 2], oc[r][4 * e + 3], w[r], w[r], v.z, v.w);
                            }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) join(gm[r], gl[r], go[r], mc[r], lc[r], oc[r]);
        }
        if ((i & 3) == 3) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float* dst = parts + ((i >> 2) * TQ + q0 + r) * (hd + 2);
                if (x == 0) { dst[0] = gm[r]; dst[1] = gl[r]; }
#pragma unroll
                for (int e = 0; e < ND; ++e) {
                    const int d = (x + 16 * e) * 4;
                    if (d < hd)
                        for (int z = 0; z < 4; ++z) dst[2 + d + z] = go[r][4 * e + z];
                }
            }
        }
        __syncthreads();                                      // the values' buffer is free
        load(i + 1, sv, p.v_pages, false);
    }
    cp_wait<0>();
    __syncthreads();
    cluster_sync_all();
    finish(p, parts, TQ, rows, n_groups, row0, rank, size, h);
    cluster_sync_all();
}

template <int ND>                   // dimensions a thread accumulates (head size up to 64 ND)
__global__ void __launch_bounds__(THREADS, 2)
attention_f32_single_kernel(Args p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float s_w[4][CHUNK], s_m[4], s_l[4];
    __shared__ long s_row[4][CHUNK];
    prb_grid_wait();
    prb_grid_launch_dependents();
    const int h = blockIdx.y;
    if ((int)blockIdx.x >= min(p.n_list, *p.count)) return;   // (the whole cluster leaves)
    const int t = p.list[blockIdx.x];
    const int rank = blockIdx.z, size = gridDim.z;
    const int hd = p.head_dim;
    float* sq = smem;                                         // [128]
    float* so = smem + 128;                                   // [4][hd]
    float* parts = so + 4 * hd;                               // [slots][1][hd + 2]
    const int tid = threadIdx.x, team = tid >> 6, x = tid & 63;
    const int b = p.seq_of_token[t];
    const int hk = h / (p.n_heads / p.kv_heads);
    const int* table = p.block_table + (size_t)b * p.max_pages;
    int lo = 0;
    const int pos = b >= 0 ? visible(p, t, &lo) : -1;
    for (int d = tid; d < hd; d += THREADS) sq[d] = p.q[(size_t)t * p.q_stride + (size_t)h * hd + d];
    __syncthreads();
    const int g0 = lo / GROUP;
    const int n_groups = pos < 0 ? 0 : pos / GROUP - g0 + 1;
    for (int g = rank, slot = 0; g < n_groups; g += size, ++slot) {
        const int key = (g0 + g) * GROUP + team * CHUNK + x;
        const long row = key <= pos && key >= lo ? key_row(p, table, hk, key, t) : -1;
        s_row[team][x] = row;
        // the first values are asked for with the keys (the rows' addresses are all that they need)
        __syncthreads();
        // (coherent loads: the launch may be placed while the kernel ahead still writes the step's rows)
        constexpr int VB = 32 / ND;                           // value rows in flight a thread
        float v[VB][ND];
        auto load_values = [&](int j0) {
#pragma unroll
            for (int j = 0; j < VB; ++j) {
                const long vrow = s_row[team][j0 + j];
#pragma unroll
                for (int e = 0; e < ND; ++e) {
                    const int d = x + 64 * e;
                    v[j][e] = vrow >= 0 && d < hd ? __ldcg(p.v_pages + (size_t)vrow * hd + d) : 0.0f;
                }
            }
        };
        float s = -INFINITY;
        {
            const float4* kr = reinterpret_cast<const float4*>(p.k_pages + (size_t)(row < 0 ? 0 : row) * hd);
            float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int d0 = 0; d0 < 16 * ND; d0 += 16) {
                float4 kv[16];
#pragma unroll
                for (int d = 0; d < 16; ++d)
                    kv[d] = row >= 0 && d0 + d < hd / 4 ? __ldcg(kr + d0 + d) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (d0 == 0) load_values(0);
#pragma unroll
                for (int d = 0; d < 16; ++d)
                    if (d0 + d < hd / 4) {
                        const float4 qv = *reinterpret_cast<const float4*>(sq + 4 * (d0 + d));
                        fma2(acc.x, acc.y, qv.x, qv.y, kv[d].x, kv[d].y);
                        fma2(acc.x, acc.y, qv.z, qv.w, kv[d].z, kv[d].w);
                    }
            }
            if (row >= 0) s = (acc.x + acc.y) * p.scale;
        }
        s_w[team][x] = s;
        __syncthreads();
        float mc = -INFINITY;                                 // (every 16 threads the whole chunk)
#pragma unroll
        for (int j = 0; j < 4; ++j) mc = fmaxf(mc, s_w[team][(x & 15) + 16 * j]);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mc = fmaxf(mc, __shfl_xor_sync(0xffffffffu, mc, o));
        __syncthreads();
        s_w[team][x] = s == -INFINITY ? 0.0f : expf(s - mc);
        __syncthreads();
        float lc = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) lc += s_w[team][(x & 15) + 16 * j];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) lc += __shfl_xor_sync(0xffffffffu, lc, o);
        if (x == 0) { s_m[team] = mc; s_l[team] = lc; }
        float oc[ND];
#pragma unroll
        for (int e = 0; e < ND; ++e) oc[e] = 0.0f;
#pragma unroll
        for (int j0 = 0; j0 < CHUNK; j0 += VB) {
            if (j0 > 0) load_values(j0);
#pragma unroll
            for (int j = 0; j < VB; ++j) {
                const float w = s_w[team][j0 + j];
                if (w != 0.0f) {
#pragma unroll
                    for (int e = 0; e < ND; ++e) oc[e] = fmaf(w, v[j][e], oc[e]);
                }
            }
        }
#pragma unroll
        for (int e = 0; e < ND; ++e)
            if (x + 64 * e < hd) so[team * hd + x + 64 * e] = oc[e];
        __syncthreads();
        for (int d = tid; d < hd; d += THREADS) {
            float m = -INFINITY, l = 0.0f, o[1] = {0.0f};
            for (int c = 0; c < 4; ++c) {
                const float part[1] = {so[c * hd + d]};
                join(m, l, o, s_m[c], s_l[c], part);
            }
            float* dst = parts + slot * (hd + 2);
            if (d == 0) { dst[0] = m; dst[1] = l; }
            dst[2 + d] = o[0];
        }
        __syncthreads();
    }
    cluster_sync_all();
    finish(p, parts, 1, 1, n_groups, t, rank, size, h);
    cluster_sync_all();
}

constexpr size_t MOST_SMEM = 220 * 1024;

template <auto Kernel>
int launch(const Args& a, dim3 grid, int threads, size_t smem, cudaStream_t stream) {
    cudaError_t e = prb_allow_shared<Kernel>((int)MOST_SMEM);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = grid.z;
    // the few CTAs of a small decoding step start while the kernel before them ends
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed =
        prb_pdl_enabled() && (long)grid.x * grid.y * grid.z <= 2L * prb_sm_count() ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, Kernel, a);
    return e == cudaSuccess ? 0 : (int)e;
}

// Shared memory of the two kernels with room for `slots` groups a CTA.
size_t tile_smem(int hd, int slots) {
    return sizeof(float) * ((size_t)(TQ + 2 * CHUNK) * (hd + 4) + CHUNK * TQP + (size_t)slots * TQ * (hd + 2));
}
size_t single_smem(int hd, int slots) { return sizeof(float) * (128 + 4ull * hd + (size_t)slots * (hd + 2)); }

// CTAs of a cluster and the groups each of them may meet.  No query sees more than `span` keys and
// `queries` consecutive ones no more than queries - 1 further; without a window they begin at a
// group's first key.  A step's contexts seldom reach behind max_context, so no more CTAs than it has
// groups: the further ones a window may touch are met in turn (128 keys of window, 64 requests x 12
// heads of 10 keys: 48.7 us as clusters of three, most of whose CTAs see nothing, 18.9 so).
struct Plan {
    int z, slots;
};
Plan plan(int max_context, int window, int queries) {
    const int span = window > 0 && window < max_context ? window : max_context;
    const int most = window > 0 ? (span + queries - 1 + GROUP - 2) / GROUP + 1 : (span + GROUP - 1) / GROUP;
    const int whole = (max_context + GROUP - 1) / GROUP;
    const int z = most < whole ? most : whole;
    const int ctas = z < MAX_CLUSTER ? z : MAX_CLUSTER;
    return {ctas, (most + ctas - 1) / ctas};
}
}  // namespace

// 1 when the kernels take these sizes (else the caller uses prb_attention_generic).
PRB_API int prb_attention_f32_supports(int head_dim, int max_context, int window) {
    if (head_dim < 4 || head_dim % 4 != 0 || head_dim > 128 || max_context <= 0) return 0;
    return tile_smem(head_dim, plan(max_context, window, TQ).slots) <= MOST_SMEM ? 1 : 0;
}

// Attention of the step's tokens: those in tiles (`tiles` true: n_list tiles of up to 128 tokens,
// tile_row0 / tile_rows), or single ones (list).  `count`: how many of them there are, on the
// device.  Page pools contiguous and 16-byte aligned.
PRB_API int prb_attention_f32(float* out, long out_stride, const float* q, long q_stride,
                              const float* k_pages, const float* v_pages, const int* block_table,
                              const int* seq_of_token, const int* positions, const int* tile_row0,
                              const int* tile_rows, const int* list, const int* count, int n_list,
                              int n_heads, int kv_heads, int head_dim, int page_size, int max_pages,
                              int num_pages, int max_context, float scale, int window, int* status,
                              cudaStream_t stream) {
    if (n_list <= 0) return 0;
    if (n_heads <= 0 || kv_heads <= 0 || n_heads % kv_heads != 0 || page_size <= 0 || max_pages <= 0 ||
        n_heads > 65535 || !prb_attention_f32_supports(head_dim, max_context, window))
        return PRB_E_SIZE;
    if (((uintptr_t)k_pages) % 16 != 0 || ((uintptr_t)v_pages) % 16 != 0) return PRB_E_ALIGN;
    if (count == nullptr || (list == nullptr) == (tile_row0 == nullptr)) return PRB_E_ARG;
    const Plan pl = plan(max_context, window, tile_row0 != nullptr ? TQ : 1);
    const int z = pl.z;
    Args a{out, q, k_pages, v_pages, block_table, seq_of_token, positions, tile_row0, tile_rows, list,
           count, n_list, out_stride, q_stride, n_heads, kv_heads, head_dim, page_size, max_pages,
           num_pages, max_context, window, scale, pl.slots, status};
    if (tile_row0 != nullptr) {
        const size_t smem = tile_smem(head_dim, a.slots);
        dim3 grid(n_list * (128 / TQ), n_heads, z);
        const int rc = head_dim <= 64 ? launch<attention_f32_tile_kernel<1>>(a, grid, TILE_THREADS, smem, stream)
                                      : launch<attention_f32_tile_kernel<2>>(a, grid, TILE_THREADS, smem, stream);
        if (rc) return rc;
    } else {
        const size_t smem = single_smem(head_dim, a.slots);
        dim3 grid(n_list, n_heads, z);
        const int rc = head_dim <= 64 ? launch<attention_f32_single_kernel<1>>(a, grid, THREADS, smem, stream)
                                      : launch<attention_f32_single_kernel<2>>(a, grid, THREADS, smem, stream);
        if (rc) return rc;
    }
    return 0;
}
