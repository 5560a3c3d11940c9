// stats.cuh -- partition statistics (app/part_eval.cpp:73-110,
// src/part_stat.hpp:77-239 of the reference) in one pass over the edges.
//
// Cut weight per part, part sizes and the number of (vertex, other part)
// pairs that share an edge come from the same read of each row, so the bound
// is one read of the CSR plus the gathers of the neighbours' parts.  Counting
// distinct parts needs no connectivity table: a short row compares the parts
// its lanes hold in registers, a longer one sets bits in a k-bit map in
// shared memory.  A 3.1 M-vertex 3D grid in 128 slabs (187 MB): 2266 us with
// one global atomic per boundary vertex and the tables built for the count,
// 280 us now, of which the row kernel takes about 200 (cold, under ncu; DRAM at 12%
// of peak, warps waiting for the gathers); the rest is the degree bins and the call.
#pragma once
#include "coarsen.cuh"

namespace jetb {

// h[p] += v for the lanes with `on` (every lane of the warp calls it).  In
// vertex orders that keep a part together the whole warp adds to one entry:
// that case takes one atomic instead of 32 serialised ones.
template <class W>
__device__ __forceinline__ void warp_hist_add(W* h, part_t p, W v, bool on) {
    const unsigned act = __ballot_sync(0xffffffffu, on);
    if (act == 0) return;
    const part_t p0 = __shfl_sync(0xffffffffu, p, __ffs(act) - 1);
    if (__all_sync(0xffffffffu, !on || p == p0)) {
        const W s = group_sum<W>(on ? v : (W)0, 32);
        if ((threadIdx.x & 31) == 0) atomic_add(&h[p0], s);
    } else if (on) {
        atomic_add(&h[p], v);
    }
}

template <class W>
struct PStatOut {
    W* per;              // k: cut weight counted at each part's vertices
    W* sizes;            // k
    long long* comm;
    int* bad;            // set when a part id is out of range
};

// Rows of at most 32 edges, G lanes each; every vertex's weight is counted
// here.  G follows the level's average degree, so most rows take one or two
// rounds of loads, all issued before the first use.
template <int G, class O, class E, class W>
__global__ void __launch_bounds__(BLOCK) k_pstat_rows(GView<O, E, W> g, const part_t* part, part_t k, PStatOut<W> out, int hist) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    W* h_per = hist ? (W*)smem_raw : out.per;
    W* h_sz = hist ? (W*)smem_raw + k : out.sizes;
    if (hist) {
        for (int p = threadIdx.x; p < 2 * k; p += blockDim.x) ((W*)smem_raw)[p] = 0;
        __syncthreads();
    }
    constexpr int R = THREAD_DEG / G;
    long long comm = 0;
#define PSTAT_BODY(x, in, lane)                                                             \
    {                                                                                       \
        part_t own = in ? part[x] : NULL_PART;                                              \
        const E s = in ? g.row[x] : (E)0;                                                   \
        E d = in ? g.row[x + 1] - s : (E)0;                                                 \
        const W vw = in && lane == 0 ? g.vw[x] : (W)0;                                      \
        bool ok = in && own >= 0 && own < k;                                                \
        if (in && !ok) atomicOr(out.bad, 8);                                                \
        if (!ok || d > THREAD_DEG) d = 0;                                                   \
        const int rounds = (int)__reduce_max_sync(0xffffffffu, (unsigned)((d + G - 1) / G)); \
        W acc = 0;                                                                          \
        part_t q[R];                                                                        \
        _Pragma("unroll") for (int r = 0; r < R; r++) {                                     \
            if (r >= rounds) break;                                                         \
            const E j = (E)(r * G + lane);                                                  \
            q[r] = NULL_PART;                                                               \
            if (j < d) {                                                                    \
                const part_t pv = part[g.adj[s + j]];                                       \
                if (pv != own) { q[r] = pv; acc += g.val[s + j]; }                          \
            }                                                                               \
        }                                                                                   \
        /* a lane's part counts where no earlier edge of the row has it */                  \
        _Pragma("unroll") for (int r = 0; r < R; r++) {                                     \
            if (r >= rounds) break;                                                         \
            bool first = q[r] != NULL_PART;                                                 \
            _Pragma("unroll") for (int r2 = 0; r2 <= r; r2++)                               \
                for (int l = 0; l < G; l++) {                                               \
                    const part_t o = __shfl_sync(0xffffffffu, q[r2], l, G);                 \
                    if (o == q[r] && (r2 < r || l < lane)) first = false;                   \
                }                                                                           \
            comm += first;                                                                  \
        }                                                                                   \
        acc = group_sum<W>(acc, G);                                                         \
        warp_hist_add<W>(h_per, own, acc, ok && lane == 0 && acc != 0);                     \
        warp_hist_add<W>(h_sz, own, vw, ok && lane == 0);                                   \
    }
    JET_GROUP_LOOP(G, g.n, PSTAT_BODY)
#undef PSTAT_BODY
    comm = group_sum<long long>(comm, 32);
    if ((threadIdx.x & 31) == 0 && comm) atomicAdd((unsigned long long*)out.comm, (unsigned long long)comm);
    if (hist) {
        __syncthreads();
        for (int p = threadIdx.x; p < k; p += blockDim.x) {
            if (h_per[p]) atomic_add(&out.per[p], h_per[p]);
            if (h_sz[p]) atomic_add(&out.sizes[p], h_sz[p]);
        }
    }
}

// Rows of more than 32 edges: one warp (BLOCKWIDE: one block) per row, the
// distinct parts in a bitmap of `words` words.
template <bool BLOCKWIDE, class O, class E, class W>
__global__ void __launch_bounds__(BLOCKWIDE ? 1024 : BLOCK) k_pstat_long(GView<O, E, W> g, const part_t* part, part_t k,
                                                                         const O* list, O count, PStatOut<W> out, int words) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int t = BLOCKWIDE ? threadIdx.x : lane, nt = BLOCKWIDE ? (int)blockDim.x : 32;
    uint32_t* bm = (uint32_t*)smem_raw + (BLOCKWIDE ? 0 : (size_t)wid * words);
    const int64_t units = BLOCKWIDE ? (int64_t)gridDim.x : (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t first = BLOCKWIDE ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * (blockDim.x >> 5) + wid;
    long long comm = 0;
    for (int64_t x = first; x < (int64_t)count; x += units) {
        const O i = list[x];
        const part_t own = part[i];
        if (own < 0 || own >= k) continue;  // reported by k_pstat_rows
        for (int w = t; w < words; w += nt) bm[w] = 0;
        if (BLOCKWIDE) __syncthreads(); else __syncwarp();
        W acc = 0;
        const Cursor<E> re = g.row[i + 1];
        for (Cursor<E> j0 = (Cursor<E>)g.row[i] + t; j0 < re; j0 += 4 * nt) {
            O v[4];
            W w[4];
            part_t p[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const Cursor<E> j = j0 + u * nt;
                v[u] = j < re ? g.adj[j] : (O)0;
                w[u] = j < re ? g.val[j] : (W)0;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) p[u] = j0 + u * nt < re ? part[v[u]] : own;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (p[u] == own || p[u] < 0 || p[u] >= k) continue;
                acc += w[u];
                const uint32_t bit = 1u << (p[u] & 31);
                if (!(((volatile uint32_t*)bm)[p[u] >> 5] & bit)) atomicOr(&bm[p[u] >> 5], bit);
            }
        }
        acc = group_sum<W>(acc, 32);
        if (lane == 0 && acc) atomic_add(&out.per[own], acc);
        if (BLOCKWIDE) __syncthreads(); else __syncwarp();
        for (int w = t; w < words; w += nt) comm += __popc(bm[w]);
        if (BLOCKWIDE) __syncthreads(); else __syncwarp();
    }
    comm = group_sum<long long>(comm, 32);
    if (lane == 0 && comm) atomicAdd((unsigned long long*)out.comm, (unsigned long long)comm);
}

}  // namespace jetb
