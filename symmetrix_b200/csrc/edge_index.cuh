// Index arrays of an edge set for structures of up to kIndexMaxNodes nodes, built by one CTA: CSR offsets of the receivers,
// nodes in element-type order, and the work items of the reverse edge kernels. Larger sets use device-wide scans and sorts
// (Evaluator::adopt_edges), where ten launches cost little against the evaluation; for a few hundred atoms those launches,
// 2 to 5 us each for a few hundred values, were a fifth of the whole call.
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"

namespace smx {

constexpr int kIndexThreads = 1024;
// Threads for `count` entries: barriers of few warps are cheaper.
inline int index_threads(int count) { return count >= kIndexThreads ? kIndexThreads : (count + 31) / 32 * 32; }
constexpr int kIndexMaxNodes = 8192;      // 8 nodes per thread: about 10 us (30,000 nodes: 130 us, three times the device-wide
                                          // launches); packed 16-bit counts stay exact
constexpr int kIndexMaxTypes = 16;        // four packed counters per 64-bit word, four words
constexpr int kIndexMaxBins = 4096;       // neighbour bins whose counts fit into 16 KB of shared memory

// Exclusive prefix sum over the threads of the CTA; `total` is the sum over all of them. `sh` holds 33 values.
template <typename U>
__device__ __forceinline__ U block_exclusive_sum(U v, U* sh, U& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    U x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const U y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        U t = lane < nwarps ? sh[lane] : U(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const U y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        sh[lane] = t;
    }
    __syncthreads();
    const U before = warp ? sh[warp - 1] : U(0);
    total = sh[nwarps - 1];
    __syncthreads();      // sh may be written again
    return before + x - v;
}

// Stable sort of the nodes by element type: perm, and the first position of every type in seg. A thread owns a contiguous
// run of nodes; its counts per type, four to a 64-bit word, are summed over the CTA with one scan per word.
__device__ __forceinline__ void index_sort_types(int n, const int* __restrict__ types, int num_types, int* __restrict__ perm,
                                                 int* __restrict__ seg, unsigned long long* sh, int* sh_seg) {
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int begin = min(static_cast<int>(threadIdx.x) * per, n), end = min(begin + per, n);
    auto type_of = [&](int i) { return min(max(types[i], 0), num_types - 1); };     // a bad type must not index out of range
    unsigned long long w[4] = {0, 0, 0, 0}, total;
    for (int i = begin; i < end; ++i) {
        const int t = type_of(i);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if ((t >> 2) == q) w[q] += 1ull << ((t & 3) * 16);
    }
    const int words = (num_types + 3) / 4;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q < words) {
            w[q] = block_exclusive_sum(w[q], sh, total);
            if (threadIdx.x < 4) sh_seg[4 * q + threadIdx.x + 1] = static_cast<int>((total >> (threadIdx.x * 16)) & 0xffffu);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        sh_seg[0] = 0;
        for (int t = 0; t < num_types; ++t) { sh_seg[t + 1] += sh_seg[t]; seg[t + 1] = sh_seg[t + 1]; }
        seg[0] = 0;
    }
    __syncthreads();
    for (int i = begin; i < end; ++i) {
        const int t = type_of(i);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if ((t >> 2) == q) {
                perm[sh_seg[t] + static_cast<int>((w[q] >> ((t & 3) * 16)) & 0xffffu)] = i;
                w[q] += 1ull << ((t & 3) * 16);
            }
    }
    __syncthreads();
}

// What an evaluation on the device leaves for the host, in front of the per-atom results.
struct EvalHead {
    long long edges;          // edges of the structure
    int shift_overflow;       // an atom lies too many cells away (see neigh_rows_kernel)
    int row_max;              // longest row, where it exceeds the capacity of a row
    int unpaired;             // edges whose opposite is not in the list
    int status;               // kernel status word (bounded waits)
    double out7[7];           // energy and virial
    double pad;
};

struct EdgeIndexArgs {
    int n;
    const int* types; int num_types; int* perm; int* seg;      // types == nullptr: perm and seg are kept
    const int* num_neigh;                                      // nullptr: first is kept
    long long* first;
    long long edges;              // number of edges, or -1: the sum of num_neigh
    int type_order;               // items follow perm (otherwise natural order)
    int want_items; int4* items; int items_cap; int* n_items; int* sched;
    double* node_energies;        // zeroed where given
    // structures built on the device: rows and edge arrays have a fixed capacity; a structure that exceeds it becomes one
    // without edges and the host, which finds the true numbers in the head, enlarges the arrays and starts again. So does one
    // with shifts beyond the ten bits a key has for them (its keys name no valid senders); the host reports that as an error
    long long edge_cap; int row_cap; EvalHead* head;
};

static __global__ void __launch_bounds__(kIndexThreads) edge_index_kernel(const EdgeIndexArgs a) {
    chain_begin();
    __shared__ unsigned long long sh[33];
    __shared__ int sh_seg[kIndexMaxTypes + 1];
    const int tid = threadIdx.x, n = a.n;
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int begin = min(tid * per, n), end = min(begin + per, n);
    if (a.types) index_sort_types(n, a.types, a.num_types, a.perm, a.seg, sh, sh_seg);
    long long edges;
    if (a.num_neigh) {
        unsigned long long mine = 0, total;
        for (int i = begin; i < end; ++i) mine += static_cast<unsigned long long>(static_cast<long long>(a.num_neigh[i]));
        unsigned long long at = block_exclusive_sum(mine, sh, total);
        const bool fits = !a.head || (static_cast<long long>(total) <= a.edge_cap && a.head->row_max <= a.row_cap && a.head->shift_overflow == 0);
        for (int i = begin; i < end; ++i) {
            a.first[i] = fits ? static_cast<long long>(at) : 0;
            at += static_cast<unsigned long long>(static_cast<long long>(a.num_neigh[i]));
        }
        edges = a.edges >= 0 ? a.edges : (fits ? static_cast<long long>(total) : 0);
        if (tid == 0) {
            a.first[n] = edges;
            if (a.head) a.head->edges = static_cast<long long>(total);
        }
        __syncthreads();
    } else {
        edges = a.first[n];
    }
    const int batch = work_batch(edges, a.want_items);
    auto degree = [&](int slot, int& i) {
        i = a.type_order ? a.perm[slot] : slot;
        return static_cast<int>(a.first[i + 1] - a.first[i]);
    };
    int mine = 0, total, i;
    for (int s = begin; s < end; ++s) { const int deg = degree(s, i); mine += deg > 0 ? (deg + batch - 1) / batch : 0; }
    int at = block_exclusive_sum(mine, reinterpret_cast<int*>(sh), total);
    for (int s = begin; s < end; ++s) {
        const int deg = degree(s, i), nb = deg > 0 ? (deg + batch - 1) / batch : 0, size = nb ? (deg + nb - 1) / nb : 0;
        for (int b = 0; b < nb; ++b, ++at)
            if (at < a.items_cap) a.items[at] = make_int4(i, b * size, min(size, deg - b * size), 0);
        if (a.node_energies) a.node_energies[s] = 0.0;
    }
    if (tid == 0) { *a.n_items = min(total, a.items_cap); a.sched[0] = 0; a.sched[1] = 0; }
}

// ---------------------------------------------------------------------------------------------
// Last kernel of an evaluation whose results go to the host: per-atom forces, energy and virial in one pass over the edges
// (a warp per atom reads the partial forces of its own row once for the force and the virial, and those of its senders' rows
// for the force), written behind the head into one block that a single copy brings to the host. The CTA that finishes last
// adds the partial sums of all CTAs in a fixed order.
// ---------------------------------------------------------------------------------------------
constexpr int kFinishThreads = 128;
static __global__ void __launch_bounds__(kFinishThreads) finish_kernel(int n, const long long* __restrict__ first_neigh, const long long* __restrict__ in_ptr,
                                                                       const int* __restrict__ in_edge, const double* __restrict__ xyz,
                                                                       const double* __restrict__ nf, const double* __restrict__ node_energies,
                                                                       const int* __restrict__ status, double* __restrict__ partials,
                                                                       unsigned* __restrict__ done, EvalHead* __restrict__ head,
                                                                       double* __restrict__ forces, double* __restrict__ energies) {
    chain_begin();
    constexpr int kWarps = kFinishThreads / 32;
    __shared__ double sh[kWarps][7];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int i = blockIdx.x * kWarps + warp; i < n; i += gridDim.x * kWarps) {
        double f0 = 0, f1 = 0, f2 = 0;
        for (long long e = first_neigh[i] + lane; e < first_neigh[i + 1]; e += 32) {
            const double x = xyz[3 * e], y = xyz[3 * e + 1], z = xyz[3 * e + 2];
            const double px = nf[3 * e], py = nf[3 * e + 1], pz = nf[3 * e + 2];
            f0 -= px; f1 -= py; f2 -= pz;
            v[1] += x * px; v[2] += y * py; v[3] += z * pz;
            v[4] += 0.5 * (x * py + y * px); v[5] += 0.5 * (x * pz + z * px); v[6] += 0.5 * (y * pz + z * py);
        }
        for (long long m = in_ptr[i] + lane; m < in_ptr[i + 1]; m += 32) {
            const long long e = in_edge[m];
            f0 += nf[3 * e]; f1 += nf[3 * e + 1]; f2 += nf[3 * e + 2];
        }
        f0 = warp_sum(f0); f1 = warp_sum(f1); f2 = warp_sum(f2);
        if (lane == 0) {
            forces[3 * i] = f0; forces[3 * i + 1] = f1; forces[3 * i + 2] = f2;
            energies[i] = node_energies[i];
            v[0] += node_energies[i];
        }
    }
#pragma unroll
    for (int c = 0; c < 7; ++c) {
        const double s = warp_sum(v[c]);
        if (lane == 0) sh[warp][c] = s;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double s = 0;
        for (int w = 0; w < kWarps; ++w) s += sh[w][threadIdx.x];
        partials[blockIdx.x * 7 + threadIdx.x] = s;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int c = warp; c < 7; c += kWarps) {
        double s = 0;
        for (unsigned b = lane; b < gridDim.x; b += 32) s += __ldcg(partials + b * 7 + c);
        s = warp_sum(s);
        if (lane == 0) head->out7[c] = s;
    }
    if (threadIdx.x == 0) { *done = 0; head->status = *status; }
}

}  // namespace smx
