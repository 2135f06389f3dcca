// Full periodic neighbour list on the device, written directly in the evaluator's CSR form.
//
// Edge rule (identical, operation for operation, to symmetrix_b200/structures.py::neighbor_list,
// which restates what the reference's callers do, pair_symmetrix/pair_symmetrix_mace.cpp:249-315):
//   p = x_j + ((n0*a0 + n1*a1) + n2*a2)        image position, float64, no fused multiply-add
//   d = p - x_i
//   keep iff (d0*d0 + d1*d1) + d2*d2 < r_cut*r_cut, excluding i == j with a zero shift
// Rows are ordered by (sender index, shift code), so the list is a pure function of its inputs. One warp builds one row.
// Candidates come from a uniform grid over fractional coordinates whose cells are at least
// r_cut(1+1e-9) thick. Positions need not lie inside the cell: along a periodic axis an atom is binned by its
// wrapped fractional coordinate, and the whole cell vectors w_i it is away from the cell are folded into the
// integer shift of its edges (n = n' + w_i - w_j for the image n' found between the wrapped positions), so xyz
// is still formed from the positions as given. Along a non-periodic axis outliers go to the edge bins.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include <cub/cub.cuh>

#include "common.cuh"
#include "edge_index.cuh"

namespace smx {

struct NeighGrid {
    double cell[9];      // rows are lattice vectors
    double inv[9];       // inverse of the cell matrix: frac = pos . inv
    int nb[3];           // bins per axis
    int reach[3];        // bins to search on each side
    int pbc[3];
    double rc2;
};

// Bin of an atom and (w3) the whole cell vectors its position is away from the cell along the periodic axes.
__device__ __forceinline__ int neigh_bin(const NeighGrid& g, const double* x, int* b3, int* w3) {
    int id = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double s = x[0] * g.inv[0 * 3 + a] + x[1] * g.inv[1 * 3 + a] + x[2] * g.inv[2 * 3 + a];
        const double wf = g.pbc[a] ? floor(s) : 0.0;
        // far outliers are clamped here and rejected by the shift-range check of neigh_rows_kernel
        w3[a] = static_cast<int>(wf < -1e6 ? -1e6 : (wf > 1e6 ? 1e6 : wf));
        s -= wf;
        int b = static_cast<int>(floor(s * g.nb[a]));
        b = b < 0 ? 0 : (b >= g.nb[a] ? g.nb[a] - 1 : b);
        b3[a] = b;
        id = id * g.nb[a] + b;
    }
    return id;
}

static __global__ void neigh_bin_kernel(int n, const double* __restrict__ pos, NeighGrid g, int* __restrict__ bin_of,
                                        int* __restrict__ wrap) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int b3[3];
        bin_of[i] = neigh_bin(g, pos + 3 * i, b3, wrap + 3 * i);
    }
}

// Exact edge test; returns true and fills d/r2 when image (j, n) of atom j is a neighbour of i.
__device__ __forceinline__ bool neigh_test(const NeighGrid& g, const double* xi, const double* xj, int n0, int n1, int n2,
                                           double* d, double* r2) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double sv = __dadd_rn(__dadd_rn(__dmul_rn(double(n0), g.cell[0 + c]), __dmul_rn(double(n1), g.cell[3 + c])),
                                    __dmul_rn(double(n2), g.cell[6 + c]));
        const double p = __dadd_rn(xj[c], sv);
        d[c] = __dsub_rn(p, xi[c]);
    }
    *r2 = __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2]));
    return *r2 < g.rc2;
}

// Sort key of an edge inside its row: sender first, then the shift in lexicographic order. Shifts are kept in
// 10 bits per axis (|n| <= kNeighMaxShift).
constexpr int kNeighMaxShift = 511;
__device__ __forceinline__ unsigned long long neigh_key(int j, int n0, int n1, int n2) {
    const unsigned long long code = (static_cast<unsigned long long>(n0 + 512) * 1024 + (n1 + 512)) * 1024 + (n2 + 512);
    return (static_cast<unsigned long long>(j) << 32) | code;
}

// One warp per receiver atom, or WPR = 4 warps where there are few atoms. The bins around the atom's bin are taken 32 at a time,
// one per lane; a scan over their sizes numbers their atoms, and the lanes then share the candidates evenly whatever the bins
// hold (a unit cell has hundreds of images of four atoms; one bin after the other with a warp cost 0.5 us of latency per
// image). The candidates' positions are stored in bin order, so a step waits for one load, not for an index and then a
// position. Keys of the row's edges are collected in the order they are found in a scratch row of `cap` keys; a row that
// does not fit reports its length in head->row_max. cap = 0: the rows have exactly their lengths, at the offsets `first`.
constexpr int kNeighWarps = 4;           // warps per CTA
constexpr int kNeighRowCap = 512;        // keys of one row ranked in shared memory
// Four warps per atom below this many atoms (about two warps per scheduler then): 420 atoms of 945 candidates, 24 us with one.
constexpr int kNeighWideRows = 1184;

__device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

template <int WPR>
static __global__ void __launch_bounds__(kNeighWarps * 32) neigh_rows_kernel(
    int n, const double* __restrict__ pos, NeighGrid g, const int* __restrict__ bin_start, const double* __restrict__ sorted_pos,
    const int4* __restrict__ sorted_atoms, int cap, const long long* __restrict__ first_neigh, unsigned long long* __restrict__ keys,
    int* __restrict__ num_neigh, EvalHead* __restrict__ head) {
    chain_begin();
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ int found[kNeighWarps];     // edges of the row so far, per row of the CTA
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slot0 = warp / WPR, part = warp % WPR;
    constexpr int kRows = kNeighWarps / WPR;
    const int w1 = 2 * g.reach[1] + 1, w2 = 2 * g.reach[2] + 1, cells = (2 * g.reach[0] + 1) * w1 * w2;
    for (int first = blockIdx.x * kRows; first < n; first += gridDim.x * kRows) {
        const int i = first + slot0;
        if (WPR > 1) __syncthreads(); else __syncwarp();
        if (part == 0 && lane == 0) found[slot0] = 0;
        if (WPR > 1) __syncthreads(); else __syncwarp();
        if (i < n) {
            const double xi[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
            unsigned long long* row = keys + (cap ? static_cast<long long>(i) * cap : first_neigh[i]);
            const int room = cap ? cap : static_cast<int>(first_neigh[i + 1] - first_neigh[i]);
            int b3[3], wi[3];
            neigh_bin(g, xi, b3, wi);
            for (int c0 = 0; c0 < cells; c0 += 32) {
                const int cell = c0 + lane;
                int start = 0, size = 0, n0 = 0, n1 = 0, n2 = 0;
                if (cell < cells) {
                    const int o0 = cell / (w1 * w2), o1 = cell / w2 % w1, o2 = cell % w2;
                    const int v0 = b3[0] + o0 - g.reach[0], v1 = b3[1] + o1 - g.reach[1], v2 = b3[2] + o2 - g.reach[2];
                    n0 = floor_div(v0, g.nb[0]); n1 = floor_div(v1, g.nb[1]); n2 = floor_div(v2, g.nb[2]);
                    if ((n0 == 0 || g.pbc[0]) && (n1 == 0 || g.pbc[1]) && (n2 == 0 || g.pbc[2])) {
                        const int bin = ((v0 - n0 * g.nb[0]) * g.nb[1] + v1 - n1 * g.nb[1]) * g.nb[2] + v2 - n2 * g.nb[2];
                        start = bin_start[bin];
                        size = bin_start[bin + 1] - start;
                    }
                }
                int upto = size;               // atoms in the bins of the lanes up to this one
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kAll, upto, o);
                    if (lane >= o) upto += y;
                }
                const int total = __shfl_sync(kAll, upto, 31);
                const int from = start - (upto - size);      // atom t of the numbering is entry from + t of its lane
                for (int t0 = 32 * part; t0 < total; t0 += 32 * WPR) {
                    const int t = t0 + lane;
                    int src = 0;               // first lane whose bins reach beyond t
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1)
                        if (__shfl_sync(kAll, upto, src + step - 1) <= t) src += step;
                    src = src < 32 ? src : 31;
                    const int s = __shfl_sync(kAll, from, src) + t;
                    const int q0 = __shfl_sync(kAll, n0, src), q1 = __shfl_sync(kAll, n1, src), q2 = __shfl_sync(kAll, n2, src);
                    bool hit = false;
                    unsigned long long key = 0;
                    if (t < total) {
                        const int4 other = sorted_atoms[s];                 // (atom, whole cells it is away from the cell)
                        const double xj[3] = {sorted_pos[3 * s], sorted_pos[3 * s + 1], sorted_pos[3 * s + 2]};
                        if (!(other.x == i && q0 == 0 && q1 == 0 && q2 == 0)) {
                            // shift between the positions as given: image between the wrapped positions + the two wraps
                            const int m0 = q0 + wi[0] - other.y, m1 = q1 + wi[1] - other.z, m2 = q2 + wi[2] - other.w;
                            double d[3], r2;
                            if (neigh_test(g, xi, xj, m0, m1, m2, d, &r2)) {
                                hit = true;
                                if (abs(m0) > kNeighMaxShift || abs(m1) > kNeighMaxShift || abs(m2) > kNeighMaxShift) head->shift_overflow = 1;
                                key = neigh_key(other.x, m0, m1, m2);
                            }
                        }
                    }
                    const unsigned mask = __ballot_sync(kAll, hit);
                    int at = 0;
                    if (mask) {
                        if (lane == 0) at = atomicAdd(&found[slot0], __popc(mask));
                        at = __shfl_sync(kAll, at, 0) + __popc(mask & ((1u << lane) - 1u));
                    }
                    if (hit && at < room) row[at] = key;
                }
            }
        }
        if (WPR > 1) __syncthreads(); else __syncwarp();
        if (i < n && part == 0 && lane == 0) {
            const int count = found[slot0];
            num_neigh[i] = count;
            if (cap && count > cap) atomicMax(&head->row_max, count);
        }
    }
}

// Ranks the keys of every row (they are unique, so a key's rank is the number of smaller ones: the row comes out ordered by
// (sender, shift) whatever order it was found in) and expands each into the edge arrays with the arithmetic that tested it.
// Does nothing when a row or the edge arrays were too small (first_neigh is zero then).
static __global__ void __launch_bounds__(kNeighWarps * 32) neigh_fill_kernel(
    int n, const double* __restrict__ pos, const int* __restrict__ types, NeighGrid g, int cap, const unsigned long long* __restrict__ keys,
    const long long* __restrict__ first_neigh, unsigned long long* __restrict__ sorted_keys, int* __restrict__ neigh_indices,
    int* __restrict__ neigh_types, int* __restrict__ shifts, double* __restrict__ xyz, double* __restrict__ r, double* __restrict__ node_forces) {
    chain_begin();
    __shared__ unsigned long long row_keys[kNeighWarps][kNeighRowCap];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = blockIdx.x * kNeighWarps + warp; i < n; i += gridDim.x * kNeighWarps) {
        const long long row_begin = first_neigh[i];
        const int count = static_cast<int>(first_neigh[i + 1] - row_begin);
        const double xi[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
        const unsigned long long* row = keys + (cap ? static_cast<long long>(i) * cap : row_begin);      // as neigh_rows_kernel
        const bool in_smem = count <= kNeighRowCap;
        __syncwarp();
        if (in_smem) for (int a = lane; a < count; a += 32) row_keys[warp][a] = row[a];
        __syncwarp();
        for (int a = lane; a < count; a += 32) {
            const unsigned long long key = in_smem ? row_keys[warp][a] : row[a];
            int rank = 0;
            for (int b = 0; b < count; ++b) rank += (in_smem ? row_keys[warp][b] : row[b]) < key ? 1 : 0;
            const long long e = row_begin + rank;
            const int j = static_cast<int>(key >> 32);
            const unsigned int code = static_cast<unsigned int>(key & 0xffffffffu);
            const int n2 = static_cast<int>(code % 1024) - 512, n1 = static_cast<int>((code / 1024) % 1024) - 512,
                      n0 = static_cast<int>(code / (1024 * 1024)) - 512;
            double d[3], r2;
            neigh_test(g, xi, pos + 3 * j, n0, n1, n2, d, &r2);
            sorted_keys[e] = key;
            neigh_indices[e] = j;
            neigh_types[e] = types[j];
            shifts[3 * e] = n0; shifts[3 * e + 1] = n1; shifts[3 * e + 2] = n2;
            xyz[3 * e] = d[0]; xyz[3 * e + 1] = d[1]; xyz[3 * e + 2] = d[2];
            r[e] = __dsqrt_rn(r2);
            node_forces[3 * e] = 0.0; node_forces[3 * e + 1] = 0.0; node_forces[3 * e + 2] = 0.0;      // what an evaluation starts from
        }
    }
}

// Edges grouped by sender without a sort: the list is full, so the edges that atom i sends are the opposites (j, i, -shift)
// of the edges (i, j, shift) it receives, and row i of `opposite` lists them in a fixed order. Each is found by bisection in
// the keys of row j. Two opposite edges are tested with differently rounded distances, so an edge within rounding of the
// cutoff can be in the list alone: such edges are counted and the caller sorts instead.
static __global__ void __launch_bounds__(128) neigh_opposite_kernel(int n, const long long* __restrict__ first_neigh,
                                                                    const unsigned long long* __restrict__ sorted_keys,
                                                                    int* __restrict__ opposite, EvalHead* __restrict__ head) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    for (int i = blockIdx.x * 4 + (threadIdx.x >> 5); i < n; i += gridDim.x * 4) {
        for (long long e = first_neigh[i] + lane; e < first_neigh[i + 1]; e += 32) {
            const unsigned long long key = sorted_keys[e];
            const int j = static_cast<int>(key >> 32);
            const unsigned int code = static_cast<unsigned int>(key & 0xffffffffu);
            const unsigned long long want = neigh_key(i, 512 - static_cast<int>(code / (1024 * 1024)), 512 - static_cast<int>((code / 1024) % 1024),
                                                      512 - static_cast<int>(code % 1024));
            long long lo = first_neigh[j], hi = first_neigh[j + 1];
            const long long end = hi;
            while (lo < hi) {
                const long long mid = (lo + hi) >> 1;
                if (sorted_keys[mid] < want) lo = mid + 1; else hi = mid;
            }
            const bool found = lo < end && sorted_keys[lo] == want;
            opposite[e] = found ? static_cast<int>(lo) : static_cast<int>(e);
            if (!found) atomicAdd(&head->unpaired, 1);
        }
    }
}

// Atom i as entry s of the bin order.
__device__ __forceinline__ void neigh_place(int i, int s, const double* pos, const int* wrap, double* sorted_pos, int4* sorted_atoms) {
    sorted_atoms[s] = make_int4(i, wrap[3 * i], wrap[3 * i + 1], wrap[3 * i + 2]);
    sorted_pos[3 * s] = pos[3 * i]; sorted_pos[3 * s + 1] = pos[3 * i + 1]; sorted_pos[3 * s + 2] = pos[3 * i + 2];
}
static __global__ void neigh_place_kernel(int n, const int* __restrict__ order, const double* __restrict__ pos, const int* __restrict__ wrap,
                                          double* __restrict__ sorted_pos, int4* __restrict__ sorted_atoms) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) neigh_place(order[s], s, pos, wrap, sorted_pos, sorted_atoms);
}

// Bins and, for the evaluation that follows, the type order of up to kIndexMaxNodes atoms in at most kIndexMaxBins bins, in one
// CTA (bin, count, scan, scatter with shared-memory counters; the order inside a bin does not matter). Clears the head.
static __global__ void __launch_bounds__(kIndexThreads) neigh_prepare_kernel(int n, const double* __restrict__ pos, NeighGrid g, int nbins,
                                                                             int* __restrict__ bin_of, int* __restrict__ wrap, int* __restrict__ bin_start,
                                                                             double* __restrict__ sorted_pos, int4* __restrict__ sorted_atoms, const int* __restrict__ types, int num_types,
                                                                             int* __restrict__ perm, int* __restrict__ seg, EvalHead* __restrict__ head) {
    chain_begin();
    __shared__ unsigned long long sh[33];
    __shared__ int sh_seg[kIndexMaxTypes + 1];
    __shared__ int counts[kIndexMaxBins];
    const int tid = threadIdx.x;
    for (int b = tid; b < nbins; b += blockDim.x) counts[b] = 0;
    if (tid == 0) { head->edges = 0; head->shift_overflow = 0; head->row_max = 0; head->unpaired = 0; }
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) {
        int b3[3];
        const int b = neigh_bin(g, pos + 3 * i, b3, wrap + 3 * i);
        bin_of[i] = b;
        atomicAdd(&counts[b], 1);
    }
    __syncthreads();
    const int per = (nbins + blockDim.x - 1) / blockDim.x, begin = min(tid * per, nbins), end = min(begin + per, nbins);
    unsigned long long mine = 0, total;
    for (int b = begin; b < end; ++b) mine += counts[b];
    int at = static_cast<int>(block_exclusive_sum(mine, sh, total));
    for (int b = begin; b < end; ++b) { const int c = counts[b]; bin_start[b] = at; counts[b] = at; at += c; }
    if (tid == 0) bin_start[nbins] = n;
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) neigh_place(i, atomicAdd(&counts[bin_of[i]], 1), pos, wrap, sorted_pos, sorted_atoms);
    __syncthreads();
    index_sort_types(n, types, num_types, perm, seg, sh, sh_seg);
}

static __global__ void neigh_iota_kernel(int n, int* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = i;
}
static __global__ void neigh_offsets_kernel(int n, const int* __restrict__ sorted_keys, int num_values, int* __restrict__ offsets) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= num_values; v += gridDim.x * blockDim.x) {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sorted_keys[mid] < v) lo = mid + 1; else hi = mid;
        }
        offsets[v] = lo;
    }
}

// Sum of the row lengths into the head (the host sizes the edge arrays by it).
static __global__ void __launch_bounds__(1024) neigh_total_kernel(int n, const int* __restrict__ num_neigh, EvalHead* __restrict__ head) {
    __shared__ unsigned long long sh[33];
    unsigned long long mine = 0, total;
    for (int i = threadIdx.x; i < n; i += blockDim.x) mine += static_cast<unsigned long long>(num_neigh[i]);
    block_exclusive_sum(mine, sh, total);
    if (threadIdx.x == 0) head->edges = static_cast<long long>(total);
}

class NeighborBuilder {
public:
    DevBuf<double> d_pos, sorted_pos;
    DevBuf<int4> sorted_atoms;
    DevBuf<int> bin_of, sorted_bins, order, iota, bin_start, wrap;
    DevBuf<unsigned long long> keys, sorted_keys;
    DevBuf<unsigned char> tmp;
    // Keys of one row: what the longest row so far needed, for structures where that is no more memory than kFreeKeys, than is
    // there, or than four times the edges; otherwise kRowCap, and if a row is longer (a dense cluster in a large sparse box) the rows
    // are found twice, the second time into exactly their lengths. (One cell with rows of 5,673 made a later box of 197,136
    // atoms allocate 11 GB of keys.)
    static constexpr int kRowCap = 128;
    static constexpr size_t kFreeKeys = 1u << 22;
    int row_cap = kRowCap;
    int cap = kRowCap;            // of the structure at hand; 0: by offsets
    NeighGrid g{};
    int nbins = 1;

    void set_cell(const double* cell, const int* pbc, double r_cut) {
        if (!(r_cut > 0.0)) throw ArgError("build_neighbors: r_cut must be positive");
        for (int q = 0; q < 9; ++q) g.cell[q] = cell[q];
        const double* a = cell;
        const double det = a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) + a[2] * (a[3] * a[7] - a[4] * a[6]);
        if (std::fabs(det) < 1e-300) throw ArgError("build_neighbors: singular cell");
        g.inv[0] = (a[4] * a[8] - a[5] * a[7]) / det; g.inv[1] = (a[2] * a[7] - a[1] * a[8]) / det; g.inv[2] = (a[1] * a[5] - a[2] * a[4]) / det;
        g.inv[3] = (a[5] * a[6] - a[3] * a[8]) / det; g.inv[4] = (a[0] * a[8] - a[2] * a[6]) / det; g.inv[5] = (a[2] * a[3] - a[0] * a[5]) / det;
        g.inv[6] = (a[3] * a[7] - a[4] * a[6]) / det; g.inv[7] = (a[1] * a[6] - a[0] * a[7]) / det; g.inv[8] = (a[0] * a[4] - a[1] * a[3]) / det;
        long long total_bins = 1;
        for (int ax = 0; ax < 3; ++ax) {
            const double* u = cell + 3 * ((ax + 1) % 3);
            const double* v = cell + 3 * ((ax + 2) % 3);
            const double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2], cz = u[0] * v[1] - u[1] * v[0];
            const double height = std::fabs(det) / std::sqrt(cx * cx + cy * cy + cz * cz);
            const double rc = r_cut * (1.0 + 1e-9);
            int bins = static_cast<int>(std::floor(height / rc));
            if (bins < 1) bins = 1;
            if (bins > 256) bins = 256;
            g.nb[ax] = bins;
            g.reach[ax] = static_cast<int>(std::ceil(rc / (height / bins)));
            if (!pbc[ax] && g.reach[ax] > bins) g.reach[ax] = bins;
            if (g.reach[ax] > 63 * bins) throw ArgError("build_neighbors: cell far smaller than r_cut");
            g.pbc[ax] = pbc[ax] ? 1 : 0;
            total_bins *= bins;
        }
        g.rc2 = r_cut * r_cut;
        nbins = static_cast<int>(total_bins);
    }
    void size_arrays(int n, cudaStream_t stream) {
        bin_of.resize(n, stream); sorted_atoms.resize(n, stream); sorted_pos.resize(3 * static_cast<size_t>(n), stream);
        bin_start.resize(static_cast<size_t>(nbins) + 1, stream);
        wrap.resize(3 * static_cast<size_t>(n), stream);
    }
    // Atoms sorted into bins with device-wide kernels (any number of atoms and bins); clears the head.
    void bin_atoms(int n, const double* dpos, EvalHead* head, cudaStream_t stream, long& launches) {
        size_arrays(n, stream);
        sorted_bins.resize(n, stream); order.resize(n, stream); iota.resize(n, stream);
        SMX_CUDA(cudaMemsetAsync(head, 0, sizeof(EvalHead), stream));
        const int blocks = std::min(4096, (n + 127) / 128);
        neigh_bin_kernel<<<blocks, 128, 0, stream>>>(n, dpos, g, bin_of.p, wrap.p);
        neigh_iota_kernel<<<blocks, 128, 0, stream>>>(n, iota.p);
        int bits = 1;
        while ((1LL << bits) < nbins) ++bits;
        size_t bytes = 0;
        SMX_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, bin_of.p, sorted_bins.p, iota.p, order.p, n, 0, bits, stream));
        tmp.resize(bytes, stream);
        SMX_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, bytes, bin_of.p, sorted_bins.p, iota.p, order.p, n, 0, bits, stream));
        neigh_offsets_kernel<<<std::min(1024, (nbins + 128) / 128), 128, 0, stream>>>(n, sorted_bins.p, nbins, bin_start.p);
        neigh_place_kernel<<<blocks, 128, 0, stream>>>(n, order.p, dpos, wrap.p, sorted_pos.p, sorted_atoms.p);
        launches += 5;
    }
    // The same for small sets in one launch, with the type order of the atoms as well.
    void bin_atoms_small(const Launcher& on, int n, const double* dpos, EvalHead* head, const int* types, int num_types, int* perm, int* seg, long& launches) {
        size_arrays(n, on.stream);
        chain_launch(on, neigh_prepare_kernel, dim3(1), index_threads(std::max(n, nbins)), 0, 1, n, dpos, g, nbins, bin_of.p, wrap.p, bin_start.p, sorted_pos.p, sorted_atoms.p, types, num_types, perm, seg, head);
        launches += 1;
    }
    static int row_blocks(int n) { return std::min(16384, (n + kNeighWarps - 1) / kNeighWarps); }      // one warp per atom
    void choose_rows(int n) { cap = static_cast<size_t>(n) * row_cap <= std::max(kFreeKeys, keys.cap) ? row_cap : kRowCap; }
    // A row was longer than `cap`: more room for every row, in steps of 32, or (false) the rows must go by their offsets.
    bool grow_rows(int n, int row_max, long long edges) {
        const int want = static_cast<int>((row_max + static_cast<long long>(row_max) / 8 + 31) / 32 * 32);
        const size_t all = static_cast<size_t>(n) * want;
        if (all > std::max(std::max(kFreeKeys, keys.cap), 4 * static_cast<size_t>(edges))) return false;
        cap = want;
        row_cap = std::max(row_cap, want);
        return true;
    }
    void rows_by_offsets() { cap = 0; }
    // first, edges: only with rows_by_offsets (the row lengths are known then and stay)
    void find_rows(const Launcher& on, int n, const double* dpos, int* num_neigh, const long long* first, size_t edges, EvalHead* head, long& launches) {
        keys.resize(cap ? static_cast<size_t>(n) * cap : edges, on.stream);
        if (n <= kNeighWideRows) chain_launch(on, neigh_rows_kernel<4>, dim3(n), kNeighWarps * 32, 0, 1, n, dpos, g, bin_start.p, sorted_pos.p, sorted_atoms.p, cap, first, keys.p, num_neigh, head);
        else chain_launch(on, neigh_rows_kernel<1>, dim3(row_blocks(n)), kNeighWarps * 32, 0, 1, n, dpos, g, bin_start.p, sorted_pos.p, sorted_atoms.p, cap, first, keys.p, num_neigh, head);
        launches += 1;
    }
    // Edge arrays (already sized) from the rows, and the edges by sender.
    void fill_rows(const Launcher& on, int n, const double* dpos, const int* types, const long long* first, size_t edges, int* neigh_indices, int* neigh_types, int* shifts,
                   double* xyz, double* r, double* node_forces, int* opposite, EvalHead* head, long& launches) {
        sorted_keys.resize(edges, on.stream);
        chain_launch(on, neigh_fill_kernel, dim3(row_blocks(n)), kNeighWarps * 32, 0, 1, n, dpos, types, g, cap, keys.p, first, sorted_keys.p, neigh_indices, neigh_types, shifts, xyz, r, node_forces);
        chain_launch(on, neigh_opposite_kernel, dim3(row_blocks(n)), 128, 0, 1, n, first, sorted_keys.p, opposite, head);
        launches += 2;
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) throw CudaError(std::string("neighbour list: ") + cudaGetErrorString(err));
    }
};

}  // namespace smx
