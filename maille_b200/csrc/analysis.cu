// analysis.cu -- symbolic analysis on the device (see analysis.cuh).
//
// Reference counterparts: Graph::from_elements (iterative.rs:38-76) builds the DOF graph from the
// elements, Csr::zeros (iterative.rs:91-114) lays out the lower profile, and FreeSystem::new
// (model.rs:1480-1492) adds every element matrix entry through Csr::add's binary search
// (iterative.rs:121-128; here the assembly walks each row's incident elements, kernels.cu). On nodes:
//  * graph: one warp per kept node collects the nodes of its incident elements in a hash set in shared
//    memory, twice (the counts, then the lists, sorted by counting smaller entries). The keys of all
//    element node pairs, sorted and made unique, gave the same lists in 3.2 ms against 1.0 (Tet10
//    40^3, 34.6 M keys); that way stays for graphs with a node of more neighbours than the set holds;
//  * pattern: the graph's rows in the new numbering, each sorted by its warp; the pairs' keys were
//    sorted a second time for it (6.1 ms with the scatter map of the assembly, against 1.7).
// Radix sorts, scans and selections are CUB's device primitives; the rest are the kernels below. Every
// step is a deterministic function of its inputs.

#include <atomic>
#include <climits>

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include "analysis.cuh"
#include "cuda_host.hpp"

namespace maille {

extern std::atomic<long long> g_kernel_launches;

namespace {

constexpr int kT = 256;
constexpr int kW = kT / 32;
constexpr int kSet = 512;       // hash set of a node's neighbours
constexpr int kSetMost = 384;   // neighbours it takes

inline unsigned grid_of(int64_t n) {
    const int64_t g = (n + kT - 1) / kT;
    return (unsigned)(g < 1 ? 1 : (g > (1 << 20) ? (1 << 20) : g));
}
inline unsigned warps_of(int64_t n) { return grid_of(n * 32); }
inline void counted(int n = 1) { g_kernel_launches.fetch_add(n, std::memory_order_relaxed); }

template <typename K>
__device__ __forceinline__ int64_t lower_bound_dev(const K* a, int64_t n, K key) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

#define GRID_STRIDE(t, n) \
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (n); t += (int64_t)gridDim.x * blockDim.x)
#define WARP_STRIDE(t, n)                                                                                     \
    for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < (n);                          \
         t += ((int64_t)gridDim.x * blockDim.x) >> 5)

__global__ void k_keep_flags(int dof, int64_t n, const uint8_t* __restrict__ fixed, int32_t* __restrict__ flag) {
    GRID_STRIDE(v, n + 1) {
        bool all = v < n;
        for (int d = 0; d < dof && v < n; ++d) all = all && fixed[dof * v + d] != 0;
        flag[v] = v < n && !all ? 1 : 0;
    }
}
// pos: exclusive sums of the flags
__global__ void k_keep(int64_t n, const int32_t* __restrict__ pos, int32_t* __restrict__ kept_of,
                       int32_t* __restrict__ kept) {
    GRID_STRIDE(v, n) {
        const bool keep = pos[v + 1] > pos[v];
        kept_of[v] = keep ? pos[v] : -1;
        if (keep) kept[pos[v]] = (int32_t)v;
    }
}

// The neighbours of kept node k in the warp's set (kSet entries, -1 free); their number, or -1 when the
// set is too small. Called by the whole warp.
__device__ __forceinline__ int neighbours(int npe, const int32_t* __restrict__ conn, const int64_t* __restrict__ inc_ptr,
                                          const int32_t* __restrict__ inc, const int32_t* __restrict__ kept_of,
                                          int32_t k, int32_t v, int32_t* set) {
    const int lane = threadIdx.x & 31;
    for (int q = lane; q < kSet; q += 32) set[q] = -1;
    __syncwarp();
    const int64_t q0 = inc_ptr[v], pairs = (inc_ptr[v + 1] - q0) * npe;
    int count = 0;
    for (int64_t t0 = 0; t0 < pairs; t0 += 32) {
        const int64_t t = t0 + lane;
        bool added = false;
        if (t < pairs) {
            const int32_t e = inc[q0 + t / npe] / npe;
            const int32_t w = kept_of[conn[(int64_t)e * npe + t % npe]];
            if (w >= 0 && w != k) {
                uint32_t h = ((uint32_t)w * 2654435761u) >> 23;  // multiplicative hashing, 9 bits
                for (int probe = 0; probe < kSet; ++probe) {
                    const int32_t old = atomicCAS(&set[h], -1, w);
                    added = old == -1;
                    if (old == -1 || old == w) break;
                    h = (h + 1) & (kSet - 1);
                }
            }
        }
        count += __popc(__ballot_sync(0xffffffffu, added));
        if (count > kSetMost) return -1;
    }
    __syncwarp();
    return count;
}

__global__ void __launch_bounds__(kT) k_graph_count(int npe, const int32_t* __restrict__ conn,
                                                    const int64_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                                                    const int32_t* __restrict__ kept_of, const int32_t* __restrict__ kept,
                                                    int32_t nk, int32_t* __restrict__ deg, int32_t* __restrict__ overflow) {
    __shared__ int32_t sets[kW][kSet];
    int32_t* set = sets[threadIdx.x >> 5];
    WARP_STRIDE(k, nk) {
        const int n = neighbours(npe, conn, inc_ptr, inc, kept_of, (int32_t)k, kept[k], set);
        if ((threadIdx.x & 31) == 0) {
            deg[k] = n < 0 ? 0 : n;
            if (n < 0) *overflow = 1;
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kT) k_graph_lists(int npe, const int32_t* __restrict__ conn,
                                                    const int64_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                                                    const int32_t* __restrict__ kept_of, const int32_t* __restrict__ kept,
                                                    int32_t nk, const int64_t* __restrict__ off, int32_t* __restrict__ adj) {
    __shared__ int32_t sets[kW][kSet], lists[kW][kSetMost];
    const int lane = threadIdx.x & 31;
    int32_t *set = sets[threadIdx.x >> 5], *list = lists[threadIdx.x >> 5];
    WARP_STRIDE(k, nk) {
        neighbours(npe, conn, inc_ptr, inc, kept_of, (int32_t)k, kept[k], set);
        int n = 0;
        for (int q = lane; q < kSet; q += 32) {
            const int32_t w = set[q];
            const uint32_t has = __ballot_sync(0xffffffffu, w >= 0);
            if (w >= 0) list[n + __popc(has & ((1u << lane) - 1u))] = w;
            n += __popc(has);
        }
        __syncwarp();
        for (int q = lane; q < n; q += 32) {
            const int32_t w = list[q];
            int smaller = 0;
            for (int p = 0; p < n; ++p) smaller += list[p] < w;
            adj[off[k] + smaller] = w;
        }
        __syncwarp();
    }
}

// *any = 1 when an element names a node twice
__global__ void k_repeats(int npe, int64_t ne, const int32_t* __restrict__ conn, int32_t* __restrict__ any) {
    GRID_STRIDE(e, ne) {
        const int32_t* c = conn + e * npe;
        bool twice = false;
        for (int a = 1; a < npe; ++a)
            for (int b = 0; b < a; ++b) twice = twice || c[a] == c[b];
        if (twice) *any = 1;
    }
}

// keys (I << sh) | J of every ordered pair of distinct kept nodes of an element, ~0 for the others
__global__ void k_graph_keys(int npe, int64_t ne, const int32_t* __restrict__ conn,
                             const int32_t* __restrict__ kept_of, int sh, uint64_t* __restrict__ keys) {
    const int64_t per = (int64_t)npe * (npe - 1);
    GRID_STRIDE(t, ne * per) {
        const int64_t e = t / per;
        const int rem = (int)(t - e * per);
        const int a = rem / (npe - 1), bi = rem % (npe - 1), b = bi < a ? bi : bi + 1;
        const int32_t I = kept_of[conn[e * npe + a]], J = kept_of[conn[e * npe + b]];
        keys[t] = (I < 0 || J < 0 || I == J) ? ~0ull : (((uint64_t)(uint32_t)I << sh) | (uint64_t)(uint32_t)J);
    }
}
__global__ void k_graph_csr(const uint64_t* __restrict__ keys, int64_t m, int32_t nk, int sh, int64_t* __restrict__ off,
                            int32_t* __restrict__ deg) {
    GRID_STRIDE(k, (int64_t)nk + 1) {
        const int64_t o = lower_bound_dev<uint64_t>(keys, m, (uint64_t)k << sh);
        off[k] = o;
        if (k < nk) deg[k] = (int32_t)(lower_bound_dev<uint64_t>(keys, m, (uint64_t)(k + 1) << sh) - o);
    }
}
__global__ void k_graph_adj(const uint64_t* __restrict__ keys, int64_t m, int sh, int32_t* __restrict__ adj) {
    GRID_STRIDE(p, m) adj[p] = (int32_t)(keys[p] & ((1ull << sh) - 1));
}

__global__ void k_rows(int dof, int32_t nk, const int32_t* __restrict__ order, const int32_t* __restrict__ kept,
                       const uint8_t* __restrict__ fixed, int32_t* __restrict__ perm, int32_t* __restrict__ rank,
                       uint8_t* __restrict__ fixmask) {
    GRID_STRIDE(r, nk) {
        const int32_t k = order[r], v = kept[k];
        perm[r] = v;
        rank[k] = (int32_t)r;
        if (dof == 3) {
            uint8_t m = 0;
            for (int d = 0; d < 3; ++d) m |= fixed[3 * (int64_t)v + d] ? (uint8_t)(1u << d) : (uint8_t)0;
            fixmask[r] = m;
        }
    }
}
__global__ void k_inv(int64_t n, const int32_t* __restrict__ kept_of, const int32_t* __restrict__ rank,
                      int32_t* __restrict__ inv) {
    GRID_STRIDE(v, n) inv[v] = kept_of[v] < 0 ? -1 : rank[kept_of[v]];
}
__global__ void k_ranks(int32_t nk, const int32_t* __restrict__ perm, const int32_t* __restrict__ kept_of,
                        int32_t* __restrict__ order, int32_t* __restrict__ rank) {
    GRID_STRIDE(r, nk) {
        const int32_t k = kept_of[perm[r]];
        order[r] = k;
        rank[k] = (int32_t)r;
    }
}

__global__ void k_row_len(int32_t nb, const int32_t* __restrict__ order, const int32_t* __restrict__ deg,
                          int64_t* __restrict__ len) {
    GRID_STRIDE(r, (int64_t)nb + 1) len[r] = r < nb ? deg[order[r]] + 1 : 0;
}
// columns of every row: its neighbours' rows and itself, ascending (each entry's place is the number of
// smaller ones)
__global__ void __launch_bounds__(kT) k_row_cols(int32_t nb, const int32_t* __restrict__ order,
                                                 const int32_t* __restrict__ rank, const int64_t* __restrict__ off,
                                                 const int32_t* __restrict__ adj, const int64_t* __restrict__ row_ptr,
                                                 int32_t* __restrict__ col, int64_t* __restrict__ diag) {
    __shared__ int32_t lists[kW][kSetMost + 1];
    const int lane = threadIdx.x & 31;
    int32_t* list = lists[threadIdx.x >> 5];
    WARP_STRIDE(r, nb) {
        const int64_t a = off[order[r]], rb = row_ptr[r];
        const int n = (int)(row_ptr[r + 1] - rb);
        const bool fits = n <= kSetMost + 1;
        auto entry = [&](int q) { return q + 1 < n ? rank[adj[a + q]] : (int32_t)r; };
        if (fits)
            for (int q = lane; q < n; q += 32) list[q] = entry(q);
        __syncwarp();
        for (int q = lane; q < n; q += 32) {
            const int32_t c = fits ? list[q] : entry(q);
            int smaller = 0;
            if (fits)
                for (int p = 0; p < n; ++p) smaller += list[p] < c;
            else
                for (int p = 0; p < n; ++p) smaller += entry(p) < c;
            col[rb + smaller] = c;
            if (c == (int32_t)r) diag[r] = rb + smaller;
        }
        __syncwarp();
    }
}
__global__ void __launch_bounds__(kT) k_row_tpos(int32_t nb, const int64_t* __restrict__ row_ptr,
                                                 const int32_t* __restrict__ col, int64_t* __restrict__ tpos) {
    const int lane = threadIdx.x & 31;
    WARP_STRIDE(r, nb)
        for (int64_t p = row_ptr[r] + lane; p < row_ptr[r + 1]; p += 32) {
            const int64_t cb = row_ptr[col[p]], ce = row_ptr[col[p] + 1];
            tpos[p] = cb + lower_bound_dev<int32_t>(col + cb, ce - cb, (int32_t)r);
        }
}

__global__ void k_boundary(int npe, int64_t ne, const int32_t* __restrict__ conn, const uint8_t* __restrict__ fixed,
                           uint8_t* __restrict__ eflag, uint8_t* __restrict__ nflag) {
    GRID_STRIDE(e, ne) {
        bool any = false;
        for (int a = 0; a < npe; ++a) {
            const int64_t v = conn[e * npe + a];
            any = any || fixed[3 * v] || fixed[3 * v + 1] || fixed[3 * v + 2];
        }
        eflag[e] = any;
        if (any)
            for (int a = 0; a < npe; ++a) nflag[conn[e * npe + a]] = 1;
    }
}
__global__ void k_elem_slot(int64_t n, const int32_t* __restrict__ belem, int32_t* __restrict__ slot) {
    GRID_STRIDE(k, n) slot[belem[k]] = (int32_t)k;
}
__global__ void k_orphans(int64_t n, const int64_t* __restrict__ inc_ptr, int32_t* __restrict__ any) {
    GRID_STRIDE(v, n) if (inc_ptr[v] == inc_ptr[v + 1]) *any = 1;
}

__global__ void k_fill_value(int64_t n, int32_t v, int32_t* __restrict__ a) {
    GRID_STRIDE(i, n) a[i] = v;
}

__device__ __forceinline__ int64_t part_start(SellKind kind, const int64_t* row_ptr, const int64_t* diag, int64_t i) {
    return kind == SELL_UPPER ? diag[i] + 1 : row_ptr[i];
}
__device__ __forceinline__ int64_t part_end(SellKind kind, const int64_t* row_ptr, const int64_t* diag, int64_t i) {
    return kind == SELL_LOWER ? diag[i] : row_ptr[i + 1];
}

__global__ void k_fill_sell(SellKind kind, int32_t lpr, int64_t nrow_slots, const int32_t* __restrict__ rowid,
                            const int64_t* __restrict__ off, const int64_t* __restrict__ row_ptr,
                            const int32_t* __restrict__ col, const int64_t* __restrict__ diag,
                            int32_t* __restrict__ slot_col, int32_t* __restrict__ slot_src) {
    const int S = 32 / lpr, per_step = 4 * lpr;
    GRID_STRIDE(t, nrow_slots) {
        const int32_t i = rowid[t];
        if (i < 0) continue;
        const int64_t s = t / S;
        const int r = (int)(t - s * S);
        const int64_t b0 = part_start(kind, row_ptr, diag, i), b1 = part_end(kind, row_ptr, diag, i);
        for (int64_t p = b0; p < b1; ++p) {
            const int64_t b = p - b0, st = b / per_step, rem = b % per_step;
            const int64_t slot = (off[s] + st) * 128 + 4 * (r * lpr + rem / 4) + rem % 4;
            slot_col[slot] = col[p];
            slot_src[slot] = (int32_t)p;
        }
    }
}

__global__ void k_fill_psell(SellKind kind, int64_t nrows, const int32_t* __restrict__ rows,
                             const int64_t* __restrict__ rstart, const int64_t* __restrict__ row_ptr,
                             const int32_t* __restrict__ col, const int64_t* __restrict__ diag,
                             int32_t* __restrict__ slot_col, int32_t* __restrict__ slot_src) {
    GRID_STRIDE(k, nrows) {
        const int32_t i = rows[k];
        const int64_t b0 = part_start(kind, row_ptr, diag, i), b1 = part_end(kind, row_ptr, diag, i);
        for (int64_t p = b0; p < b1; ++p) {
            slot_col[rstart[k] + (p - b0)] = col[p];
            slot_src[rstart[k] + (p - b0)] = (int32_t)p;
        }
    }
}

__global__ void k_fill_bsell(SellKind kind, int rows, int sub, int64_t nrow_slots, const int32_t* __restrict__ rowid,
                             const int64_t* __restrict__ off, const int64_t* __restrict__ row_ptr,
                             const int32_t* __restrict__ col, const int64_t* __restrict__ diag,
                             int32_t* __restrict__ slot_col, int32_t* __restrict__ slot_src) {
    const int per_step = 4 * sub, slots = rows * per_step;
    GRID_STRIDE(t, nrow_slots) {
        const int32_t i = rowid[t];
        if (i < 0) continue;
        const int64_t s = t / rows;
        const int r = (int)(t - s * rows);
        const int64_t b0 = part_start(kind, row_ptr, diag, i), b1 = part_end(kind, row_ptr, diag, i);
        for (int64_t p = b0; p < b1; ++p) {
            const int64_t b = p - b0, st = b / per_step, rem = b % per_step;
            const int64_t slot = (off[s] + st) * slots + 4 * (r * sub + rem / 4) + rem % 4;
            slot_col[slot] = col[p];
            slot_src[slot] = (int32_t)p;
        }
    }
}

}  // namespace

int32_t gpu_keep(int dof, int64_t n_nodes, const uint8_t* fixed, cudaStream_t st, int32_t* kept_of, int32_t* kept) {
    Scratch tmp(st);
    int32_t *flag = tmp.take<int32_t>(n_nodes + 1), *pos = tmp.take<int32_t>(n_nodes + 1);
    k_keep_flags<<<grid_of(n_nodes + 1), kT, 0, st>>>(dof, n_nodes, fixed, flag);
    CK(cudaGetLastError());
    size_t bytes = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, bytes, flag, pos, (int)(n_nodes + 1), st));
    CK(cub::DeviceScan::ExclusiveSum(tmp.take<unsigned char>(bytes), bytes, flag, pos, (int)(n_nodes + 1), st));
    k_keep<<<grid_of(n_nodes), kT, 0, st>>>(n_nodes, pos, kept_of, kept);
    CK(cudaGetLastError());
    counted(4);
    int32_t nk = 0;
    CK(cudaMemcpyAsync(&nk, pos + n_nodes, sizeof(nk), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return nk;
}

void gpu_graph(int npe, int64_t n_elems, const int32_t* conn, const int64_t* inc_ptr, const int32_t* inc,
               const int32_t* kept_of, const int32_t* kept, int32_t nk, cudaStream_t st, GraphDev& out) {
    if (nk <= 0) throw CudaFailure{"no kept node to order"};
    const int64_t nkeys = n_elems * npe * (npe - 1);
    if (nkeys >= INT_MAX || nkeys <= 0) throw CudaFailure{"mesh size outside the device ordering's range"};
    out.nk = nk;
    out.st = st;
    out.off = dalloc<int64_t>((size_t)nk + 1);
    out.deg = dalloc<int32_t>((size_t)nk + 1);
    Scratch tmp(st);
    int32_t* overflow = tmp.take<int32_t>(2);  // [1]: an element names a node twice
    CK(cudaMemsetAsync(overflow, 0, 2 * sizeof(int32_t), st));
    CK(cudaMemsetAsync(out.deg + nk, 0, sizeof(int32_t), st));
    k_graph_count<<<warps_of(nk), kT, 0, st>>>(npe, conn, inc_ptr, inc, kept_of, kept, nk, out.deg, overflow);
    k_repeats<<<grid_of(n_elems), kT, 0, st>>>(npe, n_elems, conn, overflow + 1);
    CK(cudaGetLastError());
    size_t bytes = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, bytes, out.deg, out.off, (int)(nk + 1), st));
    CK(cub::DeviceScan::ExclusiveSum(tmp.take<unsigned char>(bytes), bytes, out.deg, out.off, (int)(nk + 1), st));
    counted(4);
    int32_t flags[2] = {0, 0};
    CK(cudaMemcpyAsync(flags, overflow, sizeof(flags), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&out.m, out.off + nk, sizeof(out.m), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    out.repeats = flags[1] != 0;
    if (!flags[0]) {
        out.adj = dalloc<int32_t>((size_t)std::max<int64_t>(1, out.m));
        k_graph_lists<<<warps_of(nk), kT, 0, st>>>(npe, conn, inc_ptr, inc, kept_of, kept, nk, out.off, out.adj);
        CK(cudaGetLastError());
        counted(1);
        return;
    }
    // a node of more than kSetMost neighbours: sort the pairs' keys
    int sh = 1;
    while ((int64_t(1) << sh) <= (int64_t)nk) ++sh;  // nk < 2^sh: valid keys stay below ~0
    uint64_t *ka = tmp.take<uint64_t>(nkeys), *kb = tmp.take<uint64_t>(nkeys), *uk = tmp.take<uint64_t>(nkeys);
    int* nsel = tmp.take<int>(1);
    k_graph_keys<<<grid_of(nkeys), kT, 0, st>>>(npe, n_elems, conn, kept_of, sh, ka);
    CK(cudaGetLastError());
    cub::DoubleBuffer<uint64_t> db(ka, kb);
    size_t b0 = 0, b1 = 0;
    CK(cub::DeviceRadixSort::SortKeys(nullptr, b0, db, (int)nkeys, 0, 2 * sh, st));
    CK(cub::DeviceSelect::Unique(nullptr, b1, db.Current(), uk, nsel, (int)nkeys, st));
    unsigned char* t = tmp.take<unsigned char>(std::max(b0, b1));
    CK(cub::DeviceRadixSort::SortKeys(t, b0, db, (int)nkeys, 0, 2 * sh, st));
    CK(cub::DeviceSelect::Unique(t, b1, db.Current(), uk, nsel, (int)nkeys, st));
    int n = 0;
    CK(cudaMemcpyAsync(&n, nsel, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    uint64_t last = 0;
    if (n > 0) CK(cudaMemcpy(&last, uk + (n - 1), sizeof(uint64_t), cudaMemcpyDeviceToHost));
    out.m = (n > 0 && last == ~0ull) ? n - 1 : n;
    out.adj = dalloc<int32_t>((size_t)std::max<int64_t>(1, out.m));
    k_graph_csr<<<grid_of((int64_t)nk + 1), kT, 0, st>>>(uk, out.m, nk, sh, out.off, out.deg);
    k_graph_adj<<<grid_of(std::max<int64_t>(1, out.m)), kT, 0, st>>>(uk, out.m, sh, out.adj);
    CK(cudaGetLastError());
    counted(5);
}

void gpu_rows(int dof, int32_t nk, int64_t n_nodes, const int32_t* order, const int32_t* kept, const int32_t* kept_of,
              const uint8_t* fixed, cudaStream_t st, int32_t* perm, int32_t* inv, int32_t* rank, uint8_t* fixmask) {
    counted(2);
    k_rows<<<grid_of(nk), kT, 0, st>>>(dof, nk, order, kept, fixed, perm, rank, fixmask);
    k_inv<<<grid_of(n_nodes), kT, 0, st>>>(n_nodes, kept_of, rank, inv);
    CK(cudaGetLastError());
}

void gpu_ranks(int32_t nk, const int32_t* perm, const int32_t* kept_of, cudaStream_t st, int32_t* order, int32_t* rank) {
    counted();
    k_ranks<<<grid_of(nk), kT, 0, st>>>(nk, perm, kept_of, order, rank);
    CK(cudaGetLastError());
}

void gpu_pattern(const GraphDev& g, const int32_t* order, const int32_t* rank, cudaStream_t st, PatternDev& out,
                 std::vector<int64_t>& h_row_ptr, std::vector<int64_t>& h_diag) {
    const int32_t nb = g.nk;
    out = PatternDev{};
    out.blocks = g.m + nb;
    if (out.blocks >= (int64_t(1) << 31)) throw CudaFailure{"pattern too large for 32-bit block positions"};
    Scratch tmp(st);
    int64_t* len = tmp.take<int64_t>((size_t)nb + 1);
    size_t bytes = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, bytes, len, len, nb + 1, st));
    unsigned char* t = tmp.take<unsigned char>(bytes);
    out.row_ptr = dalloc<int64_t>((size_t)nb + 1);
    out.diag = dalloc<int64_t>(nb);
    out.col = dalloc<int32_t>(out.blocks);
    out.tpos = dalloc<int64_t>(out.blocks);
    k_row_len<<<grid_of((int64_t)nb + 1), kT, 0, st>>>(nb, order, g.deg, len);
    CK(cub::DeviceScan::ExclusiveSum(t, bytes, len, out.row_ptr, nb + 1, st));
    k_row_cols<<<warps_of(nb), kT, 0, st>>>(nb, order, rank, g.off, g.adj, out.row_ptr, out.col, out.diag);
    CK(cudaGetLastError());
    h_row_ptr.resize((size_t)nb + 1);
    h_diag.resize((size_t)nb);
    CK(cudaMemcpyAsync(h_row_ptr.data(), out.row_ptr, ((size_t)nb + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(h_diag.data(), out.diag, (size_t)nb * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    k_row_tpos<<<warps_of(nb), kT, 0, st>>>(nb, out.row_ptr, out.col, out.tpos);
    CK(cudaGetLastError());
    counted(5);
}

void gpu_boundary(int npe, int64_t n_elems, const int32_t* conn, int64_t n_nodes, const uint8_t* fixed,
                  const int64_t* inc_ptr, cudaStream_t st, BoundaryDev& out) {
    Scratch tmp(st);
    uint8_t *eflag = tmp.take<uint8_t>(n_elems), *nflag = tmp.take<uint8_t>(n_nodes);
    int32_t* count = tmp.take<int32_t>(3);
    out.belem = dalloc<int32_t>(n_elems);
    out.bnodes = dalloc<int32_t>(n_nodes);
    out.elem_slot = dalloc<int32_t>(n_elems);
    CK(cudaMemsetAsync(nflag, 0, n_nodes, st));
    CK(cudaMemsetAsync(count, 0, 3 * sizeof(int32_t), st));
    CK(cudaMemsetAsync(out.elem_slot, 0xFF, n_elems * sizeof(int32_t), st));
    k_boundary<<<grid_of(n_elems), kT, 0, st>>>(npe, n_elems, conn, fixed, eflag, nflag);
    k_orphans<<<grid_of(n_nodes), kT, 0, st>>>(n_nodes, inc_ptr, count + 2);
    CK(cudaGetLastError());
    thrust::counting_iterator<int32_t> ids(0);
    size_t b0 = 0, b1 = 0;
    CK(cub::DeviceSelect::Flagged(nullptr, b0, ids, eflag, out.belem, count, (int)n_elems, st));
    CK(cub::DeviceSelect::Flagged(nullptr, b1, ids, nflag, out.bnodes, count + 1, (int)n_nodes, st));
    unsigned char* t = tmp.take<unsigned char>(std::max(b0, b1));
    CK(cub::DeviceSelect::Flagged(t, b0, ids, eflag, out.belem, count, (int)n_elems, st));
    CK(cub::DeviceSelect::Flagged(t, b1, ids, nflag, out.bnodes, count + 1, (int)n_nodes, st));
    int32_t h[3] = {0, 0, 0};
    CK(cudaMemcpyAsync(h, count, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    out.nbelem = h[0];
    out.nbnodes = h[1];
    out.orphans = h[2] != 0;
    if (out.nbelem) k_elem_slot<<<grid_of(out.nbelem), kT, 0, st>>>(out.nbelem, out.belem, out.elem_slot);
    CK(cudaGetLastError());
    counted(7);
}

void fill_sell(SellKind kind, int32_t lpr, int32_t nslices, int64_t steps, const int32_t* rowid,
               const int64_t* off, const int64_t* row_ptr, const int32_t* col, const int64_t* diag,
               int32_t nb, int32_t* slot_col, int32_t* slot_src, cudaStream_t st) {
    const int64_t nslots = steps * 128, nrs = (int64_t)nslices * (32 / lpr);
    counted(2);
    k_fill_value<<<grid_of(nslots), kT, 0, st>>>(nslots, nb, slot_col);
    CK(cudaMemsetAsync(slot_src, 0xFF, (size_t)nslots * sizeof(int32_t), st));
    k_fill_sell<<<grid_of(nrs), kT, 0, st>>>(kind, lpr, nrs, rowid, off, row_ptr, col, diag, slot_col, slot_src);
    CK(cudaGetLastError());
}

void fill_psell(SellKind kind, int64_t nrows, int64_t steps, const int32_t* rows, const int64_t* rstart,
                const int64_t* row_ptr, const int32_t* col, const int64_t* diag, int32_t nb,
                int32_t* slot_col, int32_t* slot_src, cudaStream_t st) {
    const int64_t nslots = steps * 128;
    counted(2);
    k_fill_value<<<grid_of(nslots), kT, 0, st>>>(nslots, nb, slot_col);
    CK(cudaMemsetAsync(slot_src, 0xFF, (size_t)nslots * sizeof(int32_t), st));
    k_fill_psell<<<grid_of(nrows), kT, 0, st>>>(kind, nrows, rows, rstart, row_ptr, col, diag, slot_col, slot_src);
    CK(cudaGetLastError());
}

void fill_bsell(SellKind kind, int rows, int sub, int32_t nslices, int64_t steps, const int32_t* rowid,
                const int64_t* off, const int64_t* row_ptr, const int32_t* col, const int64_t* diag, int32_t nb,
                int32_t* slot_col, int32_t* slot_src, cudaStream_t st) {
    const int64_t nslots = steps * rows * sub * 4, nrs = (int64_t)nslices * rows;
    counted(2);
    k_fill_value<<<grid_of(nslots), kT, 0, st>>>(nslots, nb, slot_col);
    CK(cudaMemsetAsync(slot_src, 0xFF, (size_t)nslots * sizeof(int32_t), st));
    k_fill_bsell<<<grid_of(nrs), kT, 0, st>>>(kind, rows, sub, nrs, rowid, off, row_ptr, col, diag, slot_col, slot_src);
    CK(cudaGetLastError());
}

}  // namespace maille
