// coarse.cu -- plan and numeric set-up of the coarse correction (see coarse.cuh).
//
// Plan, once per pattern: every row's cell and place in it, the rows in cell order cut into chunks
// (the restriction's units), and the blocks of K sorted by their pair of cells and cut into chunks
// (the Galerkin product's units).
// Numeric set-up, once per factorisation:
//  * k_pairs: one warp per chunk of blocks of one cell pair sums w_a(i) w_b(j) K_ij for the 64
//    corner pairs (a, b), two pairs a lane, into the chunk's own slots;
//  * k_pair_sums, k_dense: every entry of E sums the slots of the cell pairs that touch it, in order;
//  * k_panel, k_trail: E^-1 by block symmetric sweeps (Beaton's sweep operator, 64 unknowns a
//    step, lower tiles only), every update a square by the tile's Cholesky factor: m^3 flops, no pivoting
//    (E with its ridge, kRidge64, is positive definite).
//    An unknown whose pivot falls below a tenth of the ridge (a coarse node without support) leaves the
//    space: its row and column of the inverse are zero;
//  * k_mirror: -A, both triangles, in the PCG's precision.
// No floating-point atomics: repeated set-ups give the same bits.

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstring>

#include <cub/cub.cuh>

#include "coarse.cuh"
#include "coarse_dev.cuh"
#include "cuda_host.hpp"

namespace maille {

extern std::atomic<long long> g_kernel_launches;

namespace {

constexpr int kT = 256;
constexpr int kTile = 64;        // unknowns a sweep step; tile side
constexpr int kRowChunk = 256;   // rows a restriction chunk, one row a lane at a time
constexpr int kBatchChunk = 64;  // rows a chunk of a batch, whose warp takes them one after the other
constexpr int kPairChunk = 256;  // blocks a Galerkin chunk
constexpr int kPairWarps = 4;    // warps a block of k_pairs
// E + ridge diag(E) is what is inverted. Where a part has fewer layers of nodes than the grid has lines, or
// touches a cell with a corner only, hats depend on one another and E is singular; its null pivots are
// rounding times the square of the multipliers (up to 1e-9), no threshold tells them from soft modes (a bar
// of 331:1: 1e-10), and one taken for a pivot made the correction indefinite: a bent strip of 4x1x19
// cells (60 of 180 unknowns dependent) did not converge in 10000 iterations where IC(0) alone takes 105, and
// takes 26 with the ridge. 1e-9 stays far above what the rounding leaves of it and below every soft mode
// that matters (bars of 120:1 and 331:1 take 151 and 509 iterations with and without it). Rounded to FP32 an
// inverse is definite only while its largest entries stay below 1 / 6e-8 of its smallest modes': 1e-5
// (3x7x6 cells of 0.44:1:0.37, mixed, IC(0) alone / without / with: 1013 / not in 10000 / 100 iterations; bars
// of 10:1, plates, shells and cubes the same). Over 260 random parts (1 to 64 cells a side, graded, bent,
// twisted, moduli over three decades) the correction with both converges wherever IC(0) alone does, in
// 0.38 (FP64) and 0.34 (mixed) of its iterations, never in more than 1.3 of them.
constexpr double kRidge64 = 1e-9, kRidge32 = 1e-5;
constexpr double kDrop = 0.1;  // a pivot below this part of its ridge is rounding
// A row this close to a grid plane, relative to the cell, lies on it: else the hats of a plane that nodes miss
// by a rounding carry weights of 1e-16, depend on the others, and cost the FP32 inverse its accuracy (a
// graded plate of one cell clamped on its face: 784 iterations against 41).
constexpr double kSnap = 1e-9;
constexpr int64_t kMinRows = 128;

inline unsigned grid_of(int64_t n) {
    const int64_t g = (n + kT - 1) / kT;
    return (unsigned)(g < 1 ? 1 : (g > (1 << 20) ? (1 << 20) : g));
}
inline void counted(int n = 1) { g_kernel_launches.fetch_add(n, std::memory_order_relaxed); }

#define GRID_STRIDE(t, n) \
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (n); t += (int64_t)gridDim.x * blockDim.x)

// ext: the largest keys of -x, -y, -z, x, y, z over the nodes of an element, in keys (an order-preserving
// image of the doubles, complemented for the minima; all zero before)
__global__ void __launch_bounds__(kT) k_box(int64_t n, const double* __restrict__ xyz, const int64_t* __restrict__ inc_ptr,
                                            unsigned long long* __restrict__ ext) {
    unsigned long long m[6] = {};
    GRID_STRIDE(v, n) {
        if (inc_ptr[v] == inc_ptr[v + 1]) continue;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const unsigned long long bits = (unsigned long long)__double_as_longlong(xyz[3 * v + a]);
            const unsigned long long key = bits >> 63 ? ~bits : bits | (1ull << 63);
            m[a] = max(m[a], ~key);
            m[3 + a] = max(m[3 + a], key);
        }
    }
#pragma unroll
    for (int a = 0; a < 6; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m[a] = max(m[a], __shfl_xor_sync(0xffffffffu, m[a], o));
        if ((threadIdx.x & 31) == 0) atomicMax(&ext[a], m[a]);
    }
}

// cell, fractions and code of every row
__global__ void k_place(int32_t nb, const double* __restrict__ xyz, const int32_t* __restrict__ perm,
                        const uint8_t* __restrict__ fixmask, const int32_t* __restrict__ inst,
                        const CoarseGrid* __restrict__ grids, double4* __restrict__ pos, int32_t* __restrict__ cell,
                        int32_t* __restrict__ rows) {
    GRID_STRIDE(i, nb) {
        const CoarseGrid& g = grids[inst ? inst[i] : 0];
        double f[3];
        int32_t c[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double t = fmin(fmax((xyz[3 * (int64_t)perm[i] + a] - g.lo[a]) * g.inv_h[a], 0.0), (double)g.k[a]);
            c[a] = min((int32_t)t, g.k[a] - 1);
            f[a] = t - (double)c[a];
            if (f[a] < kSnap) f[a] = 0.0;
            if (f[a] > 1.0 - kSnap) f[a] = 1.0;
        }
        const uint32_t base = (uint32_t)(c[0] + (g.k[0] + 1) * (c[1] + (g.k[1] + 1) * c[2]));
        const uint32_t mask = fixmask ? (uint32_t)fixmask[i] & 7u : 0u;
        pos[i] = make_double4(f[0], f[1], f[2], __longlong_as_double((long long)(base | (mask << 28))));
        cell[i] = g.cell0 + c[0] + g.k[0] * (c[1] + g.k[1] * c[2]);
        rows[i] = (int32_t)i;
    }
}

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
    static __device__ float4 make(const double4& p, uint32_t code) {
        return make_float4((float)p.x, (float)p.y, (float)p.z, __uint_as_float(code));
    }
    using type = float4;
};
template <>
struct Vec4<double> {
    static __device__ double4 make(const double4& p, uint32_t code) {
        return make_double4(p.x, p.y, p.z, __longlong_as_double((long long)code));
    }
    using type = double4;
};

template <typename T>
__global__ void k_row_weights(int32_t nb, const double4* __restrict__ pos, const int32_t* __restrict__ order,
                              typename Vec4<T>::type* __restrict__ w, typename Vec4<T>::type* __restrict__ ws) {
    GRID_STRIDE(i, nb) {
        const double4 p = pos[i];
        w[i] = Vec4<T>::make(p, (uint32_t)__double_as_longlong(p.w));
        const int32_t r = order[i];
        ws[i] = Vec4<T>::make(pos[r], (uint32_t)r | ((uint32_t)__double_as_longlong(pos[r].w) >> 28 << 29));
    }
}

template <typename K>
__device__ __forceinline__ int64_t lower_bound_dev(const K* a, int64_t n, K key) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

__global__ void k_cell_ptr(const int32_t* __restrict__ sorted, int32_t nb, int32_t ncells, int32_t* __restrict__ ptr) {
    GRID_STRIDE(c, (int64_t)ncells + 1) ptr[c] = (int32_t)lower_bound_dev<int32_t>(sorted, nb, (int32_t)c);
}

// keys (cell of the row << sh) | cell of the column of the blocks whose row's cell is not below the
// column's, ~0 for the others (their transposes stand for them); one warp per row
__global__ void k_pair_cells(int32_t nb, const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                             const int32_t* __restrict__ cell, int sh, uint64_t* __restrict__ key,
                             int32_t* __restrict__ bpos, int32_t* __restrict__ brow) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = w0; i < nb; i += nw) {
        const uint64_t ci = (uint64_t)cell[i];
        for (int64_t p = row_ptr[i] + lane; p < row_ptr[i + 1]; p += 32) {
            const uint64_t cj = (uint64_t)cell[col[p]];
            key[p] = ci >= cj ? (ci << sh) | cj : ~0ull;
            bpos[p] = (int32_t)p;
            brow[p] = (int32_t)i;
        }
    }
}

__global__ void k_sorted_rc(int64_t n, const int32_t* __restrict__ bpos, const int32_t* __restrict__ brow,
                            const int32_t* __restrict__ col, int32_t* __restrict__ srow, int32_t* __restrict__ scol) {
    GRID_STRIDE(t, n) {
        const int32_t p = bpos[t];
        srow[t] = brow[p];
        scol[t] = col[p];
    }
}

__global__ void k_table(int32_t nseg, const int64_t* __restrict__ at, int32_t* __restrict__ table) {
    GRID_STRIDE(s, nseg) table[at[s]] = (int32_t)s;
}

// One warp per chunk: 32 blocks at a time are brought to shared memory (each lane its block's values,
// masked, and the 8 + 8 hat weights of its row and column), then every lane adds all 32 to its two
// corner pairs (a, b), (a, b + 4). Bound by the FP64 pipe: 2 DOF^2 + 2 operations a lane and block.
template <int DOF>
__global__ void __launch_bounds__(kPairWarps * 32) k_pairs(int32_t nchunks, const int2* __restrict__ chunk,
                                                           const int32_t* __restrict__ bpos,
                                                           const int32_t* __restrict__ brow,
                                                           const int32_t* __restrict__ bcol,
                                                           const double4* __restrict__ pos,
                                                           const double* __restrict__ vals, double* __restrict__ part) {
    constexpr int D2 = DOF * DOF, S = 16 + D2 + (D2 & 1 ? 0 : 1);  // an odd stride: 32 lanes, 32 banks pairs
    __shared__ double sh[kPairWarps][32][S];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int a = lane & 7, b = lane >> 3;
    for (int32_t k = blockIdx.x * kPairWarps + wp; k < nchunks; k += gridDim.x * kPairWarps) {
        const int2 range = chunk[k];
        double s0[D2], s1[D2];
#pragma unroll
        for (int q = 0; q < D2; ++q) s0[q] = s1[q] = 0.0;
        for (int32_t t0 = range.x; t0 < range.y; t0 += 32) {
            const int32_t n = min(32, range.y - t0);
            __syncwarp();
            if (lane < n) {
                const int64_t p = bpos[t0 + lane];
                const double4 pi = pos[brow[t0 + lane]], pj = pos[bcol[t0 + lane]];
                double* v = sh[wp][lane];
                double f[3] = {pi.x, pi.y, pi.z}, w[8];
                coarse_weights(f, w);
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = w[q];
                f[0] = pj.x; f[1] = pj.y; f[2] = pj.z;
                coarse_weights(f, w);
#pragma unroll
                for (int q = 0; q < 8; ++q) v[8 + q] = w[q];
                const uint32_t mi = (uint32_t)__double_as_longlong(pi.w) >> 28, mj = (uint32_t)__double_as_longlong(pj.w) >> 28;
#pragma unroll
                for (int q = 0; q < D2; ++q) {
                    const bool fixed = ((mi >> (q / DOF)) | (mj >> (q % DOF))) & 1u;
                    v[16 + q] = fixed ? 0.0 : vals[p * D2 + q];
                }
            }
            __syncwarp();
            for (int32_t l = 0; l < n; ++l) {
                const double* v = sh[wp][l];
                const double wa = v[a], c0 = wa * v[8 + b], c1 = wa * v[12 + b];
#pragma unroll
                for (int q = 0; q < D2; ++q) {
                    s0[q] += c0 * v[16 + q];
                    s1[q] += c1 * v[16 + q];
                }
            }
        }
        // slot (a, b) at a + 8 b: lane, and lane + 32
#pragma unroll
        for (int q = 0; q < D2; ++q) {
            part[((int64_t)k * D2 + q) * 64 + lane] = s0[q];
            part[((int64_t)k * D2 + q) * 64 + 32 + lane] = s1[q];
        }
    }
}

// The chunks of every cell pair, summed in order into its first one.
template <int DOF>
__global__ void k_pair_sums(int32_t nseg, const int32_t* __restrict__ schunk_ptr, double* __restrict__ part) {
    constexpr int64_t N = 64 * DOF * DOF;
    GRID_STRIDE(t, nseg * N) {
        const int64_t seg = t / N, v = t - seg * N;
        const int32_t k0 = schunk_ptr[seg], k1 = schunk_ptr[seg + 1];
        if (k1 - k0 < 2) continue;
        double s = part[k0 * N + v];
        for (int32_t k = k0 + 1; k < k1; ++k) s += part[k * N + v];
        part[k0 * N + v] = s;
    }
}

// A (lower tiles, zero before) = E with its ridge and ones on the padded diagonal, diag = its diagonal: one thread per
// coarse node u, node v <= u within reach (`span`: cells that a block of K reaches across at most)
// and entry of their block.
template <int DOF>
__global__ void k_dense(const CoarseGrid* __restrict__ grids, const int32_t* __restrict__ table,
                        const int32_t* __restrict__ schunk_ptr, const double* __restrict__ part, double* __restrict__ A,
                        double* __restrict__ diag, int64_t diag_stride, double ridge) {
    constexpr int D2 = DOF * DOF;
    const CoarseGrid g = grids[blockIdx.y];
    const int32_t nx = g.k[0] + 1, ny = g.k[1] + 1, nz = g.k[2] + 1, nn = nx * ny * nz;
    const int32_t nc = g.k[0] * g.k[1] * g.k[2], reach = g.span + 1;
    const int32_t wx = min(reach, g.k[0]), wy = min(reach, g.k[1]), wz = min(reach, g.k[2]);
    const int32_t sx = 2 * wx + 1, sy = 2 * wy + 1, window = sx * sy * (2 * wz + 1);
    double* Ai = A + g.dense0;
    double* di = diag + blockIdx.y * diag_stride;
    const int32_t* tab = table + g.tab0;
    GRID_STRIDE(t, (int64_t)nn * window * D2) {
        const int32_t u = (int32_t)(t / (window * D2)), rest = (int32_t)(t - (int64_t)u * window * D2);
        const int32_t q = rest / window, o = rest - q * window;
        const int32_t ux = u % nx, uy = (u / nx) % ny, uz = u / (nx * ny);
        const int32_t vx = ux + o % sx - wx, vy = uy + o / sx % sy - wy, vz = uz + o / (sx * sy) - wz;
        if (vx < 0 || vy < 0 || vz < 0 || vx >= nx || vy >= ny || vz >= nz) continue;
        const int32_t v = vx + nx * (vy + ny * vz);
        if (v > u) continue;
        double s = 0.0;
        for (int a = 0; a < 8; ++a) {
            const int32_t cx = ux - (a & 1), cy = uy - ((a >> 1) & 1), cz = uz - (a >> 2);
            if (cx < 0 || cy < 0 || cz < 0 || cx >= g.k[0] || cy >= g.k[1] || cz >= g.k[2]) continue;
            const int32_t cu = cx + g.k[0] * (cy + g.k[1] * cz);
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const int32_t ex = vx - (b & 1), ey = vy - ((b >> 1) & 1), ez = vz - (b >> 2);
                if (ex < 0 || ey < 0 || ez < 0 || ex >= g.k[0] || ey >= g.k[1] || ez >= g.k[2]) continue;
                const int32_t cv = ex + g.k[0] * (ey + g.k[1] * ez);
                const bool direct = cu >= cv;
                const int32_t seg = direct ? tab[(int64_t)cu * nc + cv] : tab[(int64_t)cv * nc + cu];
                if (seg < 0) continue;
                const int slot = direct ? a + 8 * b : b + 8 * a;
                const int from = direct ? q : (q % DOF) * DOF + q / DOF;
                s += part[((int64_t)schunk_ptr[seg] * D2 + from) * 64 + slot];
            }
        }
        const int64_t r = (int64_t)DOF * u + q / DOF, c = (int64_t)DOF * v + q % DOF;
        if (r == c) di[r] = s *= 1.0 + ridge;
        Ai[r * g.ld + c] = s;
    }
    // the padding of the last tiles: an identity
    GRID_STRIDE(t, g.ld - g.m) {
        Ai[(g.m + t) * (g.ld + 1)] = 1.0;
        di[g.m + t] = 1.0;
    }
}

// The inverse Cholesky factor X = L^-1 of the 64 x 64 tile L L^T held by 256 threads, 4 x 4 entries a[][] each
// (thread (ty, tx): rows 4 ty .., columns 4 tx ..); x[][] the same entries of X. Four pivots at a time: the
// thread on the diagonal factors its own 4 x 4 entries, its row of threads broadcasts its rows through
// shared memory and takes its rows of X, the block forms the columns of L below, and the threads below
// take the rank-4 updates of the tile and of X. 16 such steps instead of 64 pivots: one pivot at a
// time took 105 us a tile, with a division, a load of its limit and a barrier on every pivot's path. An
// unknown whose pivot falls to its limit (kDrop) is dropped: a zero row and column of X.
struct TileMem {
    double rows[4][kTile], x[4][kTile], u[kTile][4], M[16], limit[kTile];
};
__device__ __forceinline__ void factor_tile(double a[4][4], double x[4][4], TileMem& m) {
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) x[q][p] = tx == ty && q == p ? 1.0 : 0.0;
    for (int b = 0; b < kTile / 4; ++b) {
        if (ty == b) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int p = 0; p < 4; ++p) m.rows[q][4 * tx + p] = a[q][p];
            if (tx == b) {  // M = L_bb^-1
                double r[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    r[t] = a[t][t] > m.limit[4 * b + t] ? rsqrt(a[t][t]) : 0.0;
#pragma unroll
                    for (int q = t + 1; q < 4; ++q) a[q][t] *= r[t];
#pragma unroll
                    for (int q = t + 1; q < 4; ++q)
#pragma unroll
                        for (int p = t + 1; p <= q; ++p) a[q][p] -= a[q][t] * a[p][t];
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    double c[4] = {0.0, 0.0, 0.0, 0.0};
                    c[t] = r[t];
#pragma unroll
                    for (int q = t + 1; q < 4; ++q) {
                        double d = 0.0;
#pragma unroll
                        for (int k = t; k < q; ++k) d -= a[q][k] * c[k];
                        c[q] = d * r[q];
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) m.M[4 * q + t] = c[q];
                }
            }
        }
        __syncthreads();
        if (ty == b && tx <= b)  // X is lower triangular
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const double v[4] = {x[0][p], x[1][p], x[2][p], x[3][p]};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    double d = 0.0;
#pragma unroll
                    for (int k = 0; k <= q; ++k) d += m.M[4 * q + k] * v[k];
                    m.x[q][4 * tx + p] = x[q][p] = d;
                }
            }
        {  // u = the columns of L, one entry a thread
            const int r = tid >> 2, t = tid & 3;
            double d = 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) d += m.rows[k][r] * m.M[4 * t + k];
            m.u[r][t] = d;
        }
        __syncthreads();
        if (ty > b) {
            double l[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int t = 0; t < 4; ++t) l[q][t] = m.u[4 * ty + q][t];
            if (tx > b) {
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const double w = m.u[4 * tx + p][t];
#pragma unroll
                        for (int q = 0; q < 4; ++q) a[q][p] -= l[q][t] * w;
                    }
            } else {
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const double w = m.x[t][4 * tx + p];
#pragma unroll
                        for (int q = 0; q < 4; ++q) x[q][p] -= l[q][t] * w;
                    }
            }
        }
    }
}

// v[q][p] = sum_t P[t][4 ty + q] W[t][r_p], t0 <= t < t1, for this thread's columns 4 ty .. and rows 2 tx,
// 2 tx + 1, 32 + ..
constexpr int kPanelStride = kTile + 2;
__device__ __forceinline__ void panel_product(const double* P, const double* W, int t0, int t1, int tx, int ty,
                                              double v[4][4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) v[q][p] = 0.0;
#pragma unroll 4
    for (int t = t0; t < t1; ++t) {
        const double2 w0 = *reinterpret_cast<const double2*>(W + t * kPanelStride + 2 * tx);
        const double2 w1 = *reinterpret_cast<const double2*>(W + t * kPanelStride + 32 + 2 * tx);
        const double2 c0 = *reinterpret_cast<const double2*>(P + t * kPanelStride + 4 * ty);
        const double2 c1 = *reinterpret_cast<const double2*>(P + t * kPanelStride + 4 * ty + 2);
        const double w[4] = {w0.x, w0.y, w1.x, w1.y}, c[4] = {c0.x, c0.y, c1.x, c1.y};
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int p = 0; p < 4; ++p) v[q][p] += c[q] * w[p];
    }
}

// Step s of the sweeps, panel: every block factors the pivot tile A_ss = L L^T (each for itself: a launch of
// its own would cost as much, and a block of k_trail that did it slowed that kernel by its registers);
// block i then forms W_i = A_is L^-T and V_i = W_i L^-1 = A_is A_ss^-1 (both transposed in the panels:
// unknown-major), block s leaves A_ss^-1 = L^-T L^-1 in piv. The update A_ij -= W_i W_j^T is a square: with
// the tile's explicit inverse, A_ij -= A_is (A_ss^-1 A_sj), the inverse's own rounding, eps / pivot^2,
// made a matrix of dependent hats indefinite (a graded part of 2x51x6 cells: eigenvalues of P X P^T K from
// -4200 to 4300). Bound by the tile's chain of 16 dependent steps; 40 us a step at 3993 unknowns, 33 with the
// explicit inverse and its one product.
__global__ void __launch_bounds__(kT) k_panel(int s, const CoarseGrid* __restrict__ grids, const double* __restrict__ A,
                                              const double* __restrict__ diag, int64_t diag_stride, double ridge,
                                              double* __restrict__ W, double* __restrict__ V, double* __restrict__ piv) {
    extern __shared__ __align__(16) double sm[];
    __shared__ TileMem mem;
    // X[t][c] = (L^-1)[t][c], Xt its transpose, Wt[t][r] = A_is[r][t], then W_i
    double *X = sm, *Xt = sm + kTile * kPanelStride, *Wt = sm + 2 * kTile * kPanelStride;
    const CoarseGrid& g = grids[blockIdx.y];
    const int tiles = g.ld / kTile, i = blockIdx.x;
    if (s >= tiles || i >= tiles) return;
    const double* Ai = A + g.dense0;
    const int64_t ld = g.ld, o = (int64_t)s * kTile, oi = (int64_t)i * kTile;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    if (tid < kTile) mem.limit[tid] = kDrop * ridge * diag[blockIdx.y * diag_stride + o + tid];
    double a[4][4], x[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int r = 4 * ty + q, c = 4 * tx + p;
            a[q][p] = Ai[(o + max(r, c)) * ld + o + min(r, c)];
        }
    if (i != s)
        for (int e = tid; e < kTile * kTile; e += kT) {
            const int h = e / kTile, l = e % kTile;
            if (i > s) Wt[l * kPanelStride + h] = Ai[(oi + h) * ld + o + l];
            else Wt[h * kPanelStride + l] = Ai[(o + h) * ld + oi + l];
        }
    __syncthreads();
    factor_tile(a, x, mem);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            X[(4 * ty + q) * kPanelStride + 4 * tx + p] = x[q][p];
            Xt[(4 * tx + p) * kPanelStride + 4 * ty + q] = x[q][p];
        }
    __syncthreads();
    double v[4][4];
    if (i == s) {
        panel_product(X, X, 4 * ty, kTile, tx, ty, v);
        double* out = piv + (int64_t)blockIdx.y * kTile * kTile;
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int p = 0; p < 4; ++p) out[(4 * ty + q) * kTile + 2 * tx + 16 * (p & 2) + (p & 1)] = v[q][p];
        return;
    }
    auto store = [&](double* to, int64_t stride) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            *reinterpret_cast<double2*>(to + (4 * ty + q) * stride + 2 * tx) = make_double2(v[q][0], v[q][1]);
            *reinterpret_cast<double2*>(to + (4 * ty + q) * stride + 32 + 2 * tx) = make_double2(v[q][2], v[q][3]);
        }
    };
    panel_product(Xt, Wt, 0, 4 * ty + 4, tx, ty, v);  // X is lower triangular
    store(W + g.y0 * kTile + oi, ld);
    __syncthreads();
    store(Wt, kPanelStride);
    __syncthreads();
    panel_product(X, Wt, 4 * ty, kTile, tx, ty, v);
    store(V + g.y0 * kTile + oi, ld);
}

// Step s, the rest: A_ij -= W_i W_j^T on the lower tiles, A_is = V_i, A_ss = -A_ss^-1. 64 x 64 x 64 a
// block of 128 threads, 8 x 4 entries a thread from shared memory (columns 2 tx, 2 tx + 1, 32 + ..:
// 16-byte reads without bank conflicts; 6 of them for 32 multiply-adds). Bound by the FP64 pipe once a
// step has more tiles than the device has SMs.
constexpr int kTrailT = 128;
__global__ void __launch_bounds__(kTrailT, 3) k_trail(int s, const CoarseGrid* __restrict__ grids, double* __restrict__ A,
                                                      const double* __restrict__ W, const double* __restrict__ V,
                                                      const double* __restrict__ piv) {
    extern __shared__ __align__(16) double sm[];
    const CoarseGrid& g = grids[blockIdx.y];
    const int tiles = g.ld / kTile, at = blockIdx.x;
    if (s >= tiles || at >= tiles * (tiles + 1) / 2) return;
    // tile (i, j), j <= i, of the linear index
    int i = (int)((sqrtf(8.0f * (float)at + 1.0f) - 1.0f) * 0.5f);
    while ((i + 1) * (i + 2) / 2 <= at) ++i;
    while (i * (i + 1) / 2 > at) --i;
    const int j = at - i * (i + 1) / 2;
    double* Ai = A + g.dense0;
    const int64_t ld = g.ld, oi = (int64_t)i * kTile, oj = (int64_t)j * kTile;
    const double *Wp = W + g.y0 * kTile, *Vp = V + g.y0 * kTile;
    const int tid = threadIdx.x;
    if (i == s || j == s) {
        for (int e = tid; e < kTile * kTile; e += kTrailT) {
            const int r = e / kTile, c = e % kTile;
            double x;
            if (i == s && j == s) x = -piv[(int64_t)blockIdx.y * kTile * kTile + e];
            else if (j == s) x = Vp[c * ld + oi + r];
            else x = Vp[r * ld + oj + c];
            Ai[(oi + r) * ld + oj + c] = x;
        }
        return;
    }
    double *sv = sm, *sw = sm + kTile * kTile;
#pragma unroll 4
    for (int e = tid; e < kTile * kTile / 2; e += kTrailT) {
        const int t = e / (kTile / 2), q = 2 * (e % (kTile / 2));
        *reinterpret_cast<double2*>(sv + t * kTile + q) = *reinterpret_cast<const double2*>(Wp + t * ld + oi + q);
        *reinterpret_cast<double2*>(sw + t * kTile + q) = *reinterpret_cast<const double2*>(Wp + t * ld + oj + q);
    }
    const int tx = tid & 15, ty = tid >> 4;
    double acc[8][4] = {};
    __syncthreads();
#pragma unroll 2
    for (int t = 0; t < kTile; ++t) {
        double av[8], bv[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const double2 x = *reinterpret_cast<const double2*>(sv + t * kTile + 8 * ty + 2 * h);
            av[2 * h] = x.x;
            av[2 * h + 1] = x.y;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double2 x = *reinterpret_cast<const double2*>(sw + t * kTile + 32 * h + 2 * tx);
            bv[2 * h] = x.x;
            bv[2 * h + 1] = x.y;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
            for (int p = 0; p < 4; ++p) acc[q][p] += av[q] * bv[p];
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double2* to = reinterpret_cast<double2*>(Ai + (oi + 8 * ty + q) * ld + oj + 32 * h + 2 * tx);
            double2 x = *to;
            x.x -= acc[q][2 * h];
            x.y -= acc[q][2 * h + 1];
            *to = x;
        }
}

// out = -A of the lower tiles, mirrored, in the PCG's precision; zero beyond m
template <typename T>
__global__ void __launch_bounds__(kT) k_mirror(const CoarseGrid* __restrict__ grids, const double* __restrict__ A,
                                               T* __restrict__ out) {
    __shared__ T tile[32][33];
    const CoarseGrid& g = grids[blockIdx.z];
    const int64_t ld = g.ld, r0 = 32 * (int64_t)blockIdx.y, c0 = 32 * (int64_t)blockIdx.x;
    if (r0 >= ld || c0 > r0) return;
    const double* Ai = A + g.dense0;
    T* oi = out + g.dense0;
    const int lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < 32; q += kT / 32) {
        const int64_t r = r0 + q, c = c0 + lane;
        T x = T(0);
        if (r < g.m && c < g.m) x = (T)(-(c <= r ? Ai[r * ld + c] : Ai[c * ld + r]));
        tile[q][lane] = x;
        oi[r * ld + c] = x;
    }
    __syncthreads();
    if (c0 == r0) return;
    for (int q = threadIdx.x >> 5; q < 32; q += kT / 32) oi[(c0 + q) * ld + r0 + lane] = tile[lane][q];
}

struct Temp {
    void* p = nullptr;
    explicit Temp(size_t n) : p(device_alloc(n ? n : 1)) {}
    ~Temp() { dfree(p); }
    Temp(const Temp&) = delete;
    Temp& operator=(const Temp&) = delete;
    template <typename T>
    T* as() const { return static_cast<T*>(p); }
};

}  // namespace

void coarse_box(const double* xyz, const uint8_t* used, int64_t n0, int64_t n1, double box[6]) {
    for (int a = 0; a < 3; ++a) {
        box[a] = INFINITY;
        box[3 + a] = -INFINITY;
    }
    for (int64_t v = n0; v < n1; ++v)
        for (int a = 0; a < 3 && used[v]; ++a) {
            box[a] = std::min(box[a], xyz[3 * v + a]);
            box[3 + a] = std::max(box[3 + a], xyz[3 * v + a]);
        }
}

void coarse_box(const double* xyz, const int64_t* inc_ptr, int64_t n_nodes, cudaStream_t st, double box[6]) {
    Temp ext(6 * sizeof(unsigned long long));
    unsigned long long h[6];
    CK(cudaMemsetAsync(ext.p, 0, sizeof(h), st));
    const unsigned blocks = std::min<unsigned>(grid_of(n_nodes), 4 * (unsigned)device_sms());
    k_box<<<blocks, kT, 0, st>>>(n_nodes, xyz, inc_ptr, ext.as<unsigned long long>());
    CK(cudaGetLastError());
    counted();
    CK(cudaMemcpyAsync(h, ext.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (int a = 0; a < 6; ++a) {
        const unsigned long long key = a < 3 ? ~h[a] : h[a];
        const unsigned long long bits = key >> 63 ? key & ~(1ull << 63) : ~key;
        std::memcpy(&box[a], &bits, sizeof(double));
    }
}

// About cubic cells; as many coarse nodes as a cube of 3 rows^0.44 cells has, at most 11^3 (elastic).
// A finer grid saves iterations (they go with the nodes across a cell), a coarser one set-up (m^3)
// and the product E^-1 r (m^2). Measured over the factor on the cube's side (ms a call): Tet10 40^3
// mixed 189 / 168 / 163 / 161 at 0.6 / 0.75 / 0.9 / 1, four load cases on Tet10 21x24x18 51 / 43 / 39 /
// 37, SIMP Tet4 48^3 54 / 47 / 41 / 41. One unknown a node allows a longer side: the thermal Tet10
// 40^3 step took 171 / 166 / 171 at 1 / 1.2 / 1.44 (43 / 38 / 32 iterations an increment), Tet4
// 23x30x17 26.5 / 25.4 / 24.3.
void coarse_cells(int dof, const double box[6], int64_t rows, int32_t k[3]) {
    const double more = dof == 1 ? 1.2 : 1.0;
    if (rows < kMinRows) rows = 1;
    const double side = more * std::min(10.0, std::cbrt(3.0 * std::pow((double)std::max<int64_t>(rows, 1), 0.44)));
    const double target = rows == 1 ? 8.0 : std::max(8.0, std::pow(side + 1.0, 3.0) * 1.0001);
    double ext[3], longest = 0.0;
    for (int a = 0; a < 3; ++a) {
        ext[a] = std::max(0.0, box[3 + a] - box[a]);
        longest = std::max(longest, ext[a]);
    }
    for (int a = 0; a < 3; ++a) k[a] = 1;
    if (!(longest > 0.0) || !std::isfinite(longest)) return;
    auto cells = [&](double edge, int32_t q[3]) {
        double n = 1.0;
        for (int a = 0; a < 3; ++a) {
            q[a] = (int32_t)std::max(1.0, std::min(1000.0, std::floor(ext[a] / edge + 0.5)));
            n *= q[a] + 1;
        }
        return n;
    };
    double lo = longest / 1001.0, hi = 2.0 * longest;  // edge: too many nodes at lo, one cell at hi
    for (int it = 0; it < 60; ++it) {
        const double mid = 0.5 * (lo + hi);
        int32_t q[3];
        if (cells(mid, q) > target) lo = mid; else hi = mid;
    }
    cells(hi, k);
}

Coarse::~Coarse() {
    std::vector<void*> all;
    gather(all);
    for (void* p : all) dfree(p);
}

void Coarse::gather(std::vector<void*>& out) {
    for (void** p : {(void**)&d_grids_, (void**)&node_inst_, (void**)&inst_tile_, (void**)&tile_, (void**)&dot_, (void**)&pos_, &w_, &ws_, &inv_, &part_, &rc_, &y_, (void**)&chunk_,
                     (void**)&cell_chunk_, (void**)&bpos_, (void**)&brow_, (void**)&bcol_, (void**)&schunk_ptr_,
                     (void**)&table_, (void**)&schunk_, (void**)&spart_, (void**)&A_, (void**)&diag_, (void**)&panel_w_,
                     (void**)&panel_v_, (void**)&piv_}) {
        out.push_back(*p);
        *p = nullptr;
    }
    nb_ = 0;
}

void Coarse::plan(int dof, bool fp32, int32_t nb, int64_t blocks, const double* xyz, const int32_t* perm,
                  const uint8_t* fixmask, const int64_t* row_ptr, const int32_t* col, const int32_t* row_inst,
                  const std::vector<double>& box, const std::vector<int64_t>& rows_of, cudaStream_t st, int rhs) {
    const int n_inst = (int)rows_of.size();
    if (n_inst == 0 || n_inst > 65535 || *std::max_element(rows_of.begin(), rows_of.end()) < kMinRows ||
        blocks >= INT_MAX || nb >= (1 << 28))
        return;
    dof_ = dof;
    fp32_ = fp32;
    grids_.assign(n_inst, CoarseGrid{});
    ncells_ = 0;
    int64_t nodes = 0, dense = 0, ldsum = 0, tab = 0;
    steps_ = 0;
    for (int q = 0; q < n_inst; ++q) {
        CoarseGrid& g = grids_[q];
        coarse_cells(dof, box.data() + 6 * q, rows_of[q], g.k);
        int64_t nn = 1, nc = 1;
        for (int a = 0; a < 3; ++a) {
            const double ext = box[6 * q + 3 + a] - box[6 * q + a];
            g.lo[a] = rows_of[q] > 0 ? box[6 * q + a] : 0.0;
            g.inv_h[a] = rows_of[q] > 0 && ext > 0.0 ? g.k[a] / ext : 0.0;
            nn *= g.k[a] + 1;
            nc *= g.k[a];
        }
        g.cell0 = ncells_;
        g.node0 = (int32_t)nodes;
        g.m = (int32_t)(dof * nn);
        g.ld = (g.m + kTile - 1) / kTile * kTile;
        g.dense0 = dense;
        g.y0 = ldsum;
        g.tab0 = tab;
        ncells_ += (int32_t)nc;
        nodes += nn;
        dense += (int64_t)g.ld * g.ld;
        ldsum += g.ld;
        tab += nc * nc;
        steps_ = std::max(steps_, g.ld / kTile);
    }
    nodes_ = nodes;
    dense_ = dense;
    pos_ = dalloc<double4>(nb);
    Temp cell(nb * sizeof(int32_t)), cell_sorted(nb * sizeof(int32_t)), rows(nb * sizeof(int32_t)),
        order(nb * sizeof(int32_t)), cell_ptr((ncells_ + 1) * sizeof(int32_t));
    d_grids_ = dupload(grids_.data(), grids_.size(), st);
    k_place<<<grid_of(nb), kT, 0, st>>>(nb, xyz, perm, fixmask, row_inst, d_grids_, pos_, cell.as<int32_t>(),
                                       rows.as<int32_t>());
    CK(cudaGetLastError());
    int sh = 1;
    while ((int64_t(1) << sh) <= ncells_) ++sh;
    {
        size_t bytes = 0;
        CK(cub::DeviceRadixSort::SortPairs(nullptr, bytes, cell.as<int32_t>(), cell_sorted.as<int32_t>(),
                                           rows.as<int32_t>(), order.as<int32_t>(), nb, 0, sh, st));
        Temp tmp(bytes);
        CK(cub::DeviceRadixSort::SortPairs(tmp.p, bytes, cell.as<int32_t>(), cell_sorted.as<int32_t>(),
                                           rows.as<int32_t>(), order.as<int32_t>(), nb, 0, sh, st));
        k_cell_ptr<<<grid_of(ncells_ + 1), kT, 0, st>>>(cell_sorted.as<int32_t>(), nb, ncells_, cell_ptr.as<int32_t>());
        CK(cudaGetLastError());
        counted(4);
        CK(cudaStreamSynchronize(st));  // tmp is freed
    }
    std::vector<int32_t> h_ptr(ncells_ + 1);
    CK(cudaMemcpyAsync(h_ptr.data(), cell_ptr.p, h_ptr.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    const size_t wbytes = (size_t)nb * 4 * (fp32 ? 4 : 8);
    w_ = device_alloc(wbytes);
    ws_ = device_alloc(wbytes);
    if (fp32)
        k_row_weights<float><<<grid_of(nb), kT, 0, st>>>(nb, pos_, order.as<int32_t>(), static_cast<float4*>(w_),
                                                         static_cast<float4*>(ws_));
    else
        k_row_weights<double><<<grid_of(nb), kT, 0, st>>>(nb, pos_, order.as<int32_t>(), static_cast<double4*>(w_),
                                                          static_cast<double4*>(ws_));
    CK(cudaGetLastError());
    counted(1);
    // blocks by cell pair
    Temp brow(blocks * sizeof(int32_t)), bpos(blocks * sizeof(int32_t));
    bpos_ = dalloc<int32_t>(blocks);
    std::vector<uint64_t> seg_key;
    std::vector<int32_t> seg_len;
    {
        Temp key(blocks * sizeof(uint64_t)), key_sorted(blocks * sizeof(uint64_t));
        k_pair_cells<<<grid_of((int64_t)nb * 32), kT, 0, st>>>(nb, row_ptr, col, cell.as<int32_t>(), sh, key.as<uint64_t>(),
                                                               bpos.as<int32_t>(), brow.as<int32_t>());
        CK(cudaGetLastError());
        size_t bytes = 0, rle = 0;
        CK(cub::DeviceRadixSort::SortPairs(nullptr, bytes, key.as<uint64_t>(), key_sorted.as<uint64_t>(),
                                           bpos.as<int32_t>(), bpos_, (int)blocks, 0, 2 * sh, st));
        // distinct pairs: a cell reaches few others, but no more runs than blocks
        Temp uniq(blocks * sizeof(uint64_t)), len(blocks * sizeof(int32_t)), nruns(sizeof(int32_t));
        CK(cub::DeviceRunLengthEncode::Encode(nullptr, rle, key_sorted.as<uint64_t>(), uniq.as<uint64_t>(),
                                              len.as<int32_t>(), nruns.as<int32_t>(), (int)blocks, st));
        Temp tmp(std::max(bytes, rle));
        CK(cub::DeviceRadixSort::SortPairs(tmp.p, bytes, key.as<uint64_t>(), key_sorted.as<uint64_t>(),
                                           bpos.as<int32_t>(), bpos_, (int)blocks, 0, 2 * sh, st));
        CK(cub::DeviceRunLengthEncode::Encode(tmp.p, rle, key_sorted.as<uint64_t>(), uniq.as<uint64_t>(),
                                              len.as<int32_t>(), nruns.as<int32_t>(), (int)blocks, st));
        counted(4);
        int32_t runs = 0;
        CK(cudaMemcpyAsync(&runs, nruns.p, sizeof(runs), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        seg_key.resize(runs);
        seg_len.resize(runs);
        CK(cudaMemcpyAsync(seg_key.data(), uniq.p, runs * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(seg_len.data(), len.p, runs * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    // ~0 sorts by its low 2 sh bits, all ones: above every pair of cells (cells < 2^sh - 1)
    if (!seg_key.empty() && seg_key.back() == ~0ull) {
        seg_key.pop_back();
        seg_len.pop_back();
    }
    nseg_ = (int32_t)seg_key.size();
    // chunks of rows and of blocks
    std::vector<int4> chunk;
    std::vector<int2> schunk, tile;
    std::vector<int32_t> cell_chunk(ncells_ + 1, 0), node_inst, inst_tile(1, 0);
    const int32_t step = rhs > 0 ? kBatchChunk : kRowChunk;
    for (int q = 0; q < n_inst; ++q) {
        const CoarseGrid& g = grids_[q];
        const int32_t nc = g.k[0] * g.k[1] * g.k[2];
        for (int32_t l = 0; l < nc; ++l) {
            const int32_t c = g.cell0 + l, x = l % g.k[0], y = l / g.k[0] % g.k[1], z = l / (g.k[0] * g.k[1]);
            const int32_t base = g.node0 + x + (g.k[0] + 1) * (y + (g.k[1] + 1) * z);
            for (int32_t p = h_ptr[c]; p < h_ptr[c + 1]; p += step)
                chunk.push_back(make_int4(p, std::min(p + step, h_ptr[c + 1]), base, q));
            cell_chunk[c + 1] = (int32_t)chunk.size();
        }
        if (rhs > 0) {
            node_inst.insert(node_inst.end(), g.m / dof, q);
            for (int32_t e = 0; e < g.m; e += kCoarseTileRows) tile.push_back(make_int2(q, e));
            inst_tile.push_back((int32_t)tile.size());
        }
    }
    std::vector<int32_t> schunk_ptr(nseg_ + 1, 0);
    std::vector<int64_t> at(nseg_);
    int32_t first = 0;
    size_t inst = 0;
    for (int32_t s = 0; s < nseg_; ++s) {
        const int32_t ci = (int32_t)(seg_key[s] >> sh), cj = (int32_t)(seg_key[s] & ((uint64_t(1) << sh) - 1));
        while (inst + 1 < grids_.size() && ci >= grids_[inst + 1].cell0) ++inst;
        CoarseGrid& g = grids_[inst];
        const int32_t a = ci - g.cell0, b = cj - g.cell0, nc = g.k[0] * g.k[1] * g.k[2];
        at[s] = g.tab0 + (int64_t)a * nc + b;
        const int32_t da[3] = {a % g.k[0] - b % g.k[0], a / g.k[0] % g.k[1] - b / g.k[0] % g.k[1],
                               a / (g.k[0] * g.k[1]) - b / (g.k[0] * g.k[1])};
        for (int q = 0; q < 3; ++q) g.span = std::max(g.span, std::abs(da[q]));
        for (int32_t p = 0; p < seg_len[s]; p += kPairChunk)
            schunk.push_back(make_int2(first + p, first + std::min(p + kPairChunk, seg_len[s])));
        first += seg_len[s];
        schunk_ptr[s + 1] = (int32_t)schunk.size();
    }
    nchunks_ = (int32_t)chunk.size();
    nschunks_ = (int32_t)schunk.size();
    CK(cudaMemcpyAsync(d_grids_, grids_.data(), grids_.size() * sizeof(CoarseGrid), cudaMemcpyHostToDevice, st));
    chunk_ = dupload(chunk.data(), chunk.size(), st);
    cell_chunk_ = dupload(cell_chunk.data(), cell_chunk.size(), st);
    schunk_ = dupload(schunk.data(), schunk.size(), st);
    schunk_ptr_ = dupload(schunk_ptr.data(), schunk_ptr.size(), st);
    brow_ = dalloc<int32_t>(first);
    bcol_ = dalloc<int32_t>(first);
    k_sorted_rc<<<grid_of(first), kT, 0, st>>>(first, bpos_, brow.as<int32_t>(), col, brow_, bcol_);
    table_ = dalloc<int32_t>(tab);
    CK(cudaMemsetAsync(table_, 0xFF, tab * sizeof(int32_t), st));
    int64_t* d_at = dupload(at.data(), at.size(), st);
    k_table<<<grid_of(nseg_), kT, 0, st>>>(nseg_, d_at, table_);
    CK(cudaGetLastError());
    counted(2);
    const int d2 = dof * dof;
    const size_t tb = fp32 ? 4 : 8;
    spart_ = dalloc<double>((size_t)nschunks_ * 64 * d2);
    A_ = dalloc<double>(dense_);
    diag_ = dalloc<double>((size_t)n_inst * steps_ * kTile);
    panel_w_ = dalloc<double>(ldsum * kTile);
    panel_v_ = dalloc<double>(ldsum * kTile);
    piv_ = dalloc<double>((size_t)n_inst * kTile * kTile);
    inv_ = device_alloc(dense_ * tb);
    // one system: rc by unknown, padded with zeros to ld; y 4 a node (dof 3). Batch: [node][R][3] both
    const size_t cols = rhs > 0 ? rhs : 1;
    const size_t nrc = rhs > 0 ? (size_t)nodes * dof * cols : (size_t)ldsum;
    const size_t ny = rhs > 0 ? (size_t)nodes * dof * cols : (size_t)nodes * (dof == 3 ? 4 : 1);
    part_ = device_alloc((size_t)std::max(1, nchunks_) * 8 * dof * cols * tb);
    rc_ = device_alloc(nrc * tb);
    y_ = device_alloc(ny * tb);
    CK(cudaMemsetAsync(rc_, 0, nrc * tb, st));
    CK(cudaMemsetAsync(y_, 0, ny * tb, st));
    if (rhs > 0) {
        ntiles_ = (int32_t)tile.size();
        tile_ = dupload(tile.data(), tile.size(), st);
        inst_tile_ = dupload(inst_tile.data(), inst_tile.size(), st);
        node_inst_ = dupload(node_inst.data(), node_inst.size(), st);
        dot_ = dalloc<double>((size_t)ntiles_ * (kCoarseTileRows / 4) * cols);
    }
    CK(cudaStreamSynchronize(st));  // the host lists and the temporaries go
    dfree(d_at);
    nb_ = nb;
}

void Coarse::update(const double* vals, cudaStream_t st) {
    if (!active()) return;
    const unsigned n_inst = (unsigned)grids_.size();
    const int64_t stride = (int64_t)steps_ * kTile, d2 = (int64_t)dof_ * dof_;
    const double ridge = fp32_ ? kRidge32 : kRidge64;
    const unsigned pg = (unsigned)std::max(1, (nschunks_ + kPairWarps - 1) / kPairWarps);
    int64_t most = 1;  // (coarse node, node within reach, entry) of the largest instance
    for (const CoarseGrid& g : grids_) {
        int64_t window = 1;
        for (int a = 0; a < 3; ++a) window *= 2 * std::min(g.span + 1, g.k[a]) + 1;
        most = std::max<int64_t>(most, g.m / dof_ * window * d2);
    }
    const dim3 dg(grid_of(most), n_inst);
    CK(cudaMemsetAsync(A_, 0, (size_t)dense_ * sizeof(double), st));
    if (dof_ == 3) {
        k_pairs<3><<<pg, kPairWarps * 32, 0, st>>>(nschunks_, schunk_, bpos_, brow_, bcol_, pos_, vals, spart_);
        k_pair_sums<3><<<grid_of(nseg_ * 64 * d2), kT, 0, st>>>(nseg_, schunk_ptr_, spart_);
        k_dense<3><<<dg, kT, 0, st>>>(d_grids_, table_, schunk_ptr_, spart_, A_, diag_, stride, ridge);
    } else {
        k_pairs<1><<<pg, kPairWarps * 32, 0, st>>>(nschunks_, schunk_, bpos_, brow_, bcol_, pos_, vals, spart_);
        k_pair_sums<1><<<grid_of(nseg_ * 64 * d2), kT, 0, st>>>(nseg_, schunk_ptr_, spart_);
        k_dense<1><<<dg, kT, 0, st>>>(d_grids_, table_, schunk_ptr_, spart_, A_, diag_, stride, ridge);
    }
    CK(cudaGetLastError());
    constexpr int smem = 2 * kTile * kTile * (int)sizeof(double);
    constexpr int psmem = 3 * kTile * kPanelStride * (int)sizeof(double);
    CK(cudaFuncSetAttribute(k_trail, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    CK(cudaFuncSetAttribute(k_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, psmem));
    for (int s = 0; s < steps_; ++s) {
        k_panel<<<dim3(steps_, n_inst), kT, psmem, st>>>(s, d_grids_, A_, diag_, stride, ridge, panel_w_, panel_v_, piv_);
        k_trail<<<dim3(steps_ * (steps_ + 1) / 2, n_inst), kTrailT, smem, st>>>(s, d_grids_, A_, panel_w_, panel_v_, piv_);
    }
    const dim3 mg(2 * steps_, 2 * steps_, n_inst);
    if (fp32_) k_mirror<float><<<mg, kT, 0, st>>>(d_grids_, A_, static_cast<float*>(inv_));
    else k_mirror<double><<<mg, kT, 0, st>>>(d_grids_, A_, static_cast<double*>(inv_));
    CK(cudaGetLastError());
    counted(4 + 2 * steps_);
}

template <typename T>
CoarseDev<T> Coarse::dev(int inst) const {
    CoarseDev<T> c;
    if (!active()) return c;
    const CoarseGrid& g = grids_[inst];
    c.nn = g.m / dof_;
    c.m = g.m;
    c.ld = g.ld;
    c.kx = g.k[0];
    c.ky = g.k[1];
    c.kz = g.k[2];
    c.nchunks = nchunks_;
    c.w = static_cast<const T*>(w_);
    c.ws = static_cast<const T*>(ws_);
    c.chunk = chunk_;
    c.cell_chunk = cell_chunk_ + g.cell0;
    c.inv = static_cast<const T*>(inv_) + g.dense0;
    c.part = static_cast<T*>(part_);
    c.rc = static_cast<T*>(rc_) + g.y0;
    c.y = static_cast<T*>(y_) + (int64_t)g.node0 * (dof_ == 3 ? 4 : 1);
    return c;
}
template CoarseDev<float> Coarse::dev<float>(int) const;
template CoarseDev<double> Coarse::dev<double>(int) const;

template <typename T>
CoarseBatchDev<T> Coarse::batch() const {
    CoarseBatchDev<T> c;
    if (!active()) return c;
    c.nodes = (int32_t)nodes_;
    c.nchunks = nchunks_;
    c.ntiles = ntiles_;
    c.grids = d_grids_;
    c.ws = static_cast<const T*>(ws_);
    c.chunk = chunk_;
    c.cell_chunk = cell_chunk_;
    c.node_inst = node_inst_;
    c.tile = tile_;
    c.inst_tile = inst_tile_;
    c.inv = static_cast<const T*>(inv_);
    c.part = static_cast<T*>(part_);
    c.rc = static_cast<T*>(rc_);
    c.y = static_cast<T*>(y_);
    c.dot = dot_;
    return c;
}
template CoarseBatchDev<float> Coarse::batch<float>() const;
template CoarseBatchDev<double> Coarse::batch<double>() const;

}  // namespace maille
