// coarse_dev.cuh -- device side of the coarse correction (coarse.cuh), for the persistent PCG kernels:
// z += P E^-1 P^T r in three phases separated by barriers of the caller (of its grid, or of the blocks that
// form a coarse team, coarse_team_barrier):
//   coarse_restrict  each warp sums w_a(x_i) r_i over a chunk of one cell's rows, for the cell's 8
//                    corners (r is read once; a chunk's partial sums go to its own slots, so the
//                    result does not depend on the order the warps run in);
//   coarse_gather    P^T r of a coarse node: the partial sums of its at most 8 cells, in order;
//   coarse_apply     y = E^-1 P^T r, one warp per row of the dense inverse, and this thread's
//                    share of (P^T r) . y, which is r . (P E^-1 P^T r).
// The caller adds P y to z wherever it reads z next (coarse_interpolate3, coarse_interpolate1).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "coarse.cuh"

namespace maille {

// (fx, fy, fz, code) of one row
__device__ __forceinline__ void coarse_row(const float* w, int64_t i, float f[3], uint32_t& code) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(w) + i);
    f[0] = q.x; f[1] = q.y; f[2] = q.z;
    code = __float_as_uint(q.w);
}
__device__ __forceinline__ void coarse_row(const double* w, int64_t i, double f[3], uint32_t& code) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(w + 4 * i));
    const double2 b = __ldg(reinterpret_cast<const double2*>(w + 4 * i + 2));
    f[0] = a.x; f[1] = a.y; f[2] = b.x;
    code = (uint32_t)__double_as_longlong(b.y);
}

// the 8 hat weights of a point at fractions f of its cell; corner a = x + 2 y + 4 z
template <typename T>
__device__ __forceinline__ void coarse_weights(const T f[3], T w[8]) {
    const T x1 = f[0], y1 = f[1], z1 = f[2];
    const T x0 = T(1) - x1, y0 = T(1) - y1, z0 = T(1) - z1;
    const T a = y0 * z0, b = y1 * z0, c = y0 * z1, d = y1 * z1;
    w[0] = x0 * a; w[1] = x1 * a; w[2] = x0 * b; w[3] = x1 * b;
    w[4] = x0 * c; w[5] = x1 * c; w[6] = x0 * d; w[7] = x1 * d;
}

// the DOF residuals of row i: r is padded to 4 entries a row when DOF is 3, plain when it is 1
template <int DOF>
__device__ __forceinline__ void coarse_load_r(const float* r, int64_t i, float* v) {
    if constexpr (DOF == 3) {
        const float4 q = __ldcg(reinterpret_cast<const float4*>(r) + i);
        v[0] = q.x; v[1] = q.y; v[2] = q.z;
    } else {
        v[0] = __ldcg(r + i);
    }
}
template <int DOF>
__device__ __forceinline__ void coarse_load_r(const double* r, int64_t i, double* v) {
    if constexpr (DOF == 3) {
        const double2 q = __ldcg(reinterpret_cast<const double2*>(r + 4 * i));
        v[0] = q.x; v[1] = q.y; v[2] = __ldcg(r + 4 * i + 2);
    } else {
        v[0] = __ldcg(r + i);
    }
}

// one halving step of a transposed warp sum: N values a lane, N / 2 after it
template <int N, typename T>
__device__ __forceinline__ void coarse_halve(T* v, int bit, int lane) {
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
        const T send = up ? v[q] : v[q + N / 2];
        const T keep = up ? v[q + N / 2] : v[q];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
}

// r is padded to 4 entries a row when DOF is 3, plain when it is 1. `warp` of `nwarps` in the grid.
template <typename T, int DOF>
__device__ __noinline__ void coarse_restrict(const CoarseDev<T> c, const T* r, int32_t warp, int32_t nwarps) {
    constexpr int U = DOF == 1 ? 1 : 2;  // rows a lane has in flight; more cost the sweeps registers
    const int lane = threadIdx.x & 31;
    for (int32_t k = warp; k < c.nchunks; k += nwarps) {
        const int4 range = __ldg(c.chunk + k);
        T s[8 * DOF];
#pragma unroll
        for (int q = 0; q < 8 * DOF; ++q) s[q] = T(0);
        for (int32_t p = range.x + lane; p < range.y; p += 32 * U) {
            T f[U][3], v[U][DOF];
            uint32_t row[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p + 32 * u < range.y) coarse_row(c.ws, p + 32 * u, f[u], row[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p + 32 * u < range.y) coarse_load_r<DOF>(r, (int64_t)(row[u] & kCoarseRow), v[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p + 32 * u < range.y) {
                    T w[8];
                    coarse_weights(f[u], w);
#pragma unroll
                    for (int a = 0; a < 8; ++a)
#pragma unroll
                        for (int d = 0; d < DOF; ++d) s[a * DOF + d] += w[a] * v[u][d];
                }
        }
        // lane bits 4, 3, 2 choose the corner's z, y, x; bits 1, 0 are summed
        coarse_halve<8 * DOF>(s, 16, lane);
        coarse_halve<4 * DOF>(s, 8, lane);
        coarse_halve<2 * DOF>(s, 4, lane);
#pragma unroll
        for (int d = 0; d < DOF; ++d) {
            s[d] += __shfl_xor_sync(0xffffffffu, s[d], 2);
            s[d] += __shfl_xor_sync(0xffffffffu, s[d], 1);
        }
        if ((lane & 3) == 0)
#pragma unroll
            for (int d = 0; d < DOF; ++d) c.part[((int64_t)k * 8 + (lane >> 2)) * DOF + d] = s[d];
    }
}

template <typename T, int DOF>
__device__ __noinline__ void coarse_gather(const CoarseDev<T> c, int64_t tid, int64_t nthreads) {
    for (int64_t e = tid; e < c.m; e += nthreads) {
        const int32_t g = (int32_t)(e / DOF), d = (int32_t)(e - (int64_t)g * DOF);
        const int32_t gx = g % (c.kx + 1), gq = g / (c.kx + 1), gy = gq % (c.ky + 1), gz = gq / (c.ky + 1);
        T s = T(0);
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int32_t x = gx - (a & 1), y = gy - ((a >> 1) & 1), z = gz - (a >> 2);
            if (x < 0 || y < 0 || z < 0 || x >= c.kx || y >= c.ky || z >= c.kz) continue;
            const int32_t cell = x + c.kx * (y + c.ky * z);
            const int32_t k1 = __ldg(c.cell_chunk + cell + 1);
            for (int32_t k = __ldg(c.cell_chunk + cell); k < k1; ++k)
                s += __ldcg(c.part + ((int64_t)k * 8 + a) * DOF + d);
        }
        c.rc[e] = s;
    }
}

// 16-byte pieces of a row of E^-1 against P^T r
__device__ __forceinline__ float coarse_dot16(const float* a, const float* x, float s) {
    const float4 p = __ldg(reinterpret_cast<const float4*>(a)), q = __ldcg(reinterpret_cast<const float4*>(x));
    return s + (p.x * q.x + p.y * q.y + p.z * q.z + p.w * q.w);
}
__device__ __forceinline__ double coarse_dot16(const double* a, const double* x, double s) {
    const double2 p = __ldg(reinterpret_cast<const double2*>(a)), q = __ldcg(reinterpret_cast<const double2*>(x));
    return s + (p.x * q.x + p.y * q.y);
}

template <typename T, int DOF>
__device__ __noinline__ double coarse_apply(const CoarseDev<T> c, int32_t warp, int32_t nwarps) {
    constexpr int V = 16 / (int)sizeof(T);
    const int lane = threadIdx.x & 31;
    double loc = 0.0;
    // two rows at a time: 4 KB a warp in flight
    for (int32_t e = warp; e < c.m; e += 2 * nwarps) {
        const bool two = e + nwarps < c.m;
        const T *row0 = c.inv + (int64_t)e * c.ld, *row1 = row0 + (two ? (int64_t)nwarps * c.ld : 0);
        T s[2] = {T(0), T(0)};  // ld is a multiple of 64, zero beyond m in the matrix and in rc
#pragma unroll 4
        for (int32_t q = lane * V; q < c.ld; q += 32 * V) {
            s[0] = coarse_dot16(row0 + q, c.rc + q, s[0]);
            s[1] = coarse_dot16(row1 + q, c.rc + q, s[1]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
            const int32_t i = e + j * nwarps;
            if (lane == 0 && (j == 0 || two)) {
                c.y[DOF == 3 ? 4 * (int64_t)(i / 3) + i % 3 : (int64_t)i] = s[j];
                loc += (double)__ldcg(c.rc + i) * (double)s[j];
            }
        }
    }
    return loc;
}

// Barrier among the blocks of a coarse team (co-resident with the grid): every block adds one to `arrived`
// and waits, at most `limit` reads, until it reaches `target`; on giving up raises `timeout`, which the
// caller reads after its next grid barrier.
__device__ __forceinline__ void coarse_team_barrier(int32_t* arrived, int32_t target, int32_t* timeout,
                                                    unsigned int limit) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(arrived, 1);
        int32_t n = 0;
        unsigned int k = 0;
        do {
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(n) : "l"(arrived) : "memory");
        } while (n < target && ++k < limit);
        if (n < target) atomicExch(timeout, 1);
    }
    __syncthreads();
}

// P y of a row (DOF 3) from y in shared memory (4 per coarse node), zero at fixed components
template <typename T>
__device__ __forceinline__ void coarse_interpolate3(const T* w, int64_t i, const T* y, int32_t sy, int32_t sz, T v[3]) {
    T f[3], h[8];
    uint32_t code;
    coarse_row(w, i, f, code);
    coarse_weights(f, h);
    const uint32_t g = code & kCoarseBase;
    v[0] = v[1] = v[2] = T(0);
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const T* q = y + 4 * (int64_t)(g + (a & 1) + ((a >> 1) & 1) * sy + (a >> 2) * sz);
        v[0] += h[a] * q[0];
        v[1] += h[a] * q[1];
        v[2] += h[a] * q[2];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if ((code >> (28 + d)) & 1u) v[d] = T(0);
}
template <typename T>
__device__ __forceinline__ T coarse_interpolate1(const T* w, int64_t i, const T* y, int32_t sy, int32_t sz) {
    T f[3], h[8], v = T(0);
    uint32_t code;
    coarse_row(w, i, f, code);
    coarse_weights(f, h);
    const uint32_t g = code & kCoarseBase;
#pragma unroll
    for (int a = 0; a < 8; ++a) v += h[a] * y[g + (a & 1) + ((a >> 1) & 1) * sy + (a >> 2) * sz];
    return v;
}

}  // namespace maille
