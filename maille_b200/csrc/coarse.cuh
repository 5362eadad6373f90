// coarse.cuh -- the coarse correction of the IC(0) preconditioner.
//
// IC(0) is a local preconditioner: one application moves information a few nodes, so the PCG's
// iteration count grows with the number of nodes across the mesh (Tet10 40^3 mixed: 827). The
// multicolour orderings add a coarse correction, M^-1 = (L L^T)^-1 + P E^-1 P^T:
//  * P interpolates from a coarse box grid over the mesh's bounding box with trilinear hat
//    functions (one value per DOF component), zero at fixed DOFs. The hats reproduce linear
//    displacement fields, so the smooth error modes that IC(0) leaves are in its range whatever
//    the mesh is; piecewise rigid modes per aggregate took 1.6x the iterations (Tet4 20^3, 125
//    parts: 77 against 47, and 237 without a correction);
//  * E = P^T K P is the Galerkin matrix of the assembled FP64 K, with a small ridge (kRidge64), held as its
//    dense inverse:
//    an application is one matrix-vector product read at HBM or L2 rate, with no dependent levels.
// Measured (B200, iterations and ms of the PCG alone): Tet10 40^3 mixed 827 -> 65, 264 -> 24.6 ms, with 5 ms
// more set-up; Tet4 20^3 FP64 225 -> 43, 17.0 -> 2.4 ms; SIMP Tet4 48^3 519 -> 63, 65 -> 7.9 ms; Tet4 6^3
// 63 -> 28. A part that its supports hold everywhere gains nothing (a plate of 200x200x1 cells clamped on its
// face: 19 -> 23 iterations); the call is still shorter than before the correction (24.6 -> 9.5 ms).
// Below 128 rows IC(0) alone stays.
// The sum is symmetric positive definite: IC(0) is, and E has a ridge that keeps its inverse so in the
// PCG's precision (kRidge64, kRidge32). The PCG's stopping test, statuses and caps are those of the plain
// preconditioner. The RCM ordering keeps IC(0) alone: it stands for the reference's own iteration
// counts. A device without room for the correction keeps IC(0) alone too.
//
// Independent instances (the batched solver) get a grid and a dense inverse each.
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace maille {

// One instance's coarse grid.
struct CoarseGrid {
    double lo[3], inv_h[3];  // t = (x - lo) inv_h is in [0, k]
    int32_t k[3];            // cells per axis
    int32_t cell0, node0;    // first cell and coarse node of the instance
    int32_t m;               // unknowns: dof (kx + 1)(ky + 1)(kz + 1)
    int32_t ld;              // row stride of the dense inverse (m rounded up to 64)
    int32_t span;            // cells that a block of K reaches across at most
    int64_t dense0;          // its first entry in the dense arrays
    int64_t y0;              // first entry of its vectors (4 per coarse node when dof is 3)
    int64_t tab0;            // its block of the cell-pair table
};

// What the PCG kernels read of one instance's correction; nn = 0: no correction.
template <typename T>
struct CoarseDev {
    int32_t nn = 0;      // coarse nodes
    int32_t m = 0, ld = 0;
    int32_t kx = 0, ky = 0, kz = 0;
    int32_t nchunks = 0;
    const T* w = nullptr;               // [4 nb] per row: fx, fy, fz in its cell, code (kCoarseBase)
    const T* ws = nullptr;              // [4 nb] the same in cell order, code = the row
    const int4* chunk = nullptr;        // [nchunks] (first, end) in the cell order, inside one cell
    const int32_t* cell_chunk = nullptr;  // [cells + 1] first chunk of each cell
    const T* inv = nullptr;             // [m * ld] E^-1
    T* part = nullptr;                  // [nchunks * 8 * dof] restricted residual of each chunk
    T* rc = nullptr;                    // [ld] P^T r
    T* y = nullptr;                     // [(dof == 3 ? 4 : 1) * nn] E^-1 P^T r
};

// The same for a batch of instances with R load cases each: vectors are [node][R][3], r and p
// [row][R][3], chunks and cells run over all instances.
template <typename T>
struct CoarseBatchDev {
    int32_t nodes = 0;                    // coarse nodes of all instances; 0: no correction
    int32_t nchunks = 0, ntiles = 0;
    const CoarseGrid* grids = nullptr;
    const T* ws = nullptr;                // [4 nb] in cell order: fx, fy, fz, row and fixed mask (kCoarseRow)
    const int4* chunk = nullptr;          // [nchunks] (first, end, base coarse node, instance)
    const int32_t* cell_chunk = nullptr;  // [cells + 1]
    const int32_t* node_inst = nullptr;   // [nodes] instance of each coarse node
    const int2* tile = nullptr;           // [ntiles] (instance, first unknown) of kCoarseTileRows rows
    const int32_t* inst_tile = nullptr;   // [n_inst + 1] first tile of each instance
    const T* inv = nullptr;
    T *part = nullptr, *rc = nullptr, *y = nullptr;  // [nchunks 8][R][3], [nodes][R][3], [nodes][R][3]
    double* dot = nullptr;                // [ntiles 4][R] shares of (P^T r) . y
};
constexpr int kCoarseTileRows = 16;

// Mixed forms with the correction: a reliable update when the FP32 residual fell by kCoarseDelta from the
// largest it has had since the last update (slender parts raise it by decades before it falls, and the
// recurrence drifts with the largest); when the true residual's square then differs from the recurrence's by
// more than kCoarseDrift of it, the direction starts anew (beta = 0): p is conjugate to the lost residual,
// and kept, it stalled the iteration. Iterations at tol 1e-10, IC(0) alone / p kept, 0.01 from the last true
// residual / always anew / as here: bar 10x10x60 1030 / singular / 46 / 44, 6x6x48 1082 / not in 10000 / 37 / 35,
// 4x4x32 648 / 672 / 35 / 34, Tet10 3x3x24 1119 / not / 38 / 36, quarter-cylinder shell 30x2x30 1130 / not / 83 /
// 82, plate 40x2x40 2199 / not / 70 / 68, cube Tet4 20^3 274 / 40 / 43 / 40.
constexpr double kCoarseDelta = 0.01;
constexpr double kCoarseDrift = 1e-4;

// The correction of one system (one or several instances): plan and numeric state.
class Coarse {
  public:
    ~Coarse();
    // Rows, pattern and grid of the system. xyz: [3 n_nodes] device coordinates; perm: [nb] row ->
    // node; fixmask: [nb] fixed components or null; row_ptr, col: the full pattern, dof x dof blocks.
    // row_inst: [nb] instance of each row or null (one instance). box: [6 instances] min and max
    // corners; rows_of: rows per instance; rhs: load cases of a batch (its layouts), 0: one system. Does
    // nothing (active() stays false) when no instance is large enough. Synchronises the stream. Throws
    // DeviceMemoryFull when there is no room.
    void plan(int dof, bool fp32, int32_t nb, int64_t blocks, const double* xyz, const int32_t* perm,
              const uint8_t* fixmask, const int64_t* row_ptr, const int32_t* col, const int32_t* row_inst,
              const std::vector<double>& box, const std::vector<int64_t>& rows_of, cudaStream_t st, int rhs = 0);
    // E and its inverse from the assembled values (dof x dof per block, CSR order); enqueued on st.
    void update(const double* vals, cudaStream_t st);
    bool active() const { return nb_ > 0; }
    CoarseDev<float> dev32(int inst = 0) const { return dev<float>(inst); }
    CoarseDev<double> dev64(int inst = 0) const { return dev<double>(inst); }
    template <typename T>
    CoarseBatchDev<T> batch() const;
    // the device buffers, handed over to be freed together; the correction is inactive afterwards
    void gather(std::vector<void*>& out);

  private:
    template <typename T>
    CoarseDev<T> dev(int inst) const;
    int dof_ = 3;
    bool fp32_ = false;
    int32_t nb_ = 0, nchunks_ = 0, nseg_ = 0, nschunks_ = 0, steps_ = 0, ncells_ = 0;
    int64_t dense_ = 0, nodes_ = 0;
    std::vector<CoarseGrid> grids_;
    CoarseGrid* d_grids_ = nullptr;
    double4* pos_ = nullptr;          // [nb] fractions and code, FP64 (Galerkin)
    void *w_ = nullptr, *ws_ = nullptr, *inv_ = nullptr, *part_ = nullptr, *rc_ = nullptr, *y_ = nullptr;
    int4* chunk_ = nullptr;
    int32_t *node_inst_ = nullptr, *inst_tile_ = nullptr;
    int2* tile_ = nullptr;
    double* dot_ = nullptr;
    int32_t ntiles_ = 0;
    int32_t* cell_chunk_ = nullptr;
    // Galerkin: blocks sorted by cell pair
    int32_t *bpos_ = nullptr, *brow_ = nullptr, *bcol_ = nullptr, *schunk_ptr_ = nullptr, *table_ = nullptr;
    int2* schunk_ = nullptr;
    double *spart_ = nullptr, *A_ = nullptr, *diag_ = nullptr, *panel_w_ = nullptr, *panel_v_ = nullptr, *piv_ = nullptr;
};

// Code of a row: base node of its cell in the low 28 bits, fixed components above.
constexpr uint32_t kCoarseBase = (1u << 28) - 1u;
// Cell order: the row in the low 29 bits, fixed mask above.
constexpr uint32_t kCoarseRow = (1u << 29) - 1u;

// Bounding box (min x, y, z, max x, y, z) of the nodes that an element names: a node of none, however far, would
// only take cells from the part. used: such nodes among [n0, n1), in host memory. inc_ptr: their incidence, on
// the device, enqueued on st and waited for.
void coarse_box(const double* xyz, const uint8_t* used, int64_t n0, int64_t n1, double box[6]);
void coarse_box(const double* xyz, const int64_t* inc_ptr, int64_t n_nodes, cudaStream_t st, double box[6]);
// Cells per axis for `rows` rows of `dof` unknowns in the box.
void coarse_cells(int dof, const double box[6], int64_t rows, int32_t k[3]);

}  // namespace maille
