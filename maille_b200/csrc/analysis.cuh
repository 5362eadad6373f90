// analysis.cuh -- the symbolic analysis on the device (analysis.cu, ordering.cu): kept nodes, their
// graph, the rows of the system in the order that ordering.cu finds, the full block pattern with its
// transpose positions, the boundary lists of the reactions, and the slot columns of the SpMV and
// sweep layouts. Everything is a deterministic function of the connectivity and the ordering.
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "common.hpp"
#include "cuda_host.hpp"

namespace maille {

// Device buffers of one pass, freed together once its stream is idle (a free of its own waits for the
// device each time).
class Scratch {
  public:
    explicit Scratch(cudaStream_t st) : st_(st) {}
    ~Scratch() { release(); }
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    template <typename T>
    T* take(size_t n) {
        T* p = dalloc<T>(n);
        all_.push_back(p);
        return p;
    }
    void release() {
        if (all_.empty()) return;
        cudaStreamSynchronize(st_);
        device_free_all(all_);
        all_.clear();
    }

  private:
    cudaStream_t st_;
    std::vector<void*> all_;
};

// The graph of the kept nodes: neighbours by ascending kept index, self excluded.
struct GraphDev {
    int32_t nk = 0;
    int64_t m = 0;
    int64_t* off = nullptr;  // [nk + 1]
    int32_t* adj = nullptr;  // [m]
    int32_t* deg = nullptr;  // [nk]
    bool repeats = false;    // an element names a node twice
    cudaStream_t st = nullptr;  // its last user
    GraphDev() = default;
    GraphDev(const GraphDev&) = delete;
    GraphDev& operator=(const GraphDev&) = delete;
    ~GraphDev() {
        if (!off) return;
        cudaStreamSynchronize(st);
        device_free_all({off, adj, deg});
    }
};

// Device arrays of the analysed pattern; the caller owns them once built.
struct PatternDev {
    int64_t* row_ptr = nullptr;    // [nb + 1]
    int32_t* col = nullptr;        // [blocks], ascending per row
    int64_t* diag = nullptr;       // [nb]
    int64_t* tpos = nullptr;       // [blocks] position of the transposed block
    int64_t blocks = 0;
};

// Kept nodes: a node with a free unknown of its `dof` (fixed: [dof n_nodes] on the device). kept_of:
// [n_nodes] kept index or -1, kept: [n_nodes] (the first nk entries are filled); returns nk.
int32_t gpu_keep(int dof, int64_t n_nodes, const uint8_t* fixed, cudaStream_t st, int32_t* kept_of, int32_t* kept);

// The graph from the connectivity and its node incidence (gpu_incidence). Throws CudaFailure on a
// CUDA error or a mesh that 32-bit positions do not hold.
void gpu_graph(int npe, int64_t n_elems, const int32_t* conn, const int64_t* inc_ptr, const int32_t* inc,
               const int32_t* kept_of, const int32_t* kept, int32_t nk, cudaStream_t st, GraphDev& out);

// perm (row -> node), inv (node -> row, -1 when dropped), rank (kept index -> row) and, for dof 3,
// fixmask (fixed components of each row) from order (row -> kept index).
void gpu_rows(int dof, int32_t nk, int64_t n_nodes, const int32_t* order, const int32_t* kept, const int32_t* kept_of,
              const uint8_t* fixed, cudaStream_t st, int32_t* perm, int32_t* inv, int32_t* rank, uint8_t* fixmask);
// order and rank of rows numbered elsewhere (perm).
void gpu_ranks(int32_t nk, const int32_t* perm, const int32_t* kept_of, cudaStream_t st, int32_t* order, int32_t* rank);

// The block pattern of the rows. Also returns host copies of row_ptr and diag (the layout plans need the
// row lengths). Throws CudaFailure on a CUDA error.
void gpu_pattern(const GraphDev& g, const int32_t* order, const int32_t* rank, cudaStream_t st, PatternDev& out,
                 std::vector<int64_t>& h_row_ptr, std::vector<int64_t>& h_diag);

// The elements with a fixed DOF (belem, by index), the nodes of those elements (bnodes), every
// element's place in belem or -1 (elem_slot), and whether a node has no element. The caller owns the
// arrays.
struct BoundaryDev {
    int32_t *belem = nullptr, *bnodes = nullptr, *elem_slot = nullptr;
    int64_t nbelem = 0, nbnodes = 0;
    bool orphans = false;
};
void gpu_boundary(int npe, int64_t n_elems, const int32_t* conn, int64_t n_nodes, const uint8_t* fixed,
                  const int64_t* inc_ptr, cudaStream_t st, BoundaryDev& out);

// Slot columns (col, padding = nb) and CSR sources (src, padding = -1) of a sliced K layout
// (kind SELL_FULL) from its plan (rowid, off already on the device) and the device pattern.
void fill_sell(SellKind kind, int32_t lpr, int32_t nslices, int64_t steps, const int32_t* rowid,
               const int64_t* off, const int64_t* row_ptr, const int32_t* col, const int64_t* diag,
               int32_t nb, int32_t* slot_col, int32_t* slot_src, cudaStream_t st);

// The same for a packed factor layout (rows, rstart of the plan on the device).
void fill_psell(SellKind kind, int64_t nrows, int64_t steps, const int32_t* rows, const int64_t* rstart,
                const int64_t* row_ptr, const int32_t* col, const int64_t* diag, int32_t nb,
                int32_t* slot_col, int32_t* slot_src, cudaStream_t st);

// The same for a batched layout of `rows` rows a slice and `sub` lanes a row.
void fill_bsell(SellKind kind, int rows, int sub, int32_t nslices, int64_t steps, const int32_t* rowid,
                const int64_t* off, const int64_t* row_ptr, const int32_t* col, const int64_t* diag, int32_t nb,
                int32_t* slot_col, int32_t* slot_src, cudaStream_t st);

}  // namespace maille
