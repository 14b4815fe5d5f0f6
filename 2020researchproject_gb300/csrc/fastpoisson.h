// Fast diagonalisation of the pressure-Poisson rows: the BiCGSTAB
// preconditioner of the mixed modes, and of FP64 solves without a body or
// with transforms of few operations.
//
// Without a body the fluid rows are separable: coeffsum times the
// normalised row is Ax + Ay + Az with one tridiagonal (periodic axes:
// cyclic) matrix per axis, the outer boundary rows folded in.  Each is
// D^-1 S with D the cell widths and S symmetric, so with S's eigenvectors Q
// the transform W = Q^T D^1/2 and its inverse D^-1/2 Q diagonalise it
// (Lynch, Rice and Thomas, "Direct solution of partial difference equations
// by tensor product methods", Numer. Math. 6, 1964).  Two axes are
// transformed by dense products; along the third each mode is a tridiagonal
// system, solved from pivots factored once at set-up (when neither x nor y
// can take that part because both wrap, all three axes are transformed and
// the modes divided by the eigenvalue sums).
//
// With a body the same solve ignores it (solid rows get no source, a ghost
// row the source of a fluid row over its diagonal 1 - w_self): the result
// is exact away from the body, and a few Gauss-Seidel sweeps over the cells
// near it, in overlapping patches, repair the rows there.
//
// The pinned row p'(0,0,0) of problems without a pressure boundary value is
// kept exactly: its fluid row's source is chosen so that the singular
// system is consistent, and the solution shifted by a constant to meet the
// pinned value.
//
// Measured (GB300, per application and BiCGSTAB iterations per step, against
// the multigrid V-cycle that served these cases before): channel
// 128x96x128 FP32 0.09 ms, 1 iteration (0.47 ms, 14); cavity 64^3 FP64
// 0.17 ms, 1 (0.31 ms, 10); sphere 192x128x128 FP32 0.13 ms, 3.1 (0.53 ms,
// 3.9); boxes 95x61x47 FP32 0.05 ms, 4.4 (0.25 ms, 4.9).
#pragma once

#include <vector>

#include "krylov.h"

namespace ibm {

// Host tables of the patches near the body (FpPatches).
template <typename T>
struct FpPatchTables {
    std::vector<int> P, to, start, count, loc;
    std::vector<int16_t> ref;
    std::vector<T> w, self, rw;
    bool near_outer = false;   // a swept cell is the partner of an outer row
};

// Host description of the pressure rows (interior cells, per axis).
struct FastPoissonGeom {
    std::vector<double> km[3], kp[3], d[3];
    std::vector<uint8_t> flag;         // padded
    std::vector<int> gcell, gidx;      // per ghost id: padded index, 8 stencil entries (-1: none)
    std::vector<double> gwself;
};

// Largest axes the dense transforms and the tridiagonal sweep take.
constexpr int FP_MAX_DENSE = 512, FP_MAX_TRI = 512;
constexpr int FP_SEG = 16;   // rows of the tridiagonal axis per thread

// A body is left to the multigrid where the cells near it (FP_LAYERS) are
// more than FP_NEAR of the fluid ones on a grid of more than FP_NEAR_GRID
// cells: the solve that ignores the body is then exact hardly anywhere, and
// takes up to 1.8 times the multigrid's iterations.  On smaller grids the
// multigrid's launches are short of work.  ms per step against the multigrid's,
// near cells over fluid ones in brackets.  FP64: a square duct in a solid
// block 48x32x32 (1.0) 2.2, 3.2; 64x40x40 (0.9) 4.5, 3.8; 72x48x48 (0.8) 5.5,
// 4.5; 144x72x72 (0.5) 15.7, 8.2; three baffles 48x32x32 (0.42) 3.3, 4.7;
// 96x48x48 (0.24) 9.3, 7.5; 144x72x72 (0.154) 28, 16; 18 square tubes 64x40x40
// (0.6) 3.9, 4.8; 96x48x48 (0.5) 6.4, 5.6; a slit 72x48x48 (0.13) 5.1, 6.2;
// two boxes 96x48x48 (0.08) 3.9, 4.5.  FP32: duct 120x64x64 (0.6) 2.3, 2.9;
// 192x96x96 (0.4) 5.7, 4.9; tubes 120x64x64 (0.4) 3.8, 3.8; 192x96x96 (0.3)
// 7.8, 6.9; baffles 120x64x64 (0.19) 4.6, 6.4; 144x72x72 (0.154) 9.3, 8.6;
// 192x96x96 (0.12) 11.9, 12.4; a slit 192x96x96 (0.05) 5.9, 7.1.
constexpr double FP_NEAR = 0.14;
template <typename T>
constexpr long long FP_NEAR_GRID = sizeof(T) == 4 ? 600000 : 131072;

// Modes of a transformed axis.  fold: the axis is mirror-symmetric, its
// modes split into ne even and no odd ones; otherwise all n are in the
// first part.  The second part starts at off (along z: a column on a vector
// boundary, and rows hold ld entries).
struct FpModes {
    int fold, ne, no, off, ld;
    int ldm[2];   // row lengths of the two parts' matrices
};

// The cells near the body, cut into patches (k_fp_patch).  Pressure
// iterations per step with 2, 3, 5, 8 and 16 sweeps: sphere 192x128x128 3.7,
// 3.5, 3.35, 3.35, 3.15; boxes 95x61x47 6.2, 6.0, 5.35, 4.75, 4.4; the
// twelve-case ensemble 5.75, 5.0, 4.5, 3.9, 3.8.  Sweeps of a patch: 16 in
// FP32, whose sweep is barriers (8 against 16, ms for 20 steps: boxes 20.1,
// 19.4; sphere 256x128x128, 15 steps, 54.0, 51.9; the others equal), 8 in
// FP64, whose sweep is arithmetic (boxes 64x48x40, 4 steps: 13.3, 14.3).
// Thinner or thicker layers and overlaps are within 3 %.
constexpr int FP_LAYERS = 3;     // fluid layers around the ghosts
template <typename T>
constexpr int FP_SWEEPS = sizeof(T) == 4 ? 16 : 8;
// Side of the cubes the cells are cut by, and the cells a patch takes beyond
// them.  FP64, bound by each SM's two multiply-adds per clock: more and
// smaller patches (a tenth of the step on boxes 64x48x40 against FP32's sizes);
// FP32 steps are within 3 % for sides of 6 and 8 and overlaps of 2 to 4.
template <typename T>
constexpr int FP_CUBE = sizeof(T) == 4 ? 8 : 5;
template <typename T>
constexpr int FP_OVERLAP = sizeof(T) == 4 ? 3 : 2;
template <typename T>
struct FpPatches {
    const int *P, *to;     // per cell: padded index, couplings ([8][ncell] padded indices, -1: none)
    int ncell;
    const int *start, *count;   // per patch: its first local cell; its red, black and ghost cells
    // Per local cell: the cell (~cell when another patch owns it), the local
    // cells it couples to ([8][nloc]; -1: outside the patch or none) and the
    // weights ([8][nloc]), the weights of the old value (ghost rows; 0 for
    // fluid ones) and of the residual.
    const int *loc;
    const int16_t *ref;
    const T *w, *self, *rw;
    int nloc;
};

template <typename T>
class FastPoisson : public Preconditioner<T> {
  public:
    ~FastPoisson() override;
    // 0: ready; 1: not for this case (the multigrid serves it: an axis is too
    // long, the transforms take more than max_ops operations, or the body is
    // near too many cells); -1: error.
    int setup(cudaStream_t s, const OpT<double> &A64, const OpT<T> &A, const FastPoissonGeom &h, double max_ops);
    void apply(cudaStream_t s, const T *r, T *z, const int *gate) override;
    bool apply_from64(cudaStream_t s, const double *r, T *z, const int *gate) override;
    bool apply_from_df(cudaStream_t s, const dfloat *r, T *z, const int *gate) override;
    int launches() const override { return launches_; }

  private:
    OpT<T> A_{};
    int ld_ = 0;                   // row length of the compact arrays
    int tri_ = 0;                  // tridiagonal axis: 0, 1, or -1
    FpModes modes_[3] = {};
    T *F_[2] = {nullptr, nullptr};
    T *fwd_[3][2] = {}, *bwd_[3][2] = {};   // per parity: (cell, mode) and (mode, cell)
    T *row0_[3] = {};              // value of cell 0 in every mode
    T *v0_ = nullptr;              // z: weight of every mode in cell 0
    T *inv_ = nullptr;             // inverse pivots (or eigenvalue sums), compact layout
    T *dtri_ = nullptr;            // widths of the tridiagonal axis
    int zero_[3] = {0, 0, 0};      // each axis's constant mode
    T *gscale_ = nullptr;          // per ghost id: 1 / max(1 - w_self, 1e-3)
    FpPatches<T> patch_{};
    T *near_val_ = nullptr;        // swept values of the cells near the body
    int npatch_ = 0, nghost_ = 0, nsolid_ = 0;
    int *solid_ = nullptr;
    int solid_partners_ = 0;       // some lie in the two layers that outer rows take their partners from
    bool near_outer_ = false;
    int launches_ = 0;
    bool plane_ = false;           // the slice kernels (fastplane.cuh) take both ends
    std::vector<void *> allocs_;
    template <typename S>
    void run(cudaStream_t s, const S *r, T *z, const int *gate);
    template <int TM, typename S>
    void run_tiled(cudaStream_t s, const S *r, T *z, const int *gate);
    template <typename S>
    void front(cudaStream_t s, const S *r, T *out, const int *gate);
    template <typename S>
    void rear(cudaStream_t s, const S *r, const T *in, T *z, const int *gate);
    template <int TM>
    void forward(cudaStream_t s, int axis, const T *in, T *out, const int *gate);
    template <int TM>
    void backward(cudaStream_t s, int axis, const T *in, T *out, const int *gate);
};

}  // namespace ibm
