// Fast diagonalisation of the pressure-Poisson rows: the BiCGSTAB
// preconditioner of the mixed modes, and of FP64 solves without a body.
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
// within three cells of a ghost repair the rows near it.
//
// The pinned row p'(0,0,0) of problems without a pressure boundary value is
// kept exactly: its fluid row's source is chosen so that the singular
// system is consistent, and the solution shifted by a constant to meet the
// pinned value.
//
// Measured (GB300, per application and BiCGSTAB iterations per step, against
// the multigrid V-cycle that served these cases before): channel
// 128x96x128 FP32 0.12 ms, 1 iteration (0.47 ms, 14); cavity 64^3 FP64
// 0.37 ms, 1 (0.31 ms, 10); sphere 192x128x128 FP32 0.17 ms, 3.7 (0.53 ms,
// 3.9); boxes 95x61x47 FP32 0.073 ms, 6.2 (0.25 ms, 4.9).  In FP64 with a
// body the transforms, bound by the FP64 pipe, cost more than the V-cycles
// they replace (3.2 GFLOP at 1.05 TFLOP/s against 1.2 ms on the sphere), so
// the multigrid stays there, and where an axis exceeds the limits below.
#pragma once

#include <vector>

#include "krylov.h"

namespace ibm {

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

template <typename T>
class FastPoisson : public Preconditioner<T> {
  public:
    ~FastPoisson() override;
    // 0: ready; 1: not for this case (the multigrid serves it); -1: error.
    int setup(cudaStream_t s, const OpT<double> &A64, const OpT<T> &A, const FastPoissonGeom &h);
    void apply(cudaStream_t s, const T *r, T *z, const int *gate) override { run(s, r, z, gate); }
    bool apply_from64(cudaStream_t s, const double *r, T *z, const int *gate) override;
    bool apply_from_df(cudaStream_t s, const dfloat *r, T *z, const int *gate) override;
    int launches() const override { return launches_; }

  private:
    OpT<T> A_{};
    int ld_ = 0;                   // nz rounded up to 4: row length of the compact arrays
    int tri_ = 0;                  // tridiagonal axis: 0, 1, or -1
    T *F_[2] = {nullptr, nullptr};
    T *fwd_[3] = {}, *bwd_[3] = {};
    int ldm_[3] = {0, 0, 0};
    T *inv_ = nullptr;             // inverse pivots (or eigenvalue sums), compact layout
    T *dtri_ = nullptr;            // widths of the tridiagonal axis
    int zero_[3] = {0, 0, 0};      // index of each axis's constant mode
    T *gscale_ = nullptr;          // per ghost id: 1 / max(1 - w_self, 1e-3)
    T *gidiv_ = nullptr, *gtmp_ = nullptr;
    int *near_ = nullptr;          // red, black and ghost cells near the body
    int nred_ = 0, nblack_ = 0, nghost_ = 0, nsolid_ = 0;
    const int *gcell_ = nullptr;
    int *solid_ = nullptr;
    bool near_outer_ = false;
    int launches_ = 0;
    std::vector<void *> allocs_;
    template <typename S>
    void run(cudaStream_t s, const S *r, T *z, const int *gate);
    void gemm_rows(cudaStream_t s, const T *a, int axis, bool forward, T *c, const int *gate);
    void gemm_cols(cudaStream_t s, const T *b, int axis, bool forward, T *c, const int *gate);
};

}  // namespace ibm
