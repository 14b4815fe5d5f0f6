// Fast-diagonalisation preconditioner of the pressure rows (fastpoisson.h).
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "fastpoisson.h"
#include "kernels.h"

namespace ibm {

#define FP_GATE(gate)                       \
    pdl_enter();                            \
    if ((gate) && *(gate) != KS_RUN) return;

template <typename T, typename S>
__device__ __forceinline__ T fp_value(S x) { return (T)x; }
template <>
__device__ __forceinline__ float fp_value<float, double>(double x) { return d2f_int(x); }
template <>
__device__ __forceinline__ float fp_value<float, dfloat>(dfloat x) { return x.hi; }
template <>
__device__ __forceinline__ double fp_value<double, dfloat>(dfloat x) { return (double)x; }

// Source of the fluid row beside a boundary from its outer row's residual
// ro: the outer value is ro / dir_o (Dirichlet) or ro (Neumann, periodic)
// plus a multiple of an interior one, which the axis matrix carries.
template <typename T>
__device__ __forceinline__ T fp_outer(const BCRow<T> &F, T ro) {
    return F.type == BCT_PRESSURE || F.type == BCT_VELPERIODIC ? ro / F.dir_o[0] : ro;
}

// ---------------------------------------------------------------- gather --
// The padded residual as the compact source coeffsum r of the separable
// system: 0 on solid rows and the pinned row, scaled on ghost rows, with
// the outer rows' residuals folded into the rows beside them.  Padding
// columns (k >= nz) are 0.  Bound by its bytes (8 read, 4 written per cell
// from double-float residuals).  Grid (ld / 32, ny / 8, nx / 4).
constexpr int FP_GPLANES = 4;

template <typename T, typename S>
__global__ void __launch_bounds__(256)
k_fp_gather(const OpT<T> c, const S *__restrict__ r, T *__restrict__ f, const int ld, const int body,
            const T *__restrict__ gscale, const int *gate) {
    FP_GATE(gate);
    const Grid &g = c.g;
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
    if (k >= ld || j >= g.ny) return;
    const bool in = k < g.nz;
    const int kk = min(k, g.nz - 1);
    const T ksyz = c.ks[1][j + 2] + c.ks[2][kk + 2];
    const bool edge = j == 0 || j == g.ny - 1 || kk == 0 || kk == g.nz - 1;
#pragma unroll
    for (int p = 0; p < FP_GPLANES; p++) {
        const int i = blockIdx.z * FP_GPLANES + p;
        if (i >= g.nx) break;
        const long long P = cidx(g, i, j, kk);
        T v = (c.ks[0][i + 2] + ksyz) * fp_value<T, S>(r[P]);
        if (body) {
            const uint8_t fl = c.flag[P];
            if (fl == GHOST) v *= gscale[c.gid[P]];
            else if (fl != FLUID) v = 0;
        }
        if (edge || i == 0 || i == g.nx - 1) {
            if (!body || c.flag[P] == FLUID) {
                if (i == 0) v += c.km[0][2] * fp_outer(c.bc[F_W], fp_value<T, S>(r[P - g.sx]));
                if (i == g.nx - 1) v += c.kp[0][i + 2] * fp_outer(c.bc[F_E], fp_value<T, S>(r[P + g.sx]));
                if (j == 0) v += c.km[1][2] * fp_outer(c.bc[F_S], fp_value<T, S>(r[P - g.sy]));
                if (j == g.ny - 1) v += c.kp[1][j + 2] * fp_outer(c.bc[F_N], fp_value<T, S>(r[P + g.sy]));
                if (kk == 0) v += c.km[2][2] * fp_outer(c.bc[F_D], fp_value<T, S>(r[P - 1]));
                if (kk == g.nz - 1) v += c.kp[2][kk + 2] * fp_outer(c.bc[F_U], fp_value<T, S>(r[P + 1]));
            }
            if (c.p_singular && P == c.pinned) v = 0;
        }
        f[((long long)i * g.ny + j) * ld + k] = in ? v : (T)0;
    }
}

// ------------------------------------------------------------ transforms --
// C = A B for row-major operands in tiles of TM x TM, 64 threads with an
// R x R register tile each (as 2 x 2 sub-tiles, so that shared-memory reads
// are conflict-free 16-byte ones or broadcasts), the k loop in steps of 16
// through two shared-memory buffers with the next step's loads in flight.
// TA = false: A(m, k) with k contiguous (the data, when the contiguous axis
// is transformed); TA = true: A given as its transpose, (k, m) with m
// contiguous (the axis matrix, applied to another axis).  A and C or B and
// C advance by their batch strides.  out (with SCATTER): row m is the grid
// line (i, j), written to the padded array, shifted so that the pinned cell
// takes its residual's value.  Bound by the FP32 (FP64) multiply-add pipe.
template <typename T>
struct FpTile;
template <>
struct FpTile<float> {
    static constexpr int TM = 64, R = 8, V = 4;
};
template <>
struct FpTile<double> {
    static constexpr int TM = 32, R = 4, V = 2;
};
constexpr int FP_TK = 16;

template <typename T>
struct FpGemm {
    const T *a, *b;
    T *c;
    int M, N, K;
    int lda, ldb, ldc;
    long long sa, sb, sc;   // batch strides
};

template <typename T, typename S>
struct FpScatter {
    Grid g;
    FastDiv dny;
    const S *r;             // residual (pinned shift)
    const T *brow;          // row 0 of the backward transform's result basis: V(0, .)
    long long pinned;
    int singular;
};

template <typename T, bool TA, bool SCATTER, typename S>
__global__ void __launch_bounds__(64)
k_fp_gemm(const FpGemm<T> p, const FpScatter<T, S> sc, const int *gate) {
    FP_GATE(gate);
    constexpr int TM = FpTile<T>::TM, R = FpTile<T>::R, V = FpTile<T>::V, H = TM / 2, R2 = R / 2;
    constexpr int PITCH = TA ? TM : TM + V;
    constexpr int NQ = TM * FP_TK / V / 64;   // vector loads per thread and operand
    struct alignas(16) Vec {
        T v[V];
    };
    __shared__ alignas(16) T As[2][FP_TK][PITCH];
    __shared__ alignas(16) T Bs[2][FP_TK][TM];
    const T *A = p.a + blockIdx.z * p.sa, *B = p.b + blockIdx.z * p.sb;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TM;
    const int t = threadIdx.x, tx = t & 7, ty = t >> 3;
    Vec ra[NQ], rb[NQ];
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int e = t + 64 * q;
            {
                constexpr int PER = TM / V;
                const int k = k0 + e / PER, n = n0 + (e % PER) * V;
                if (k < p.K && n < p.N) rb[q] = *reinterpret_cast<const Vec *>(B + (long long)k * p.ldb + n);
                else rb[q] = Vec{};
                if (TA) {
                    const int m = m0 + (e % PER) * V;
                    if (k < p.K && m < p.lda) ra[q] = *reinterpret_cast<const Vec *>(A + (long long)k * p.lda + m);
                    else ra[q] = Vec{};
                }
            }
            if (!TA) {
                constexpr int PER = FP_TK / V;
                const int m = m0 + e / PER, k = k0 + (e % PER) * V;
                if (m < p.M && k < p.lda) ra[q] = *reinterpret_cast<const Vec *>(A + (long long)m * p.lda + k);
                else ra[q] = Vec{};
            }
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int e = t + 64 * q;
            constexpr int PER = TM / V;
            *reinterpret_cast<Vec *>(&Bs[buf][e / PER][(e % PER) * V]) = rb[q];
            if (TA) {
                *reinterpret_cast<Vec *>(&As[buf][e / PER][(e % PER) * V]) = ra[q];
            } else {
                constexpr int PK = FP_TK / V;
#pragma unroll
                for (int l = 0; l < V; l++) As[buf][(e % PK) * V + l][e / PK] = ra[q].v[l];
            }
        }
    };
    T acc[R][R];
#pragma unroll
    for (int x = 0; x < R; x++)
#pragma unroll
        for (int y = 0; y < R; y++) acc[x][y] = 0;
    T shift = 0;
    if (SCATTER && sc.singular) {
        // z(0,0,0) of the unshifted solution: one line's product, by every
        // block for itself.
        __shared__ T red[2];
        T s = 0;
        for (int q = t; q < p.K; q += 64) s += A[q] * sc.brow[(long long)q * p.ldb];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((t & 31) == 0) red[t >> 5] = s;
        __syncthreads();
        shift = fp_value<T, S>(sc.r[sc.pinned]) - (red[0] + red[1]);
    }
    load(0);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < p.K; k0 += FP_TK) {
        const bool more = k0 + FP_TK < p.K;
        if (more) load(k0 + FP_TK);
#pragma unroll
        for (int k = 0; k < FP_TK; k++) {
            T av[R], bv[R];
#pragma unroll
            for (int h = 0; h < 2; h++) {
#pragma unroll
                for (int l = 0; l < R2; l += V) {
                    *reinterpret_cast<Vec *>(&av[h * R2 + l]) = *reinterpret_cast<const Vec *>(&As[buf][k][h * H + ty * R2 + l]);
                    *reinterpret_cast<Vec *>(&bv[h * R2 + l]) = *reinterpret_cast<const Vec *>(&Bs[buf][k][h * H + tx * R2 + l]);
                }
            }
#pragma unroll
            for (int x = 0; x < R; x++)
#pragma unroll
                for (int y = 0; y < R; y++) acc[x][y] += av[x] * bv[y];
        }
        if (more) {
            store(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
#pragma unroll
    for (int x = 0; x < R; x++) {
        const int m = m0 + (x / R2) * H + ty * R2 + x % R2;
        if (m >= p.M) continue;
        if (SCATTER) {
            const int i = (int)fdiv(sc.dny, (uint32_t)m), j = m - i * sc.g.ny;
            T *row = p.c + cidx(sc.g, i, j, 0);
            const bool pair = ((sc.g.sy | sc.g.sx) & 1) == 0;
#pragma unroll
            for (int y = 0; y < R; y += 2) {
                const int n = n0 + (y / R2) * H + tx * R2 + y % R2;
                struct alignas(2 * sizeof(T)) Two {
                    T v[2];
                };
                if (pair && n + 1 < sc.g.nz) {
                    *reinterpret_cast<Two *>(row + n) = Two{{acc[x][y] + shift, acc[x][y + 1] + shift}};
                } else {
                    if (n < sc.g.nz) row[n] = acc[x][y] + shift;
                    if (n + 1 < sc.g.nz) row[n + 1] = acc[x][y + 1] + shift;
                }
            }
        } else {
            T *row = p.c + blockIdx.z * p.sc + (long long)m * p.ldc;
#pragma unroll
            for (int y = 0; y < R; y += V) {
                const int n = n0 + (y / R2) * H + tx * R2 + y % R2;
                if (n < p.N) {
                    Vec o;
#pragma unroll
                    for (int l = 0; l < V; l++) o.v[l] = acc[x][y + l];
                    *reinterpret_cast<Vec *>(row + n) = o;
                }
            }
        }
    }
}

// ------------------------------------------------- tridiagonal / diagonal --
// Pinned problems: the source c of the pinned cell that makes the singular
// system consistent, from the constant mode's line (n values, stride st,
// widths w): c u0 w0 = -sum w f, u0 the constant mode's part of a unit
// source there.  Computed by every block for itself.
template <typename T>
struct FpPin {
    int singular;
    const T *w;             // widths along the tridiagonal axis (null: one value)
    long long zero;         // compact index of the constant mode's line
    const T *f1, *f2;       // row 0 of the two forward transforms (value of cell 0 in mode m)
    int z1, z2;             // constant modes
};

template <typename T>
__device__ __forceinline__ T fp_pin(const FpPin<T> &pin, const T *f, int n, long long st, T *smem) {
    const int tid = threadIdx.y * 32 + threadIdx.x;
    T s = 0;
    for (int q = tid; q < n; q += blockDim.x * blockDim.y) s += (pin.w ? pin.w[q] : (T)1) * f[pin.zero + q * st];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) smem[threadIdx.y] = s;
    __syncthreads();
    s = 0;
    for (int q = 0; q < (int)blockDim.y; q++) s += smem[q];
    __syncthreads();
    return -s / ((pin.w ? pin.w[0] : (T)1) * pin.f1[pin.z1] * pin.f2[pin.z2]);
}

// (A_tri + lambda) t = f along the tridiagonal axis for every mode.  With the inverse pivots iv: g_i = iv_i (f_i + km_i g_(i-1)), then
// t_i = g_i + iv_i kp_i t_(i+1).  A thread keeps FP_SEG rows of one mode in
// registers (every load in flight at once, coalesced across the modes); the
// two recurrences cross the block's threads by composing each segment's
// affine map through shared memory, so the serial chain is FP_SEG rows and
// the number of segments instead of n.  Block (32 modes, segments); grid
// (ld / 32, outer lines).  Bound by its bytes (f and iv read, t written).
// MAXT: the block's bound (512 threads keep an FP64 thread's rows in
// registers; axes over 256 cells take 1024).
template <typename T, int MAXT>
__global__ void __launch_bounds__(MAXT)
k_fp_tri(const T *__restrict__ iv, const T *__restrict__ km, const T *__restrict__ kp,
         const int n, const long long st, const long long outer, const int ld, const FpPin<T> pin, const T *fin,
         T *out, const int *gate) {
    FP_GATE(gate);
    __shared__ T sa[32][33], sh[32][33];
    const int c = blockIdx.x * 32 + threadIdx.x, seg = threadIdx.y, ns = blockDim.y;
    const long long base = blockIdx.y * outer + min(c, ld - 1);
    const int i0 = seg * FP_SEG;
    T h[FP_SEG], v[FP_SEG];
#pragma unroll
    for (int q = 0; q < FP_SEG; q++) {
        const bool ok = i0 + q < n;
        h[q] = ok ? fin[base + (i0 + q) * st] : (T)0;
        v[q] = ok ? iv[base + (i0 + q) * st] : (T)0;
    }
    if (pin.singular) {
        const T cc = fp_pin(pin, fin, n, st, &sa[0][0]);
        if (seg == 0) h[0] += cc * pin.f1[blockIdx.y] * pin.f2[min(c, ld - 1)];
    }
    // forward: local recurrence from 0 and the segment's multiplier
    T a = 1, g = 0;
#pragma unroll
    for (int q = 0; q < FP_SEG; q++) {
        const T m = i0 + q < n ? km[i0 + q] * v[q] : (T)0;
        g = v[q] * h[q] + m * g;
        a *= m;
    }
    sa[seg][threadIdx.x] = a;
    sh[seg][threadIdx.x] = g;
    __syncthreads();
    g = 0;
    for (int q = 0; q < seg; q++) g = sh[q][threadIdx.x] + sa[q][threadIdx.x] * g;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < FP_SEG; q++) {
        const T m = i0 + q < n ? km[i0 + q] * v[q] : (T)0;
        g = v[q] * h[q] + m * g;
        h[q] = g;
    }
    // backward
    a = 1;
    g = 0;
#pragma unroll
    for (int q = FP_SEG - 1; q >= 0; q--) {
        const T m = i0 + q < n ? kp[i0 + q] * v[q] : (T)0;
        g = h[q] + m * g;
        a *= m;
    }
    sa[seg][threadIdx.x] = a;
    sh[seg][threadIdx.x] = g;
    __syncthreads();
    g = 0;
    for (int q = ns - 1; q > seg; q--) g = sh[q][threadIdx.x] + sa[q][threadIdx.x] * g;
#pragma unroll
    for (int q = FP_SEG - 1; q >= 0; q--) {
        const T m = i0 + q < n ? kp[i0 + q] * v[q] : (T)0;
        g = h[q] + m * g;
        if (i0 + q < n && c < ld) out[base + (i0 + q) * st] = g;
    }
}

// All three axes transformed: divide by the eigenvalue sums.  Block (32, 8)
// over one compact plane, grid (ld / 32, ny / 8, nx).
template <typename T>
__global__ void __launch_bounds__(256)
k_fp_diag(const T *__restrict__ iv, const int ny, const int ld, const FpPin<T> pin, const T *__restrict__ f0,
          const T *fin, T *out, const int *gate) {
    FP_GATE(gate);
    __shared__ T sm[32];
    const int c = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    T cc = 0;
    if (pin.singular) cc = fp_pin(pin, fin, 1, 0, sm) / f0[0];
    if (c >= ld || j >= ny) return;
    const long long q = ((long long)i * ny + j) * ld + c;
    T v = fin[q];
    if (pin.singular) v += cc * f0[1 + i] * pin.f1[j] * pin.f2[c];
    out[q] = v * iv[q];
}

// Inverse pivots of every mode along the tridiagonal axis, factored in
// FP64; the last pivot of the constant mode of a pinned problem (exactly
// singular) is replaced by 0.  One thread per mode (set-up).
template <typename T>
__global__ void k_fp_pivots(const double *__restrict__ diag, const double *__restrict__ km,
                            const double *__restrict__ kp, const double *__restrict__ l1, const double *__restrict__ l2,
                            T *iv, const int n, const long long st, const long long outer, const int n1, const int n2,
                            const int ld, const int z1, const int z2) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, o = blockIdx.y;
    if (c >= ld) return;
    const long long base = o * outer + c;
    if (c >= n2) {
        for (int i = 0; i < n; i++) iv[base + i * st] = 0;
        return;
    }
    const double lam = l1[o] + l2[c];
    double u = 0;
    for (int i = 0; i < n; i++) {
        double p = diag[i] + lam;
        if (i > 0) p -= km[i] * kp[i - 1] * u;
        u = (i == n - 1 && o == z1 && c == z2) ? 0.0 : 1.0 / p;
        iv[base + i * st] = (T)u;
    }
}

template <typename T>
__global__ void k_fp_sums(const double *__restrict__ l0, const double *__restrict__ l1, const double *__restrict__ l2,
                          T *iv, const int ny, const int nz, const int ld, const int z0, const int z1, const int z2) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
    if (c >= ld) return;
    const bool zero = i == z0 && j == z1 && c == z2;
    iv[((long long)i * ny + j) * ld + c] = c >= nz || zero ? (T)0 : (T)(1.0 / (l0[i] + l1[j] + l2[c]));
}

// ------------------------------------------------------- outer rows, body --
// Outer rows solved for the outer values, each through its chain of
// partners down to an interior cell (as the multigrid's outer pass), and
// the identity rows of solid cells.
template <typename T, typename S>
__global__ void __launch_bounds__(256)
k_fp_edges(const OpT<T> c, const S *__restrict__ r, T *z, const int *__restrict__ outer, const int nout,
           const int *__restrict__ solid, const int nsolid, const int *gate) {
    FP_GATE(gate);
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (t >= nout) {
        if (t - nout < nsolid) {
            const int P = solid[t - nout];
            z[P] = fp_value<T, S>(r[P]);
        }
        return;
    }
    long long chain[3];
    int face[3], layer[3], n = 0;
    long long Q = outer[t];
    while (true) {
        int i, j, k, L;
        cijk_fast(c.g, c.fdx, c.fdy, Q, i, j, k);
        const int f = owner_face(c.g, i, j, k, L);
        if (f < 0 || n == 3) break;
        chain[n] = Q;
        face[n] = f;
        layer[n++] = L;
        if (c.bc[f].type == BCT_PERIODIC) {
            Q = periodic_image(c.g, i, j, k);
        } else {
            const int axis = face_axis(f);
            const long long s = axis == 0 ? c.g.sx : axis == 1 ? c.g.sy : 1;
            Q += (2 * L - 1) * (face_low(f) ? s : -s);
        }
    }
    T v = z[Q];
    for (int q = n - 1; q >= 0; q--) {
        const BCRow<T> &F = c.bc[face[q]];
        const T rv = fp_value<T, S>(r[chain[q]]);
        if (F.type == BCT_PRESSURE || F.type == BCT_VELPERIODIC)
            v = (rv - F.dir_m[layer[q] - 1] * v) / F.dir_o[layer[q] - 1];
        else
            v = rv + v;
    }
    z[outer[t]] = v;
}

// Gauss-Seidel sweeps over the cells near the body (red fluid cells, black
// ones, then the ghost rows Jacobi-style through tmp), all in one launch of
// one thread-block cluster whose barrier separates the passes: the lists
// hold some thousands of cells, so a pass is one latency, and a launch per
// pass would cost more than the pass.  Values cross the cluster's blocks
// through L2 (ld/st.cg).
constexpr int FP_CLUSTER = 8, FP_CT = 1024;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

template <typename T, typename S>
__global__ void __cluster_dims__(FP_CLUSTER, 1, 1) __launch_bounds__(FP_CT)
k_fp_near(const OpT<T> c, const S *__restrict__ r, T *z, const int *__restrict__ near, const int nred,
          const int nblack, const int *__restrict__ gcell, const int ng, const T *__restrict__ gidiv, T *tmp,
          const int sweeps, const int *gate) {
    FP_GATE(gate);
    const int t0 = blockIdx.x * FP_CT + threadIdx.x;
    constexpr int NT = FP_CLUSTER * FP_CT;
    const long long sx = c.g.sx, sy = c.g.sy;
    for (int s = 0; s < sweeps; s++) {
        for (int col = 0; col < 2; col++) {
            const int lo = col ? nred : 0, hi = col ? nred + nblack : nred;
            for (int q = lo + t0; q < hi; q += NT) {
                const int P = near[q];
                int i, j, k;
                cijk_fast(c.g, c.fdx, c.fdy, P, i, j, k);
                const T zw = __ldcg(z + P - sx), ze = __ldcg(z + P + sx), zs = __ldcg(z + P - sy),
                        zn = __ldcg(z + P + sy), zd = __ldcg(z + P - 1), zu = __ldcg(z + P + 1);
                const T nb = sum6(c.km[0][i + 2], zw, c.kp[0][i + 2], ze, c.km[1][j + 2], zs, c.kp[1][j + 2], zn,
                                  c.km[2][k + 2], zd, c.kp[2][k + 2], zu);
                __stcg(z + P, fp_value<T, S>(r[P]) + c.dinv[P] * nb);
            }
            cluster_barrier();
        }
        for (int g = t0; g < ng; g += NT) {
            const int P = gcell[g];
            T sum = 0;
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const int q = c.gidx[8 * g + e];
                if (q >= 0) sum += c.gw[8 * g + e] * __ldcg(z + q);
            }
            const T zp = __ldcg(z + P);
            tmp[g] = zp + (fp_value<T, S>(r[P]) + sum - ((T)1 - c.gwself[g]) * zp) * gidiv[g];
        }
        cluster_barrier();
        for (int g = t0; g < ng; g += NT) __stcg(z + gcell[g], tmp[g]);   // this thread's own tmp entries
        cluster_barrier();
    }
}

// ----------------------------------------------------------------- set-up --
namespace {

// Eigenvalues w and eigenvectors (row m of q belongs to w[m]) of the
// symmetric tridiagonal matrix with diagonal w and off-diagonals e (e[i]
// couples i and i + 1), the rotations accumulated onto the rows q holds on
// entry.  Shifted QR steps A - mu = Q R, A <- R Q + mu on the trailing
// unreduced block, R and R Q formed explicitly from the Givens rotations
// (Golub and Van Loan, Matrix Computations, section 8.3); a rotation acts on
// two contiguous rows of q.
bool tridiag_eigen(int n, std::vector<double> &w, std::vector<double> e, std::vector<double> &q) {
    auto small = [&](int i) { return std::fabs(e[i]) <= 1e-16 * (std::fabs(w[i]) + std::fabs(w[i + 1])); };
    std::vector<double> c(n), s(n), d(n), u(n);
    int hi = n - 1;
    for (int it = 0; hi > 0; it++) {
        if (it > 60 * n) return false;
        if (small(hi - 1)) {
            e[--hi] = 0.0;
            continue;
        }
        int lo = hi - 1;
        while (lo > 0 && !small(lo - 1)) lo--;
        // Wilkinson's shift: the eigenvalue of the trailing 2 x 2 block
        // nearer its last entry.
        const double h = (w[hi - 1] - w[hi]) / 2, b = e[hi - 1], rad = std::sqrt(h * h + b * b);
        const double mu = w[hi] - b * b / (h >= 0 ? h + rad : h - rad);
        // R: diagonal d, first superdiagonal u.
        double x = w[lo] - mu, y = e[lo];
        for (int i = lo; i < hi; i++) {
            const double r = std::sqrt(x * x + e[i] * e[i]), a1 = w[i + 1] - mu;
            c[i] = r > 0 ? x / r : 1.0;
            s[i] = r > 0 ? e[i] / r : 0.0;
            d[i] = r;
            u[i] = c[i] * y + s[i] * a1;
            x = c[i] * a1 - s[i] * y;
            if (i + 1 < hi) y = c[i] * e[i + 1];
        }
        d[hi] = x;
        for (int i = lo; i < hi; i++) {
            w[i] = (i > lo ? c[i - 1] : 1.0) * c[i] * d[i] + s[i] * u[i] + mu;
            e[i] = s[i] * d[i + 1];
        }
        w[hi] = c[hi - 1] * d[hi] + mu;
        for (int i = lo; i < hi; i++) {
            double *q0 = &q[(size_t)i * n], *q1 = q0 + n;
            const double ci = c[i], si = s[i];
            for (int k = 0; k < n; k++) {
                const double t = q0[k];
                q0[k] = ci * t + si * q1[k];
                q1[k] = ci * q1[k] - si * t;
            }
        }
    }
    return true;
}

// Eigenvalues and eigenvectors (rows of q) of the dense symmetric matrix a
// (row-major): Householder reduction to tridiagonal form, then
// the QR steps above.
bool dense_eigen(int n, std::vector<double> a, std::vector<double> &w, std::vector<double> &q) {
    // q starts as the identity; each reflector H = I - 2 v v^T (v on rows
    // c+1 .. n-1) is applied as A <- H A H and Q <- H Q (rows of q are the
    // rows of the accumulated H ... H).
    q.assign((size_t)n * n, 0.0);
    for (int i = 0; i < n; i++) q[(size_t)i * n + i] = 1;
    std::vector<double> v(n), p(n);
    for (int c = 0; c + 2 < n; c++) {
        double s2 = 0;
        for (int i = c + 1; i < n; i++) s2 += a[(size_t)i * n + c] * a[(size_t)i * n + c];
        const double head = a[(size_t)(c + 1) * n + c];
        const double alpha = head > 0 ? -std::sqrt(s2) : std::sqrt(s2);
        double vn = 0;
        for (int i = c + 1; i < n; i++) {
            v[i] = a[(size_t)i * n + c] - (i == c + 1 ? alpha : 0.0);
            vn += v[i] * v[i];
        }
        if (vn == 0.0) continue;
        const double sc = 1 / std::sqrt(vn);
        for (int i = c + 1; i < n; i++) v[i] *= sc;
        double vp = 0;
        for (int i = c; i < n; i++) {
            double t = 0;
            for (int k = c + 1; k < n; k++) t += a[(size_t)i * n + k] * v[k];
            p[i] = t;
        }
        for (int i = c + 1; i < n; i++) vp += v[i] * p[i];
        v[c] = 0;
        for (int i = c; i < n; i++)
            for (int k = c; k < n; k++)
                a[(size_t)i * n + k] += -2 * (v[i] * p[k] + p[i] * v[k]) + 4 * vp * v[i] * v[k];
        for (int k = 0; k < n; k++) p[k] = 0;
        for (int i = c + 1; i < n; i++)
            for (int k = 0; k < n; k++) p[k] += v[i] * q[(size_t)i * n + k];
        for (int i = c + 1; i < n; i++)
            for (int k = 0; k < n; k++) q[(size_t)i * n + k] -= 2 * v[i] * p[k];
    }
    w.resize(n);
    std::vector<double> e(n, 0.0);
    for (int i = 0; i < n; i++) w[i] = a[(size_t)i * n + i];
    for (int i = 0; i + 1 < n; i++) e[i] = a[(size_t)(i + 1) * n + i];
    return tridiag_eigen(n, w, e, q);
}

bool dirichlet_face(int type) { return type == BCT_PRESSURE || type == BCT_VELPERIODIC; }

}  // namespace

template <typename T>
FastPoisson<T>::~FastPoisson() {
    for (void *p : allocs_) cudaFree(p);
}

template <typename T>
int FastPoisson<T>::setup(cudaStream_t s, const OpT<double> &A64, const OpT<T> &A, const FastPoissonGeom &h) {
    const Grid &g = A.g;
    const int n[3] = {g.nx, g.ny, g.nz};
    const int lo[3] = {F_W, F_S, F_D}, hi[3] = {F_E, F_N, F_U};
    bool per[3];
    for (int a = 0; a < 3; a++) per[a] = A64.bc[lo[a]].type == BCT_PERIODIC;
    // The tridiagonal axis: the longer of x and y that does not wrap.
    tri_ = -1;
    for (int a = 0; a < 2; a++)
        if (!per[a] && n[a] <= FP_MAX_TRI && (tri_ < 0 || n[a] > n[tri_])) tri_ = a;
    for (int a = 0; a < 3; a++)
        if (n[a] < 3 || (a != tri_ && n[a] > FP_MAX_DENSE)) return 1;
    A_ = A;
    ld_ = (n[2] + 3) & ~3;
    nghost_ = (int)h.gcell.size();
    gcell_ = nullptr;
    bool ok = true;
    auto put = [&](const void *src, size_t bytes) -> void * {
        void *p = nullptr;
        if (!ok || cudaMalloc(&p, std::max<size_t>(bytes, 16)) != cudaSuccess) {
            ok = false;
            return nullptr;
        }
        allocs_.push_back(p);
        if (src) ok = cudaMemcpyAsync(p, src, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess &&
                      cudaStreamSynchronize(s) == cudaSuccess;
        return p;
    };
    std::vector<double> lam[3], diag;
    std::vector<T> row0[3];
    for (int a = 0; a < 3 && ok; a++) {
        const int N = n[a];
        const std::vector<double> &km = h.km[a], &kp = h.kp[a], &d = h.d[a];
        std::vector<double> dg(N);
        for (int i = 0; i < N; i++) dg[i] = km[i] + kp[i];
        if (!per[a]) {
            const BCRow<double> &L = A64.bc[lo[a]], &U = A64.bc[hi[a]];
            dg[0] += dirichlet_face(L.type) ? km[0] * (L.dir_m[0] / L.dir_o[0]) : -km[0];
            dg[N - 1] += dirichlet_face(U.type) ? kp[N - 1] * (U.dir_m[0] / U.dir_o[0]) : -kp[N - 1];
        }
        if (a == tri_) {
            diag = dg;
            continue;
        }
        std::vector<double> w = dg, e(N, 0.0), q;
        for (int i = 0; i + 1 < N; i++) e[i] = -std::sqrt(kp[i] * km[i + 1]);
        bool good;
        if (per[a]) {
            std::vector<double> m((size_t)N * N, 0.0);
            for (int i = 0; i < N; i++) {
                m[(size_t)i * N + i] = dg[i];
                if (i + 1 < N) m[(size_t)i * N + i + 1] = m[(size_t)(i + 1) * N + i] = e[i];
            }
            m[N - 1] = m[(size_t)(N - 1) * N] = -std::sqrt(km[0] * kp[N - 1]);
            good = dense_eigen(N, m, w, q);
        } else {
            q.assign((size_t)N * N, 0.0);
            for (int i = 0; i < N; i++) q[(size_t)i * N + i] = 1;
            good = tridiag_eigen(N, w, e, q);
        }
        if (!good) return 1;
        int z = 0;
        for (int i = 1; i < N; i++)
            if (std::fabs(w[i]) < std::fabs(w[z])) z = i;
        zero_[a] = z;
        if (A.p_singular) w[z] = 0.0;   // the constants
        lam[a] = w;
        const int ld = (N + 3) & ~3;
        ldm_[a] = ld;
        std::vector<T> f((size_t)N * ld, (T)0), b((size_t)N * ld, (T)0);
        for (int m = 0; m < N; m++)
            for (int i = 0; i < N; i++) {
                const double sd = std::sqrt(d[i]), v = q[(size_t)m * N + i];
                f[(size_t)i * ld + m] = (T)(v * sd);
                b[(size_t)m * ld + i] = (T)(v / sd);
            }
        row0[a].assign(f.begin(), f.begin() + ld);
        fwd_[a] = (T *)put(f.data(), sizeof(T) * f.size());
        bwd_[a] = (T *)put(b.data(), sizeof(T) * b.size());
    }
    const size_t cells = (size_t)n[0] * n[1] * ld_;
    for (T *&f : F_) f = (T *)put(nullptr, sizeof(T) * cells);
    inv_ = (T *)put(nullptr, sizeof(T) * cells);
    if (!ok) return -1;
    double *dl[3] = {nullptr, nullptr, nullptr}, *dk[3] = {nullptr, nullptr, nullptr};
    auto tmp = [&](const std::vector<double> &v) {
        double *p = (double *)put(v.data(), sizeof(double) * v.size());
        return p;
    };
    for (int a = 0; a < 3; a++)
        if (a != tri_) dl[a] = tmp(lam[a]);
    if (!ok) return -1;
    if (tri_ >= 0) {
        const int N = n[tri_], o = tri_ == 0 ? 1 : 0;
        dk[0] = tmp(diag);
        dk[1] = tmp(h.km[tri_]);
        dk[2] = tmp(h.kp[tri_]);
        std::vector<T> w(N);
        for (int i = 0; i < N; i++) w[i] = (T)h.d[tri_][i];
        dtri_ = (T *)put(w.data(), sizeof(T) * N);
        if (!ok) return -1;
        const long long st = tri_ == 0 ? (long long)n[1] * ld_ : ld_, outer = tri_ == 0 ? ld_ : (long long)n[1] * ld_;
        const bool sing = A.p_singular != 0;
        k_fp_pivots<T><<<dim3((ld_ + 127) / 128, n[o]), 128, 0, s>>>(dk[0], dk[1], dk[2], dl[o], dl[2], inv_, N, st, outer,
                                                                      n[o], n[2], ld_, sing ? zero_[o] : -1,
                                                                      sing ? zero_[2] : -1);
    } else {
        // f0: the x transform's constant-mode value of cell 0, then row 0.
        std::vector<T> w(1 + ldm_[0]);
        w[0] = row0[0][zero_[0]];
        std::copy(row0[0].begin(), row0[0].end(), w.begin() + 1);
        dtri_ = (T *)put(w.data(), sizeof(T) * w.size());
        if (!ok) return -1;
        const bool sing = A.p_singular != 0;
        k_fp_sums<T><<<dim3((ld_ + 127) / 128, n[1], n[0]), 128, 0, s>>>(dl[0], dl[1], dl[2], inv_, n[1], n[2], ld_,
                                                                         sing ? zero_[0] : -1, zero_[1], zero_[2]);
    }
    // Solid cells, and the cells near the body.
    std::vector<int> solid;
    const long long st[3] = {g.sx, g.sy, 1};
    for (int i = 0; i < n[0]; i++)
        for (int j = 0; j < n[1]; j++) {
            const long long P0 = cidx(g, i, j, 0);
            for (int k = 0; k < n[2]; k++)
                if (h.flag[P0 + k] == SOLID) solid.push_back((int)(P0 + k));
        }
    nsolid_ = (int)solid.size();
    solid_ = (int *)put(solid.data(), sizeof(int) * solid.size());
    if (nghost_ > 0) {
        std::vector<uint8_t> mark(g.ncell, 0);
        std::vector<int> cur = h.gcell, all;
        for (int P : cur) mark[P] = 1;
        auto add = [&](long long Q, std::vector<int> &to) {
            int i, j, k;
            cijk(g, Q, i, j, k);
            if (i < 0 || i >= n[0] || j < 0 || j >= n[1] || k < 0 || k >= n[2] || mark[Q] || h.flag[Q] != FLUID) return;
            if (A.p_singular && Q == A.pinned) return;
            mark[Q] = 1;
            to.push_back((int)Q);
        };
        for (int layer = 0; layer < 3; layer++) {
            std::vector<int> next;
            if (layer == 0)
                for (int q : h.gidx)
                    if (q >= 0) add(q, next);
            for (int P : cur)
                for (int a = 0; a < 3; a++) {
                    add(P - st[a], next);
                    add(P + st[a], next);
                }
            all.insert(all.end(), next.begin(), next.end());
            cur = next;
        }
        std::sort(all.begin(), all.end());
        std::vector<int> red, black;
        for (int P : all) {
            int i, j, k;
            cijk(g, P, i, j, k);
            ((i + j + k) & 1 ? black : red).push_back(P);
            near_outer_ = near_outer_ || i < 2 || i >= n[0] - 2 || j < 2 || j >= n[1] - 2 || k < 2 || k >= n[2] - 2;
        }
        nred_ = (int)red.size();
        nblack_ = (int)black.size();
        red.insert(red.end(), black.begin(), black.end());
        near_ = (int *)put(red.data(), sizeof(int) * red.size());
        gcell_ = (const int *)put(h.gcell.data(), sizeof(int) * nghost_);
        // Divisors of the ghost rows' relaxation (as the multigrid's) and
        // the scale of their sources.
        std::vector<double> gw(8 * (size_t)nghost_);
        cudaMemcpyAsync(gw.data(), A64.gw, sizeof(double) * gw.size(), cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
        std::vector<T> sc(nghost_), dv(nghost_);
        for (int q = 0; q < nghost_; q++) {
            double off = 0;
            for (int e = 0; e < 8; e++) {
                const int P = h.gidx[8 * (size_t)q + e];
                if (P >= 0 && h.flag[P] == GHOST) off += std::fabs(gw[8 * (size_t)q + e]);
            }
            const double dgl = 1.0 - h.gwself[q];
            sc[q] = (T)(1.0 / std::max(dgl, 1e-3));
            dv[q] = (T)(1.0 / std::max({dgl, 2.0 * off, 1e-3}));
        }
        gscale_ = (T *)put(sc.data(), sizeof(T) * nghost_);
        gidiv_ = (T *)put(dv.data(), sizeof(T) * nghost_);
        gtmp_ = (T *)put(nullptr, sizeof(T) * nghost_);
    }
    if (!ok) return -1;
    return cudaStreamSynchronize(s) == cudaSuccess ? 0 : -1;
}

// ------------------------------------------------------------ application --
// The contiguous axis: rows of `a` times the axis matrix.
template <typename T>
void FastPoisson<T>::gemm_rows(cudaStream_t s, const T *a, int axis, bool forward, T *c, const int *gate) {
    constexpr int TM = FpTile<T>::TM;
    const Grid &g = A_.g;
    FpGemm<T> p{a, forward ? fwd_[axis] : bwd_[axis], c, g.nx * g.ny, ld_, g.nz, ld_, ldm_[axis], ld_, 0, 0, 0};
    launch_pdl(k_fp_gemm<T, false, false, T>, dim3((p.N + TM - 1) / TM, (p.M + TM - 1) / TM), 64, 0, s, p,
               FpScatter<T, T>{}, gate);
}

// x or y: the axis matrix times the lines of `b`.
template <typename T>
void FastPoisson<T>::gemm_cols(cudaStream_t s, const T *b, int axis, bool forward, T *c, const int *gate) {
    constexpr int TM = FpTile<T>::TM;
    const Grid &g = A_.g;
    const T *w = forward ? fwd_[axis] : bwd_[axis];
    const long long plane = (long long)g.ny * ld_;
    FpGemm<T> p;
    if (axis == 0) p = FpGemm<T>{w, b, c, g.nx, (int)plane, g.nx, ldm_[0], (int)plane, (int)plane, 0, 0, 0};
    else p = FpGemm<T>{w, b, c, g.ny, ld_, g.ny, ldm_[1], ld_, ld_, 0, plane, plane};
    launch_pdl(k_fp_gemm<T, true, false, T>, dim3((p.N + TM - 1) / TM, (p.M + TM - 1) / TM, axis == 0 ? 1 : g.nx), 64,
               0, s, p, FpScatter<T, T>{}, gate);
}

template <typename T>
template <typename S>
void FastPoisson<T>::run(cudaStream_t s, const S *r, T *z, const int *gate) {
    constexpr int TM = FpTile<T>::TM;
    const Grid &g = A_.g;
    int k = 0;
    const int body = nghost_ > 0 || nsolid_ > 0;
    launch_pdl(k_fp_gather<T, S>, dim3((ld_ + 31) / 32, (g.ny + 7) / 8, (g.nx + FP_GPLANES - 1) / FP_GPLANES),
               dim3(32, 8), 0, s, A_, r, F_[0], ld_, body, (const T *)gscale_, gate);
    T *x = F_[0], *y = F_[1];
    auto turn = [&](int axis, bool forward) {
        if (axis == 2) gemm_rows(s, x, axis, forward, y, gate);
        else gemm_cols(s, x, axis, forward, y, gate);
        std::swap(x, y);
        k++;
    };
    turn(2, true);
    if (tri_ != 1) turn(1, true);
    if (tri_ != 0) turn(0, true);
    FpPin<T> pin{};
    pin.singular = A_.p_singular;
    const long long plane = (long long)g.ny * ld_;
    if (tri_ >= 0) {
        const int o = tri_ == 0 ? 1 : 0, n = tri_ == 0 ? g.nx : g.ny;
        const long long st = tri_ == 0 ? plane : ld_, outer = tri_ == 0 ? ld_ : plane;
        pin.w = dtri_;
        pin.zero = zero_[o] * outer + zero_[2];
        pin.f1 = fwd_[o];
        pin.f2 = fwd_[2];
        pin.z1 = zero_[o];
        pin.z2 = zero_[2];
        launch_pdl(n <= 16 * FP_SEG ? k_fp_tri<T, 512> : k_fp_tri<T, 1024>,
                   dim3((ld_ + 31) / 32, o == 1 ? g.ny : g.nx), dim3(32, (n + FP_SEG - 1) / FP_SEG), 0, s, (const T *)inv_, A_.km[tri_] + 2, A_.kp[tri_] + 2, n, st, outer, ld_, pin, (const T *)x, y, gate);
    } else {
        pin.w = nullptr;
        pin.zero = zero_[0] * plane + (long long)zero_[1] * ld_ + zero_[2];
        pin.f1 = fwd_[1];
        pin.f2 = fwd_[2];
        pin.z1 = zero_[1];
        pin.z2 = zero_[2];
        launch_pdl(k_fp_diag<T>, dim3((ld_ + 31) / 32, (g.ny + 7) / 8, g.nx), dim3(32, 8), 0, s, (const T *)inv_,
                   g.ny, ld_, pin, (const T *)dtri_, (const T *)x, y, gate);
    }
    std::swap(x, y);
    if (tri_ != 0) turn(0, false);
    if (tri_ != 1) turn(1, false);
    FpScatter<T, S> sc{g, g.dny, r, bwd_[2], A_.pinned, A_.p_singular};
    FpGemm<T> p{x, bwd_[2], z, g.nx * g.ny, ld_, g.nz, ld_, ldm_[2], 0, 0, 0, 0};
    launch_pdl(k_fp_gemm<T, false, true, S>, dim3((p.N + TM - 1) / TM, (p.M + TM - 1) / TM), 64, 0, s, p, sc, gate);
    const int nout = A_.sw.nout;
    auto edges = [&](int solids) {
        launch_pdl(k_fp_edges<T, S>, (nout + solids + 255) / 256, 256, 0, s, A_, r, z, A_.sw.outer, nout,
                   (const int *)solid_, solids, gate);
        k++;
    };
    edges(nsolid_);
    k += 3;
    if (nghost_ > 0) {
        launch_pdl(k_fp_near<T, S>, FP_CLUSTER, FP_CT, 0, s, A_, r, z, (const int *)near_, nred_, nblack_, gcell_,
                   nghost_, (const T *)gidiv_, gtmp_, 2, gate);
        k++;
        if (near_outer_) edges(0);
    }
    note_launches(k);
    launches_ = k;
}

template <typename T>
bool FastPoisson<T>::apply_from64(cudaStream_t s, const double *r, T *z, const int *gate) {
    run(s, r, z, gate);
    return true;
}

template <typename T>
bool FastPoisson<T>::apply_from_df(cudaStream_t s, const dfloat *r, T *z, const int *gate) {
    if constexpr (sizeof(T) == 4) {
        run(s, r, z, gate);
        return true;
    }
    return false;
}

template class FastPoisson<float>;
template class FastPoisson<double>;

}  // namespace ibm
