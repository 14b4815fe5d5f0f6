// Fast-diagonalisation preconditioner of the pressure rows (fastpoisson.h).
#include <algorithm>
#include <array>
#include <cmath>
#include <utility>
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
// The source of one interior cell: coeffsum r, 0 on solid rows and the
// pinned row, scaled on ghost rows, the residuals of the outer rows beside
// it folded in.
template <typename T, typename S>
__device__ __forceinline__ T fp_source(const OpT<T> &c, const S *__restrict__ r, T v, const long long P, const int i,
                                       const int j, const int k, const uint8_t fl, const T *__restrict__ gscale) {
    const Grid &g = c.g;
    v *= c.ks[0][i + 2] + c.ks[1][j + 2] + c.ks[2][k + 2];
    if (fl == GHOST) v *= gscale[c.gid[P]];
    else if (fl != FLUID) v = 0;
    if (i == 0 || i == g.nx - 1 || j == 0 || j == g.ny - 1 || k == 0 || k == g.nz - 1) {
        if (fl == FLUID) {
            if (i == 0) v += c.km[0][2] * fp_outer(c.bc[F_W], fp_value<T, S>(r[P - g.sx]));
            if (i == g.nx - 1) v += c.kp[0][i + 2] * fp_outer(c.bc[F_E], fp_value<T, S>(r[P + g.sx]));
            if (j == 0) v += c.km[1][2] * fp_outer(c.bc[F_S], fp_value<T, S>(r[P - g.sy]));
            if (j == g.ny - 1) v += c.kp[1][j + 2] * fp_outer(c.bc[F_N], fp_value<T, S>(r[P + g.sy]));
            if (k == 0) v += c.km[2][2] * fp_outer(c.bc[F_D], fp_value<T, S>(r[P - 1]));
            if (k == g.nz - 1) v += c.kp[2][k + 2] * fp_outer(c.bc[F_U], fp_value<T, S>(r[P + 1]));
        }
        if (c.p_singular && P == c.pinned) v = 0;
    }
    return v;
}

// The padded residual as the compact source of the separable system.  On a
// mirror-symmetric z axis (z.fold) a thread takes the cells k and nz-1-k and
// writes their sum to column k and their difference to column off + k, the
// inputs of the even and the odd modes.  Columns that hold no value are 0.
// Bound by its bytes (8 read, 4 written per cell from double-float
// residuals); every plane's loads are issued before any is used (128^2
// planes of 192: 24 -> 20 us, cold).  Grid (off / 32, ny / 8, nx / 4).
constexpr int FP_GPLANES = 4;

template <typename T, typename S>
__global__ void __launch_bounds__(256)
k_fp_gather(const OpT<T> c, const S *__restrict__ r, T *__restrict__ f, const FpModes z, const int ld, const int body,
            const T *__restrict__ gscale, const int *gate) {
    FP_GATE(gate);
    const Grid &g = c.g;
    const int q = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
    if (q >= z.off || j >= g.ny) return;
    const int i0 = blockIdx.z * FP_GPLANES;
    const int k1 = min(q, g.nz - 1), k2 = z.fold ? max(g.nz - 1 - q, 0) : k1;
    S a[FP_GPLANES], b[FP_GPLANES];
    uint8_t fa[FP_GPLANES], fb[FP_GPLANES];
#pragma unroll
    for (int p = 0; p < FP_GPLANES; p++) {
        const long long P = cidx(g, min(i0 + p, g.nx - 1), j, 0);
        a[p] = r[P + k1];
        if (z.fold) b[p] = r[P + k2];
        fa[p] = fb[p] = FLUID;
        if (body) {
            fa[p] = c.flag[P + k1];
            if (z.fold) fb[p] = c.flag[P + k2];
        }
    }
#pragma unroll
    for (int p = 0; p < FP_GPLANES; p++) {
        const int i = i0 + p;
        if (i >= g.nx) break;
        const long long P = cidx(g, i, j, 0);
        T *row = f + ((long long)i * g.ny + j) * ld;
        T v = fp_source<T, S>(c, r, fp_value<T, S>(a[p]), P + k1, i, j, k1, fa[p], gscale);
        if (!z.fold) {
            row[q] = q < g.nz ? v : (T)0;
            continue;
        }
        T d = 0;
        if (q < z.no) {
            const T w = fp_source<T, S>(c, r, fp_value<T, S>(b[p]), P + k2, i, j, k2, fb[p], gscale);
            d = v - w;
            v += w;
        }
        row[q] = q < z.ne ? v : (T)0;
        if (z.off + q < ld) row[z.off + q] = d;
    }
}

// ------------------------------------------------------------ transforms --
// Dense transforms as tiled products C = A B, 64 threads with register
// tiles of R x R made of 2 x 2 sub-tiles (shared-memory reads are
// conflict-free vectors or broadcasts), k in steps of 16 through two
// shared-memory buffers with the next step's loads in flight.  Bound by the
// FP32 (FP64) multiply-add pipe.
//
// On a mirror-symmetric axis the modes are even or odd, so a transform
// splits into two of half the size, half the multiplications: forward, from
// the sums and differences of mirrored cells (k_fp_gemm: formed by the
// gather along z, while loading along x and y); backward, both parities'
// parts E and O of the first half's cells at once, x_i = E + O and
// x_(n-1-i) = E - O (k_fp_back).
//
// Sphere 192x128x128 FP32, cold: forward z 26 -> 16, forward y 25 -> 21,
// backward y 25 -> 18 (25 with four blocks to an SM, a wave and a quarter;
// six), backward z 27 -> 22 us (half the products; the loads of both halves
// and the register tiles' shared-memory reads bound them now); cavity 64^3 FP64, an application: 0.36 -> 0.23 ms.
//
// Tiles: TM = 64 (R = 8) or 32 in FP32, 32 (R = 4) or 16 in FP64 (run).
template <typename T, int TM>
struct FpTile {
    static constexpr int R = TM / 8, R2 = R / 2, V = 16 / (int)sizeof(T);
    static constexpr int VR = R2 < V ? R2 : V;   // elements per shared-memory read
};
constexpr int FP_TK = 16;

template <typename T, int N>
struct alignas(sizeof(T) * N) FpVec {
    T v[N];
};

// Operands per parity (blockIdx.z & 1 when nb = 2); batch strides over the
// remaining part of blockIdx.z.
template <typename T>
struct FpGemm {
    const T *a[2], *b[2];
    T *c[2];
    int M[2], N[2], K[2];
    int lda[2], ldb[2], ldc;
    long long sb, sc;
    int nb;
    int fold;   // > 0: row k of B is B(k) + sign B(fold - 1 - k), sign by parity
};

// TA = false: A(m, k) with k contiguous (the data, when the contiguous axis
// is transformed); TA = true: A given as its transpose, (k, m) with m
// contiguous (the axis matrix, applied to another axis).
template <typename T, int TM, bool TA>
__global__ void __launch_bounds__(64)
k_fp_gemm(const FpGemm<T> p, const int *gate) {
    FP_GATE(gate);
    using Tile = FpTile<T, TM>;
    constexpr int R = Tile::R, R2 = Tile::R2, V = Tile::V, VR = Tile::VR, H = TM / 2;
    constexpr int PITCH = TA ? TM : TM + V;
    constexpr int NQ = TM * FP_TK / V / 64;   // vector loads per thread and operand
    using Vec = FpVec<T, V>;
    using Rd = FpVec<T, VR>;
    __shared__ alignas(16) T As[2][FP_TK][PITCH];
    __shared__ alignas(16) T Bs[2][FP_TK][TM];
    const int par = p.nb == 2 ? blockIdx.z & 1 : 0, batch = p.nb == 2 ? blockIdx.z >> 1 : blockIdx.z;
    const T *A = par ? p.a[1] : p.a[0], *B = (par ? p.b[1] : p.b[0]) + batch * p.sb;
    const int M = par ? p.M[1] : p.M[0], N = par ? p.N[1] : p.N[0], K = par ? p.K[1] : p.K[0];
    const int lda = par ? p.lda[1] : p.lda[0], ldb = par ? p.ldb[1] : p.ldb[0];
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TM;
    if (m0 >= M || n0 >= N) return;
    const int t = threadIdx.x, tx = t & 7, ty = t >> 3;
    Vec ra[NQ], rb[NQ];
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int e = t + 64 * q;
            constexpr int PER = TM / V;
            const int k = k0 + e / PER, n = n0 + (e % PER) * V;
            rb[q] = Vec{};
            if (k < K && n < N) {
                rb[q] = *reinterpret_cast<const Vec *>(B + (long long)k * ldb + n);
                const int km = p.fold - 1 - k;
                if (TA && p.fold && km != k) {
                    const Vec m = *reinterpret_cast<const Vec *>(B + (long long)km * ldb + n);
#pragma unroll
                    for (int l = 0; l < V; l++) rb[q].v[l] = par ? rb[q].v[l] - m.v[l] : rb[q].v[l] + m.v[l];
                }
            }
            ra[q] = Vec{};
            if (TA) {
                const int m = m0 + (e % PER) * V;
                if (k < K && m < lda) ra[q] = *reinterpret_cast<const Vec *>(A + (long long)k * lda + m);
            } else {
                constexpr int PK = FP_TK / V;
                const int m = m0 + e / PK, ka = k0 + (e % PK) * V;
                if (m < M && ka < K) ra[q] = *reinterpret_cast<const Vec *>(A + (long long)m * lda + ka);
            }
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int e = t + 64 * q;
            constexpr int PER = TM / V, PK = FP_TK / V;
            *reinterpret_cast<Vec *>(&Bs[buf][e / PER][(e % PER) * V]) = rb[q];
            if (TA) {
                *reinterpret_cast<Vec *>(&As[buf][e / PER][(e % PER) * V]) = ra[q];
            } else {
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
    load(0);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += FP_TK) {
        const bool more = k0 + FP_TK < K;
        if (more) load(k0 + FP_TK);
#pragma unroll
        for (int k = 0; k < FP_TK; k++) {
            T av[R], bv[R];
#pragma unroll
            for (int h = 0; h < 2; h++) {
#pragma unroll
                for (int l = 0; l < R2; l += VR) {
                    *reinterpret_cast<Rd *>(&av[h * R2 + l]) = *reinterpret_cast<const Rd *>(&As[buf][k][h * H + ty * R2 + l]);
                    *reinterpret_cast<Rd *>(&bv[h * R2 + l]) = *reinterpret_cast<const Rd *>(&Bs[buf][k][h * H + tx * R2 + l]);
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
    T *C = (par ? p.c[1] : p.c[0]) + batch * p.sc;
#pragma unroll
    for (int x = 0; x < R; x++) {
        const int m = m0 + (x / R2) * H + ty * R2 + x % R2;
        if (m >= M) continue;
        T *row = C + (long long)m * p.ldc;
#pragma unroll
        for (int y = 0; y < R; y += VR) {
            const int n = n0 + (y / R2) * H + tx * R2 + y % R2;
            if (n < N) {
                Rd o;
#pragma unroll
                for (int l = 0; l < VR; l++) o.v[l] = acc[x][y + l];
                *reinterpret_cast<Rd *>(row + n) = o;
            }
        }
    }
}

// Where the last backward transform (along z) writes: the padded array,
// grid line (i, j) per row, shifted so that the pinned cell takes its
// residual's value.
template <typename T, typename S>
struct FpScatter {
    Grid g;
    const S *r;             // residual (pinned shift)
    const T *v0;            // z(0, 0, 0) of line (0, 0) in terms of its modes
    long long pinned;
    int singular, ld;
};

template <typename T, typename S>
__device__ __forceinline__ T fp_shift(const FpScatter<T, S> &sc, const T *__restrict__ line) {
    if (!sc.singular) return 0;
    // z(0,0,0) of the unshifted solution: one line's product, by every
    // block for itself.
    __shared__ T red[2];
    const int t = threadIdx.x;
    T s = 0;
    for (int q = t; q < sc.ld; q += 64) s += line[q] * sc.v0[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((t & 31) == 0) red[t >> 5] = s;
    __syncthreads();
    return fp_value<T, S>(sc.r[sc.pinned]) - (red[0] + red[1]);
}

// Backward transform of an axis, one product for both parities: E = Ae Be
// and O = Ao Bo over the first half's cells.  ROWS (the contiguous axis): A
// is the data, row m its modes (even, then odd from column off), B the axis
// matrices (mode, cell); the result goes to the padded array.  Otherwise A
// holds the axis matrices (mode, cell), B the data's mode rows (even, then
// odd from row ne), and C receives rows i and n - 1 - i.  An axis without
// the symmetry passes fold = 0: E alone over all its cells.
template <typename T>
struct FpBack {
    const T *a[2], *b[2];
    T *c;
    int M, N;               // rows and columns of E
    int K[2];
    int lda[2], ldb[2], ldc;
    long long sb, sc;       // batch strides (blockIdx.z)
    int fold, n;            // fold: both parities; n: cells of the axis
};

template <typename T, int TM, bool ROWS, bool FOLD, typename S>
__global__ void __launch_bounds__(64, sizeof(T) == 4 && TM == 64 ? 6 : 0)
k_fp_back(const FpBack<T> p, const FpScatter<T, S> sc, const int *gate) {
    FP_GATE(gate);
    using Tile = FpTile<T, TM>;
    constexpr int R = Tile::R, V = Tile::V, VR = Tile::VR;
    constexpr int NP = FOLD ? 2 : 1;
    // The side that is halved by the two parities sharing the tile.
    constexpr int MA = FOLD && !ROWS ? TM / 2 : TM, NB = FOLD && ROWS ? TM / 2 : TM;
    constexpr int RA = MA / 8, RB = NB / 8;              // register tile per parity
    constexpr int GA = RA == R ? 2 : 1, GB = RB == R ? 2 : 1;   // sub-tile groups
    constexpr int PITCH = ROWS ? MA + V : MA;
    constexpr int QA = MA * FP_TK / V / 64, QB = NB * FP_TK / V / 64;
    static_assert(QA >= 1 && QB >= 1, "tile too small for 64 threads");
    using Vec = FpVec<T, V>;
    using Rd = FpVec<T, VR>;
    __shared__ alignas(16) T As[2][NP][FP_TK][PITCH];
    __shared__ alignas(16) T Bs[2][NP][FP_TK][NB];
    const int m0 = blockIdx.y * MA, n0 = blockIdx.x * NB;
    const int t = threadIdx.x, tx = t & 7, ty = t >> 3;
    Vec ra[NP][QA], rb[NP][QB];
    auto load = [&](int k0) {
#pragma unroll
        for (int h = 0; h < NP; h++) {
            const T *A = p.a[h], *B = p.b[h] + blockIdx.z * p.sb;
#pragma unroll
            for (int q = 0; q < QB; q++) {
                const int e = t + 64 * q, k = k0 + e / (NB / V), n = n0 + (e % (NB / V)) * V;
                rb[h][q] = Vec{};
                if (k < p.K[h] && n < p.ldb[h]) rb[h][q] = *reinterpret_cast<const Vec *>(B + (long long)k * p.ldb[h] + n);
            }
#pragma unroll
            for (int q = 0; q < QA; q++) {
                const int e = t + 64 * q;
                ra[h][q] = Vec{};
                if (ROWS) {
                    const int m = m0 + e / (FP_TK / V), k = k0 + (e % (FP_TK / V)) * V;
                    if (m < p.M && k < p.K[h]) ra[h][q] = *reinterpret_cast<const Vec *>(A + (long long)m * p.lda[h] + k);
                } else {
                    const int k = k0 + e / (MA / V), m = m0 + (e % (MA / V)) * V;
                    if (k < p.K[h] && m < p.lda[h]) ra[h][q] = *reinterpret_cast<const Vec *>(A + (long long)k * p.lda[h] + m);
                }
            }
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int h = 0; h < NP; h++) {
#pragma unroll
            for (int q = 0; q < QB; q++) {
                const int e = t + 64 * q;
                *reinterpret_cast<Vec *>(&Bs[buf][h][e / (NB / V)][(e % (NB / V)) * V]) = rb[h][q];
            }
#pragma unroll
            for (int q = 0; q < QA; q++) {
                const int e = t + 64 * q;
                if (ROWS) {
#pragma unroll
                    for (int l = 0; l < V; l++)
                        As[buf][h][(e % (FP_TK / V)) * V + l][e / (FP_TK / V)] = ra[h][q].v[l];
                } else {
                    *reinterpret_cast<Vec *>(&As[buf][h][e / (MA / V)][(e % (MA / V)) * V]) = ra[h][q];
                }
            }
        }
    };
    T acc[NP][RA][RB];
#pragma unroll
    for (int h = 0; h < NP; h++)
#pragma unroll
        for (int x = 0; x < RA; x++)
#pragma unroll
            for (int y = 0; y < RB; y++) acc[h][x][y] = 0;
    T shift = 0;
    if constexpr (ROWS) shift = fp_shift(sc, p.a[0]);
    load(0);
    store(0);
    __syncthreads();
    int buf = 0;
    const int K = p.K[0];   // the even part is never the shorter one
    for (int k0 = 0; k0 < K; k0 += FP_TK) {
        const bool more = k0 + FP_TK < K;
        if (more) load(k0 + FP_TK);
#pragma unroll
        for (int k = 0; k < FP_TK; k++) {
#pragma unroll
            for (int h = 0; h < NP; h++) {
                T av[RA], bv[RB];
#pragma unroll
                for (int gq = 0; gq < GA; gq++)
#pragma unroll
                    for (int l = 0; l < RA / GA; l += VR)
                        *reinterpret_cast<Rd *>(&av[gq * (RA / GA) + l]) =
                            *reinterpret_cast<const Rd *>(&As[buf][h][k][gq * (MA / 2) + ty * (RA / GA) + l]);
#pragma unroll
                for (int gq = 0; gq < GB; gq++)
#pragma unroll
                    for (int l = 0; l < RB / GB; l += VR)
                        *reinterpret_cast<Rd *>(&bv[gq * (RB / GB) + l]) =
                            *reinterpret_cast<const Rd *>(&Bs[buf][h][k][gq * (NB / 2) + tx * (RB / GB) + l]);
#pragma unroll
                for (int x = 0; x < RA; x++)
#pragma unroll
                    for (int y = 0; y < RB; y++) acc[h][x][y] += av[x] * bv[y];
            }
        }
        if (more) {
            store(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
#pragma unroll
    for (int x = 0; x < RA; x++) {
        const int m = m0 + (x / (RA / GA)) * (MA / 2) + ty * (RA / GA) + x % (RA / GA);
        if (m >= p.M) continue;
        if constexpr (ROWS) {
            const int i = (int)fdiv(sc.g.dny, (uint32_t)m), j = m - i * sc.g.ny;
            T *row = p.c + cidx(sc.g, i, j, 0);
#pragma unroll
            for (int y = 0; y < RB; y++) {
                const int n = n0 + (y / (RB / GB)) * (NB / 2) + tx * (RB / GB) + y % (RB / GB);
                if (n >= p.N) continue;
                const T e = acc[0][x][y] + shift, o = FOLD ? acc[NP - 1][x][y] : (T)0;
                row[n] = e + o;
                if (FOLD && p.n - 1 - n != n) row[p.n - 1 - n] = e - o;
            }
        } else {
            T *C = p.c + blockIdx.z * p.sc;
            T *row = C + (long long)m * p.ldc, *mir = C + (long long)(p.n - 1 - m) * p.ldc;
#pragma unroll
            for (int y = 0; y < RB; y += VR) {
                const int n = n0 + (y / (RB / GB)) * (NB / 2) + tx * (RB / GB) + y % (RB / GB);
                if (n >= p.N) continue;
                Rd e, o;
#pragma unroll
                for (int l = 0; l < VR; l++) {
                    const T E = acc[0][x][y + l], O = FOLD ? acc[NP - 1][x][y + l] : (T)0;
                    e.v[l] = E + O;
                    o.v[l] = E - O;
                }
                *reinterpret_cast<Rd *>(row + n) = e;
                if (FOLD && p.n - 1 - m != m) *reinterpret_cast<Rd *>(mir + n) = o;
            }
        }
    }
}

}  // namespace ibm

#include "fastplane.cuh"

namespace ibm {

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
    __shared__ T sa[32][33], sh[32][33];
    const int c = blockIdx.x * 32 + threadIdx.x, seg = threadIdx.y, ns = blockDim.y;
    const long long base = blockIdx.y * outer + min(c, ld - 1);
    const int i0 = seg * FP_SEG;
    T h[FP_SEG], v[FP_SEG];
#pragma unroll
    for (int q = 0; q < FP_SEG; q++) v[q] = i0 + q < n ? iv[base + (i0 + q) * st] : (T)0;
    FP_GATE(gate);
#pragma unroll
    for (int q = 0; q < FP_SEG; q++) h[q] = i0 + q < n ? fin[base + (i0 + q) * st] : (T)0;
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
                            T *iv, const int n, const long long st, const long long outer, const int ld, const int z1,
                            const int z2) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, o = blockIdx.y;
    if (c >= ld) return;
    const long long base = o * outer + c;
    const double lam = l1[o] + l2[c];
    if (!(lam == lam)) {   // no mode in this column (NaN)
        for (int i = 0; i < n; i++) iv[base + i * st] = 0;
        return;
    }
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
                          T *iv, const int ny, const int ld, const int z0, const int z1, const int z2) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
    if (c >= ld) return;
    const double lam = l0[i] + l1[j] + l2[c];
    const bool zero = i == z0 && j == z1 && c == z2;
    iv[((long long)i * ny + j) * ld + c] = !(lam == lam) || zero ? (T)0 : (T)(1.0 / lam);
}

// ------------------------------------------------------- outer rows, body --
// Outer rows solved for the outer values, each through its chain of
// partners down to an interior cell (as the multigrid's outer pass), the
// identity rows of solid cells, and the swept values of the cells near the
// body (cell[q] takes val[q]).  The three lists write different cells, and no
// outer row reads a cell that another thread of the launch writes: a partner
// that is solid (partners: there are some) gives its residual, the value its
// identity row takes, and a
// body whose swept cells are partners of outer rows gets its outer rows in
// a launch of their own.
template <typename T, typename S>
__global__ void __launch_bounds__(256)
k_fp_edges(const OpT<T> c, const S *__restrict__ r, T *z, const int *__restrict__ outer, const int nout,
           const int *__restrict__ solid, const int nsolid, const int partners, const int *__restrict__ cell,
           const T *__restrict__ val, const int ncell, const int *gate) {
    const int t = blockIdx.x * 256 + threadIdx.x, ts = t - nout, tc = ts - nsolid;
    const int own = t < nout ? outer[t] : ts < nsolid ? solid[ts] : tc < ncell ? cell[tc] : -1;
    FP_GATE(gate);
    if (own < 0) return;
    if (t >= nout) {
        z[own] = ts < nsolid ? fp_value<T, S>(r[own]) : val[tc];
        return;
    }
    long long chain[3];
    int face[3], layer[3], n = 0;
    long long Q = own;
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
    T v = partners && c.flag[Q] == SOLID ? fp_value<T, S>(r[Q]) : z[Q];
    for (int q = n - 1; q >= 0; q--) {
        const BCRow<T> &F = c.bc[face[q]];
        const T rv = fp_value<T, S>(r[chain[q]]);
        if (F.type == BCT_PRESSURE || F.type == BCT_VELPERIODIC)
            v = (rv - F.dir_m[layer[q] - 1] * v) / F.dir_o[layer[q] - 1];
        else
            v = rv + v;
    }
    z[own] = v;
}

// Sweeps over the cells near the body: an overlapping Schwarz step.  The
// cells (fluid ones within FP_LAYERS of a ghost, and the ghosts) are cut
// into patches by the cubes of the grid; a block takes one patch with the
// cells FP_OVERLAP beyond it, keeps their rows in registers (at most FP_PU
// cells per thread) and their values in shared memory (couplings to cells
// outside go into the right-hand side), runs its sweeps there (red, black,
// then the ghost rows Jacobi-style) and returns the values of its own cells,
// which k_fp_edges writes to z.  (Sweeps over all the cells at once with a
// barrier per pass, across the blocks of a cluster or as launches, spend 3-4
// us per pass on the L2 round trip; rows read again from L1 in every pass
// made an application of boxes 95x61x47 62 us, in registers 56.)  Bound by
// latency: FP_SWEEPS x 4 block barriers; the tables' chain of loads runs
// before the wait for the predecessor.
constexpr int FP_PT = 512;               // threads of a patch block
constexpr int FP_PU = 3;                 // cells per thread
constexpr int FP_PMAX = FP_PT * FP_PU;   // cells of a patch, overlap included

template <typename T, typename S>
__global__ void __launch_bounds__(FP_PT)
k_fp_patch(const FpPatches<T> p, const S *__restrict__ r, const T *__restrict__ z, T *__restrict__ out,
           const int sweeps, const int *gate) {
    __shared__ T v[FP_PMAX];
    const int b = blockIdx.x, s0 = p.start[b], nr = p.count[3 * b], nf = nr + p.count[3 * b + 1];
    const int n = nf + p.count[3 * b + 2];
    T w[FP_PU][8], f[FP_PU], self[FP_PU];
    int m[FP_PU][8], own[FP_PU], P[FP_PU];
    // The tables, before the wait for the values.
#pragma unroll
    for (int u = 0; u < FP_PU; u++) {
        const int q = u * FP_PT + threadIdx.x;
        own[u] = -1;
        P[u] = -1;
        if (q >= n) continue;
        own[u] = p.loc[s0 + q];
        const int c = own[u] < 0 ? ~own[u] : own[u];
        P[u] = p.P[c];
        self[u] = p.self[s0 + q];
        f[u] = p.rw[s0 + q];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            w[u][e] = p.w[(size_t)e * p.nloc + s0 + q];
            m[u][e] = p.ref[(size_t)e * p.nloc + s0 + q];
            if (m[u][e] < 0) m[u][e] = ~p.to[e * p.ncell + c];   // outside: ~its index; 0: no coupling
            else m[u][e]++;                                       // inside: its place + 1
        }
    }
    FP_GATE(gate);
#pragma unroll
    for (int u = 0; u < FP_PU; u++) {
        const int q = u * FP_PT + threadIdx.x;
        if (P[u] < 0) continue;
        v[q] = z[P[u]];
        f[u] *= fp_value<T, S>(r[P[u]]);
#pragma unroll
        for (int e = 0; e < 8; e++) {
            if (m[u][e] > 0) {
                m[u][e]--;
                continue;
            }
            if (m[u][e] < 0) f[u] += w[u][e] * z[~m[u][e]];
            w[u][e] = 0;
            m[u][e] = q;
        }
    }
    __syncthreads();
    // The rows of this thread's cells [lo, hi): a pass over one colour.
    auto pass = [&](int lo, int hi) {
#pragma unroll
        for (int u = 0; u < FP_PU; u++) {
            const int q = u * FP_PT + threadIdx.x;
            if (q < lo || q >= hi) continue;
            T t = f[u];
#pragma unroll
            for (int e = 0; e < 6; e++) t += w[u][e] * v[m[u][e]];
            v[q] = t;
        }
        __syncthreads();
    };
    for (int s = 0; s < sweeps; s++) {
        pass(0, nr);
        pass(nr, nf);
        T g[FP_PU];
#pragma unroll
        for (int u = 0; u < FP_PU; u++) {
            const int q = u * FP_PT + threadIdx.x;
            if (q < nf || q >= n) continue;
            g[u] = f[u] + self[u] * v[q];
#pragma unroll
            for (int e = 0; e < 8; e++) g[u] += w[u][e] * v[m[u][e]];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < FP_PU; u++) {
            const int q = u * FP_PT + threadIdx.x;
            if (q >= nf && q < n) v[q] = g[u];
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < FP_PU; u++)
        if (own[u] >= 0) out[own[u]] = v[u * FP_PT + threadIdx.x];
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

// The cells near the body, their rows and the patches (k_fp_patch), cut by
// cubes of side `cube`; false when the cells are more than `most` or a patch
// cannot be made small enough.
template <typename T>
static bool build_patches(const OpT<double> &A, const FastPoissonGeom &h, const std::vector<double> &gw, int cube,
                          size_t most, FpPatchTables<T> &t_) {
    const Grid &g = A.g;
    const int n[3] = {g.nx, g.ny, g.nz};
    const long long st[3] = {g.sx, g.sy, 1};
    std::vector<int> id(g.ncell, -1);   // near cell number of a padded index
    std::vector<int> cells, ijk;
    const int ng = (int)h.gcell.size();
    cells.reserve(32 * (size_t)ng);
    ijk.reserve(96 * (size_t)ng);
    auto push = [&](long long Q, int i, int j, int k) {
        id[Q] = (int)cells.size();
        cells.push_back((int)Q);
        ijk.push_back(i);
        ijk.push_back(j);
        ijk.push_back(k);
    };
    auto add = [&](long long Q, int i, int j, int k) {
        if (i < 0 || i >= n[0] || j < 0 || j >= n[1] || k < 0 || k >= n[2] || id[Q] >= 0 || h.flag[Q] != FLUID) return;
        if (!(A.p_singular && Q == A.pinned)) push(Q, i, j, k);
    };
    auto split = [&](int Q, int &i, int &j, int &k) {
        const uint32_t I = (uint32_t)Q / (uint32_t)g.sx, r = (uint32_t)Q - I * (uint32_t)g.sx, J = r / (uint32_t)g.sy;
        i = (int)I - 2;
        j = (int)J - 2;
        k = (int)(r - J * (uint32_t)g.sy) - 2;
    };
    int i, j, k;
    for (int Q : h.gcell) {
        split(Q, i, j, k);
        push(Q, i, j, k);
    }
    size_t first = 0;   // the last layer's cells
    for (int layer = 0; layer < FP_LAYERS; layer++) {
        const size_t last = cells.size();
        if (layer == 0)
            for (int Q : h.gidx)
                if (Q >= 0 && id[Q] < 0) {
                    split(Q, i, j, k);
                    add(Q, i, j, k);
                }
        for (size_t q = first; q < last; q++) {
            const long long Q = cells[q];
            i = ijk[3 * q];
            j = ijk[3 * q + 1];
            k = ijk[3 * q + 2];
            add(Q - st[0], i - 1, j, k);
            add(Q + st[0], i + 1, j, k);
            add(Q - st[1], i, j - 1, k);
            add(Q + st[1], i, j + 1, k);
            add(Q - st[2], i, j, k - 1);
            add(Q + st[2], i, j, k + 1);
        }
        first = last;
    }
    if (cells.size() > most) return false;
    const int nc = (int)cells.size();
    // Rows: couplings (padded index, weight), weight of the old value and of
    // the residual.  Ghost rows are relaxed as the multigrid relaxes them.
    t_.to.assign((size_t)nc * 8, -1);
    std::vector<T> w((size_t)nc * 8, (T)0), self(nc, (T)0), rw(nc, (T)1);   // w: [cell][8]
    std::vector<int> &to = t_.to;   // [8][nc]
    for (int q = 0; q < nc; q++) {
        const int *x = &ijk[3 * (size_t)q];
        for (int a = 0; a < 3; a++) t_.near_outer = t_.near_outer || x[a] < 2 || x[a] >= n[a] - 2;
        if (q < ng) {
            double off = 0;
            for (int e = 0; e < 8; e++) {
                const int P = h.gidx[8 * (size_t)q + e];
                if (P >= 0 && h.flag[P] == GHOST) off += std::fabs(gw[8 * (size_t)q + e]);
            }
            const double dg = 1.0 - h.gwself[q], dv = 1.0 / std::max({dg, 2.0 * off, 1e-3});
            for (int e = 0; e < 8; e++) {
                to[(size_t)e * nc + q] = h.gidx[8 * (size_t)q + e];
                w[8 * (size_t)q + e] = (T)(dv * gw[8 * (size_t)q + e]);
            }
            self[q] = (T)(1.0 - dg * dv);
            rw[q] = (T)dv;
        } else {
            double sum = 0;
            for (int a = 0; a < 3; a++) sum += h.km[a][x[a]] + h.kp[a][x[a]];
            for (int a = 0; a < 3; a++) {
                to[(size_t)(2 * a) * nc + q] = (int)(cells[q] - st[a]);
                to[(size_t)(2 * a + 1) * nc + q] = (int)(cells[q] + st[a]);
                w[8 * (size_t)q + 2 * a] = (T)(h.km[a][x[a]] / sum);
                w[8 * (size_t)q + 2 * a + 1] = (T)(h.kp[a][x[a]] / sum);
            }
        }
    }
    // The cells each row couples to, by number (-1: not near the body).
    std::vector<int> nbr((size_t)nc * 8);
    for (int q = 0; q < nc; q++)
        for (int e = 0; e < 8; e++) {
            const int Q = to[(size_t)e * nc + q];
            nbr[8 * (size_t)q + e] = Q >= 0 ? id[Q] : -1;
        }
    // Patches: the occupied cubes of the grid, halved until each fits with
    // the cells within FP_OVERLAP of it (along every axis).
    struct Box {
        int lo[3], hi[3];
    };
    std::vector<Box> todo;
    {
        const int cy = (n[1] + cube - 1) / cube, cz = (n[2] + cube - 1) / cube;
        std::vector<uint8_t> seen((size_t)((n[0] + cube - 1) / cube) * cy * cz, 0);
        for (int q = 0; q < nc; q++) {
            const int *x = &ijk[3 * (size_t)q], b[3] = {x[0] / cube, x[1] / cube, x[2] / cube};
            uint8_t &s = seen[((size_t)b[0] * cy + b[1]) * cz + b[2]];
            if (s) continue;
            s = 1;
            Box box;
            for (int a = 0; a < 3; a++) {
                box.lo[a] = b[a] * cube;
                box.hi[a] = std::min(box.lo[a] + cube, n[a]);
            }
            todo.push_back(box);
        }
    }
    std::vector<int> mark(nc, -1), list[3], pos(nc);
    std::vector<int16_t> refs;   // [local][8] of every patch
    std::vector<T> lw;
    for (size_t t = 0; t < todo.size(); t++) {
        const Box box = todo[t];
        const int stamp = (int)t;
        int lo[3], hi[3], own = 0;
        for (int a = 0; a < 3; a++) {
            lo[a] = std::max(0, box.lo[a] - FP_OVERLAP<T>);
            hi[a] = std::min(n[a], box.hi[a] + FP_OVERLAP<T>);
        }
        // Local order: red, black, ghost; by padded index within each.
        for (auto &l : list) l.clear();
        for (i = lo[0]; i < hi[0]; i++)
            for (j = lo[1]; j < hi[1]; j++) {
                const bool in = i >= box.lo[0] && i < box.hi[0] && j >= box.lo[1] && j < box.hi[1];
                const long long P0 = cidx(g, i, j, 0);
                for (k = lo[2]; k < hi[2]; k++) {
                    const int q = id[P0 + k];
                    if (q < 0) continue;
                    const bool mine = in && k >= box.lo[2] && k < box.hi[2];
                    own += mine;
                    list[q < ng ? 2 : (i + j + k) & 1].push_back(mine ? q : ~q);
                    mark[q] = stamp;
                }
            }
        if (own == 0) continue;   // half of a split cube
        const int total = (int)(list[0].size() + list[1].size() + list[2].size());
        if (total > FP_PMAX) {
            int a = 0;
            for (int b = 1; b < 3; b++)
                if (box.hi[b] - box.lo[b] > box.hi[a] - box.lo[a]) a = b;
            if (box.hi[a] - box.lo[a] < 2) return false;
            Box b0 = box, b1 = box;
            b0.hi[a] = b1.lo[a] = (box.lo[a] + box.hi[a]) / 2;
            todo.push_back(b0);
            todo.push_back(b1);
            continue;
        }
        t_.start.push_back((int)t_.loc.size());
        int at = 0;
        for (const auto &l : list) {
            t_.count.push_back((int)l.size());
            for (int u : l) {
                t_.loc.push_back(u);
                pos[u < 0 ? ~u : u] = at++;
            }
        }
        for (const auto &l : list)
            for (int u : l) {
                const int q = u < 0 ? ~u : u;
                t_.self.push_back(self[q]);
                t_.rw.push_back(rw[q]);
                for (int e = 0; e < 8; e++) {
                    const int m = nbr[8 * (size_t)q + e];
                    refs.push_back(m >= 0 && mark[m] == stamp ? (int16_t)pos[m] : (int16_t)-1);
                    lw.push_back(w[8 * (size_t)q + e]);
                }
            }
    }
    const size_t nloc = t_.loc.size();
    t_.ref.resize(8 * nloc);
    t_.w.resize(8 * nloc);
    for (size_t l = 0; l < nloc; l++)
        for (int e = 0; e < 8; e++) {
            t_.ref[e * nloc + l] = refs[8 * l + e];
            t_.w[e * nloc + l] = lw[8 * l + e];
        }
    t_.P = cells;
    return true;
}

template <typename T>
int FastPoisson<T>::setup(cudaStream_t s, const OpT<double> &A64, const OpT<T> &A, const FastPoissonGeom &h,
                          double max_ops) {
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
    nghost_ = (int)h.gcell.size();
    // The 1-D problems (diagonal dg, off-diagonals e, wrap couples the ends of
    // a periodic axis), mirror-symmetric up to the rounding of the face
    // coordinates, and the transforms' operations.
    std::vector<double> dg[3], e[3];
    double wrap[3], ops = 0;
    for (int a = 0; a < 3; a++) {
        const int N = n[a];
        const std::vector<double> &km = h.km[a], &kp = h.kp[a], &d = h.d[a];
        dg[a].resize(N);
        for (int i = 0; i < N; i++) dg[a][i] = km[i] + kp[i];
        if (!per[a]) {
            const BCRow<double> &L = A64.bc[lo[a]], &U = A64.bc[hi[a]];
            dg[a][0] += dirichlet_face(L.type) ? km[0] * (L.dir_m[0] / L.dir_o[0]) : -km[0];
            dg[a][N - 1] += dirichlet_face(U.type) ? kp[N - 1] * (U.dir_m[0] / U.dir_o[0]) : -kp[N - 1];
        }
        if (a == tri_) continue;
        e[a].assign(N, 0.0);
        for (int i = 0; i + 1 < N; i++) e[a][i] = -std::sqrt(kp[i] * km[i + 1]);
        wrap[a] = per[a] ? -std::sqrt(km[0] * kp[N - 1]) : 0.0;
        auto near_ = [](double x, double y) { return std::fabs(x - y) <= 1e-11 * (std::fabs(x) + std::fabs(y)); };
        bool sym = true;
        for (int i = 0; i < N; i++) sym = sym && near_(d[i], d[N - 1 - i]) && near_(dg[a][i], dg[a][N - 1 - i]);
        for (int i = 0; i + 1 < N; i++) sym = sym && near_(e[a][i], e[a][N - 2 - i]);
        FpModes &m = modes_[a];
        m.fold = sym;
        m.no = sym ? N / 2 : 0;
        m.ne = N - m.no;
        // Columns of the odd modes start on a vector boundary along z.
        m.off = a == 2 ? (m.ne + 3) & ~3 : m.ne;
        m.ld = a == 2 ? m.off + ((m.no + 3) & ~3) : N;
        ops += 4.0 * n[0] * n[1] * n[2] * m.ne;
    }
    if (ops > max_ops) return 1;
    std::vector<int> solid;
    size_t fluid = 0;
    for (int i = 0; i < n[0]; i++)
        for (int j = 0; j < n[1]; j++) {
            const long long P0 = cidx(g, i, j, 0);
            for (int k = 0; k < n[2]; k++) {
                if (h.flag[P0 + k] == SOLID) {
                    solid.push_back((int)(P0 + k));
                    if (i < 2 || i >= n[0] - 2 || j < 2 || j >= n[1] - 2 || k < 2 || k >= n[2] - 2) solid_partners_ = 1;
                }
                fluid += h.flag[P0 + k] == FLUID;
            }
        }
    nsolid_ = (int)solid.size();
    FpPatchTables<T> t;
    if (nghost_ > 0) {
        std::vector<double> gw(8 * (size_t)nghost_);
        cudaMemcpyAsync(gw.data(), A64.gw, sizeof(double) * gw.size(), cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
        const bool large = (long long)n[0] * n[1] * n[2] > FP_NEAR_GRID<T>;
        const size_t most = large ? (size_t)(FP_NEAR * (double)fluid) : (size_t)g.ncell;
        if (!build_patches(A64, h, gw, FP_CUBE<T>, most, t)) return 1;
    }
    bool ok = true;
    // Device arrays from chunks (an allocation each would be most of the
    // set-up of a small case).  A copy from pageable memory has read its
    // source when the call returns.
    char *chunk = nullptr;
    size_t left = 0;
    auto put = [&](const void *src, size_t bytes) -> void * {
        const size_t need = (bytes + 255) & ~(size_t)255;
        if (ok && need > left) {
            const size_t size = std::max(need, (size_t)1 << 20);
            ok = cudaMalloc((void **)&chunk, size) == cudaSuccess;
            if (ok) allocs_.push_back(chunk);
            left = size;
        }
        if (!ok) return nullptr;
        void *p = chunk;
        chunk += need;
        left -= need;
        if (src && bytes) ok = cudaMemcpyAsync(p, src, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess;
        return p;
    };
    std::vector<double> lam[3];
    std::vector<T> row0[3], v0;
    for (int a = 0; a < 3 && ok; a++) {
        if (a == tri_) continue;
        const int N = n[a];
        const std::vector<double> &d = h.d[a];
        FpModes &m = modes_[a];
        const bool sym = m.fold != 0;
        lam[a].assign(m.ld, __builtin_nan(""));
        row0[a].assign(m.ld, (T)0);
        if (a == 2) v0.assign(m.ld, (T)0);
        double best = INFINITY;
        for (int odd = 0; odd < (sym ? 2 : 1); odd++) {
            const int H = odd ? m.no : m.ne;   // size of this parity's problem
            std::vector<double> w(H), eh(H, 0.0), q;
            bool good;
            if (!sym && per[a]) {
                std::vector<double> f((size_t)N * N, 0.0);
                for (int i = 0; i < N; i++) {
                    f[(size_t)i * N + i] = dg[a][i];
                    if (i + 1 < N) f[(size_t)i * N + i + 1] = f[(size_t)(i + 1) * N + i] = e[a][i];
                }
                f[N - 1] = f[(size_t)(N - 1) * N] = wrap[a];
                good = dense_eigen(N, f, w, q);
            } else {
                // On vectors even (odd) about the middle: the first half's
                // rows, the couplings to the mirrored half folded in.
                for (int i = 0; i < H; i++) {
                    w[i] = sym ? (dg[a][i] + dg[a][N - 1 - i]) / 2 : dg[a][i];
                    if (i + 1 < H) eh[i] = sym ? (e[a][i] + e[a][N - 2 - i]) / 2 : e[a][i];
                }
                if (sym) {
                    const double sg = odd ? -1.0 : 1.0;
                    w[0] += sg * wrap[a];
                    if (N % 2 == 0) w[H - 1] += sg * e[a][N / 2 - 1];
                    else if (!odd) eh[H - 2] *= std::sqrt(2.0);
                }
                q.assign((size_t)H * H, 0.0);
                for (int i = 0; i < H; i++) q[(size_t)i * H + i] = 1;
                good = tridiag_eigen(H, w, eh, q);
            }
            if (!good) return 1;
            const int ld = (H + 3) & ~3, base = odd ? m.off : 0;
            m.ldm[odd] = ld;
            std::vector<T> f((size_t)H * ld, (T)0), b((size_t)H * ld, (T)0);
            for (int k = 0; k < H; k++) {
                lam[a][base + k] = w[k];
                if (std::fabs(w[k]) < best) {
                    best = std::fabs(w[k]);
                    zero_[a] = base + k;
                }
                for (int i = 0; i < H; i++) {
                    const bool pair = sym && i < N / 2;
                    const double sd = std::sqrt(sym ? (d[i] + d[N - 1 - i]) / 2 : d[i]);
                    const double v = q[(size_t)k * H + i] * (pair ? std::sqrt(0.5) : 1.0);
                    f[(size_t)i * ld + k] = (T)(v * sd);
                    b[(size_t)k * ld + i] = (T)(v / sd);
                }
                row0[a][base + k] = f[k];
                if (a == 2) v0[base + k] = b[(size_t)k * ld];
            }
            fwd_[a][odd] = (T *)put(f.data(), sizeof(T) * f.size());
            bwd_[a][odd] = (T *)put(b.data(), sizeof(T) * b.size());
        }
        if (A.p_singular) lam[a][zero_[a]] = 0.0;   // the constants
        row0_[a] = (T *)put(row0[a].data(), sizeof(T) * row0[a].size());
    }
    ld_ = modes_[2].ld;
    v0_ = (T *)put(v0.data(), sizeof(T) * v0.size());
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
        dk[0] = tmp(dg[tri_]);
        dk[1] = tmp(h.km[tri_]);
        dk[2] = tmp(h.kp[tri_]);
        std::vector<T> w(N);
        for (int i = 0; i < N; i++) w[i] = (T)h.d[tri_][i];
        dtri_ = (T *)put(w.data(), sizeof(T) * N);
        if (!ok) return -1;
        const long long st = tri_ == 0 ? (long long)n[1] * ld_ : ld_, outer = tri_ == 0 ? ld_ : (long long)n[1] * ld_;
        const bool sing = A.p_singular != 0;
        k_fp_pivots<T><<<dim3((ld_ + 127) / 128, n[o]), 128, 0, s>>>(dk[0], dk[1], dk[2], dl[o], dl[2], inv_, N, st, outer,
                                                                      ld_, sing ? zero_[o] : -1, sing ? zero_[2] : -1);
    } else {
        // f0: the x transform's constant-mode value of cell 0, then row 0.
        std::vector<T> w(1 + row0[0].size());
        w[0] = row0[0][zero_[0]];
        std::copy(row0[0].begin(), row0[0].end(), w.begin() + 1);
        dtri_ = (T *)put(w.data(), sizeof(T) * w.size());
        if (!ok) return -1;
        const bool sing = A.p_singular != 0;
        k_fp_sums<T><<<dim3((ld_ + 127) / 128, n[1], n[0]), 128, 0, s>>>(dl[0], dl[1], dl[2], inv_, n[1], ld_,
                                                                         sing ? zero_[0] : -1, zero_[1], zero_[2]);
    }
    solid_ = (int *)put(solid.data(), sizeof(int) * solid.size());
    if (nghost_ > 0) {
        std::vector<T> sc(nghost_);
        for (int q = 0; q < nghost_; q++) sc[q] = (T)(1.0 / std::max(1.0 - h.gwself[q], 1e-3));
        gscale_ = (T *)put(sc.data(), sizeof(T) * nghost_);
        auto ints = [&](const std::vector<int> &v) { return (const int *)put(v.data(), sizeof(int) * v.size()); };
        auto reals = [&](const std::vector<T> &v) { return (const T *)put(v.data(), sizeof(T) * v.size()); };
        npatch_ = (int)t.start.size();
        near_outer_ = t.near_outer;
        patch_ = FpPatches<T>{ints(t.P), ints(t.to), (int)t.P.size(), ints(t.start), ints(t.count), ints(t.loc),
                              (const int16_t *)put(t.ref.data(), sizeof(int16_t) * t.ref.size()), reals(t.w),
                              reals(t.self), reals(t.rw), (int)t.loc.size()};
        near_val_ = (T *)put(nullptr, sizeof(T) * t.P.size());
    }
    if (!ok) return -1;
    if constexpr (sizeof(T) == 4) {
        // Slices of one tile.  Larger ones keep the general kernels, whose
        // blocks share the work of a slice: with a tile of 64 rows by 128
        // columns the sphere of 192x128x128 took 65 + 40 us (front, rear)
        // against 57 + 46 and the same time per step.
        plane_ = modes_[tri_ == 1 ? 0 : 1].ne <= FPP_ROWS && ld_ <= FPP_COLS;
    }
    return cudaStreamSynchronize(s) == cudaSuccess ? 0 : -1;
}

// ------------------------------------------------------------ application --
// What the slice kernels share: sizes and strides, matrices m (forward or
// backward).  Their shared memory follows in front and rear.
template <typename T>
static FpPlane fpp_plane(const Grid &g, int tri, const FpModes (&modes)[3], int ld, T *const (&m)[3][2]) {
    FpPlane p{};
    p.o = tri == 1 ? 0 : 1;
    const FpModes &mr = modes[p.o], &mz = modes[2];
    const long long plane = (long long)g.ny * ld;
    p.nr = p.o ? g.ny : g.nx;
    p.nz = g.nz;
    p.fo = mr.fold;
    p.he = mr.ne;
    p.ho = mr.no;
    p.fz = mz.fold;
    p.ne = mz.ne;
    p.no = mz.no;
    p.off = mz.off;
    p.ld = ld;
    for (int h = 0; h < 2; h++) {
        p.mz[h] = m[2][h];
        p.mr[h] = m[p.o][h];
        p.lz[h] = mz.ldm[h];
        p.lr[h] = mr.ldm[h];
    }
    p.sr = p.o ? ld : plane;
    p.sb = p.o ? plane : ld;
    return p;
}

template <typename T>
template <typename S>
void FastPoisson<T>::front(cudaStream_t s, const S *r, T *out, const int *gate) {
    if constexpr (sizeof(T) == 4) {
        FpPlane p = fpp_plane(A_.g, tri_, modes_, ld_, fwd_);
        p.s2 = std::max((p.fz ? p.off + p.ne : p.nz) * FPP_PITCH, p.he * FPP_COLS);
        p.s3 = p.s2 + p.ne * FPP_COLS;
        launch_pdl(k_fp_front<S>, dim3(p.o ? A_.g.nx : A_.g.ny, p.fo ? 2 : 1), FPP_THREADS,
                   sizeof(float) * (p.s3 + p.he * FPP_ROWS), s, A_, r, out, p, nghost_ > 0 || nsolid_ > 0 ? 1 : 0,
                   (const T *)gscale_, gate);
    }
}

template <typename T>
template <typename S>
void FastPoisson<T>::rear(cudaStream_t s, const S *r, const T *in, T *z, const int *gate) {
    if constexpr (sizeof(T) == 4) {
        FpPlane p = fpp_plane(A_.g, tri_, modes_, ld_, bwd_);
        const int nkz = (p.ne + FPP_ROWS - 1) / FPP_ROWS * FPP_ROWS;
        p.s2 = std::max((p.he + p.ho) * FPP_COLS, p.ld * FPP_PITCH);
        p.s3 = p.s2 + (p.he + p.ho) * FPP_HALF;
        launch_pdl(k_fp_rear<S>, dim3(p.o ? A_.g.nx : A_.g.ny, (p.he + FPP_HALF - 1) / FPP_HALF), FPP_THREADS,
                   sizeof(float) * (p.s3 + (p.ne + p.no) * nkz), s, A_.g, r, in, z, p, (const T *)v0_, A_.p_singular,
                   A_.pinned, gate);
    }
}

// Forward transform of an axis, from F_[0] to F_[1] or back.
template <typename T>
template <int TM>
void FastPoisson<T>::forward(cudaStream_t s, int axis, const T *in, T *out, const int *gate) {
    const Grid &g = A_.g;
    const FpModes &m = modes_[axis];
    const int np = m.fold ? 2 : 1, H[2] = {m.ne, m.no};
    const long long plane = (long long)g.ny * ld_;
    FpGemm<T> p{};
    p.nb = np;
    unsigned gx = 0, gy = 0, batch = 1;
    for (int h = 0; h < np; h++) {
        p.K[h] = H[h];
        if (axis == 2) {   // rows of the data times the axis matrix
            p.a[h] = in + h * m.off;
            p.b[h] = fwd_[2][h];
            p.c[h] = out + h * m.off;
            p.M[h] = g.nx * g.ny;
            p.N[h] = p.ldb[h] = m.ldm[h];
            p.lda[h] = ld_;
        } else {           // the axis matrix times the lines of the data
            p.a[h] = fwd_[axis][h];
            p.b[h] = in;
            p.c[h] = out + (long long)h * m.off * (axis == 0 ? plane : ld_);
            p.M[h] = H[h];
            p.N[h] = p.ldb[h] = axis == 0 ? (int)plane : ld_;
            p.lda[h] = m.ldm[h];
        }
        gx = std::max(gx, (unsigned)((p.N[h] + TM - 1) / TM));
        gy = std::max(gy, (unsigned)((p.M[h] + TM - 1) / TM));
    }
    p.ldc = axis == 0 ? (int)plane : ld_;
    if (axis == 1) {
        p.sb = p.sc = plane;
        batch = g.nx;
    }
    p.fold = m.fold && axis != 2 ? (axis == 0 ? g.nx : g.ny) : 0;
    const dim3 grd(gx, gy, batch * np);
    if (axis == 2) launch_pdl(k_fp_gemm<T, TM, false>, grd, 64, 0, s, p, gate);
    else launch_pdl(k_fp_gemm<T, TM, true>, grd, 64, 0, s, p, gate);
}

// Backward transform along x or y.
template <typename T>
template <int TM>
void FastPoisson<T>::backward(cudaStream_t s, int axis, const T *in, T *out, const int *gate) {
    const Grid &g = A_.g;
    const FpModes &m = modes_[axis];
    const long long plane = (long long)g.ny * ld_;
    FpBack<T> p{};
    p.c = out;
    p.M = m.ne;
    p.N = p.ldc = axis == 0 ? (int)plane : ld_;
    for (int h = 0; h < 2; h++) {
        p.a[h] = bwd_[axis][h];
        p.b[h] = in + (long long)h * m.off * p.ldc;
        p.K[h] = h ? m.no : m.ne;
        p.lda[h] = m.ldm[h];
        p.ldb[h] = p.ldc;
    }
    if (axis == 1) p.sb = p.sc = plane;
    p.fold = m.fold;
    p.n = axis == 0 ? g.nx : g.ny;
    const int MA = m.fold ? TM / 2 : TM;
    const dim3 grd((p.N + TM - 1) / TM, (p.M + MA - 1) / MA, axis == 1 ? g.nx : 1);
    if (m.fold) launch_pdl(k_fp_back<T, TM, false, true, T>, grd, 64, 0, s, p, FpScatter<T, T>{}, gate);
    else launch_pdl(k_fp_back<T, TM, false, false, T>, grd, 64, 0, s, p, FpScatter<T, T>{}, gate);
}

template <typename T>
template <typename S>
void FastPoisson<T>::run(cudaStream_t s, const S *r, T *z, const int *gate) {
    // The smaller tile where the larger would leave SMs without work: FP32
    // below two 64-tiles per SM, FP64 (two multiply-adds per clock and SM, so
    // an uneven share of tiles is an uneven share of the time) below twelve
    // 32-tiles per SM.
    const Grid &g = A_.g;
    auto tiles = [&](int t) { return (long long)((g.nx * g.ny + t - 1) / t) * ((ld_ + t - 1) / t); };
    if constexpr (sizeof(T) == 8) {
        if (tiles(32) < 12 * 152) run_tiled<16, S>(s, r, z, gate);
        else run_tiled<32, S>(s, r, z, gate);
    } else {
        if (tiles(64) < 2 * 152) run_tiled<32, S>(s, r, z, gate);
        else run_tiled<64, S>(s, r, z, gate);
    }
}

template <typename T>
template <int TM, typename S>
void FastPoisson<T>::run_tiled(cudaStream_t s, const S *r, T *z, const int *gate) {
    const Grid &g = A_.g;
    const FpModes &mz = modes_[2];
    int k = 0;
    const int body = nghost_ > 0 || nsolid_ > 0;
    T *x = F_[0], *y = F_[1];
    auto turn = [&](int axis, bool fwd) {
        if (fwd) forward<TM>(s, axis, x, y, gate);
        else backward<TM>(s, axis, x, y, gate);
        std::swap(x, y);
        k++;
    };
    if (plane_) {
        front(s, r, x, gate);
    } else {
        launch_pdl(k_fp_gather<T, S>, dim3((mz.off + 31) / 32, (g.ny + 7) / 8, (g.nx + FP_GPLANES - 1) / FP_GPLANES),
                   dim3(32, 8), 0, s, A_, r, F_[0], mz, ld_, body, (const T *)gscale_, gate);
        turn(2, true);
        if (tri_ != 1) turn(1, true);
    }
    if (tri_ == -1 || (tri_ == 1 && !plane_)) turn(0, true);
    FpPin<T> pin{};
    pin.singular = A_.p_singular;
    pin.f2 = row0_[2];
    pin.z2 = zero_[2];
    const long long plane = (long long)g.ny * ld_;
    if (tri_ >= 0) {
        const int o = tri_ == 0 ? 1 : 0, n = tri_ == 0 ? g.nx : g.ny;
        const long long st = tri_ == 0 ? plane : ld_, outer = tri_ == 0 ? ld_ : plane;
        pin.w = dtri_;
        pin.zero = zero_[o] * outer + zero_[2];
        pin.f1 = row0_[o];
        pin.z1 = zero_[o];
        launch_pdl(n <= 16 * FP_SEG ? k_fp_tri<T, 512> : k_fp_tri<T, 1024>,
                   dim3((ld_ + 31) / 32, o == 1 ? g.ny : g.nx), dim3(32, (n + FP_SEG - 1) / FP_SEG), 0, s, (const T *)inv_,
                   A_.km[tri_] + 2, A_.kp[tri_] + 2, n, st, outer, ld_, pin, (const T *)x, y, gate);
    } else {
        pin.w = nullptr;
        pin.zero = zero_[0] * plane + (long long)zero_[1] * ld_ + zero_[2];
        pin.f1 = row0_[1];
        pin.z1 = zero_[1];
        launch_pdl(k_fp_diag<T>, dim3((ld_ + 31) / 32, (g.ny + 7) / 8, g.nx), dim3(32, 8), 0, s, (const T *)inv_,
                   g.ny, ld_, pin, (const T *)dtri_, (const T *)x, y, gate);
    }
    std::swap(x, y);
    if (tri_ == -1 || (tri_ == 1 && !plane_)) turn(0, false);
    if (plane_) {
        rear(s, r, x, z, gate);
    } else {
        if (tri_ != 1) turn(1, false);
        // Along z, into the padded array.
        FpScatter<T, S> sc{g, r, v0_, A_.pinned, A_.p_singular, ld_};
        FpBack<T> p{};
        p.c = z;
        p.M = g.nx * g.ny;
        p.N = mz.ne;
        for (int h = 0; h < 2; h++) {
            p.a[h] = x + h * mz.off;
            p.b[h] = bwd_[2][h];
            p.K[h] = h ? mz.no : mz.ne;
            p.lda[h] = ld_;
            p.ldb[h] = mz.ldm[h];
        }
        p.fold = mz.fold;
        p.n = g.nz;
        const int NB = mz.fold ? TM / 2 : TM;
        const dim3 grd((p.N + NB - 1) / NB, (p.M + TM - 1) / TM);
        if (mz.fold) launch_pdl(k_fp_back<T, TM, true, true, S>, grd, 64, 0, s, p, sc, gate);
        else launch_pdl(k_fp_back<T, TM, true, false, S>, grd, 64, 0, s, p, sc, gate);
    }
    const int nout = A_.sw.nout;
    auto edges = [&](int outer, int solids, int swept) {
        launch_pdl(k_fp_edges<T, S>, (outer + solids + swept + 255) / 256, 256, 0, s, A_, r, z, A_.sw.outer, outer,
                   (const int *)solid_, solids, solid_partners_, patch_.P, (const T *)near_val_, swept, gate);
        k++;
    };
    k += 3;
    if (nghost_ > 0) {
        if (near_outer_) edges(nout, nsolid_, 0);   // the sweeps read outer values
        launch_pdl(k_fp_patch<T, S>, npatch_, FP_PT, 0, s, patch_, r, (const T *)z, near_val_, FP_SWEEPS<T>, gate);
        k++;
        if (near_outer_) edges(0, 0, patch_.ncell);
    }
    if (near_outer_ || nghost_ == 0) edges(nout, nsolid_, 0);
    else edges(nout, nsolid_, patch_.ncell);
    note_launches(k);
    launches_ = k;
}

template <typename T>
void FastPoisson<T>::apply(cudaStream_t s, const T *r, T *z, const int *gate) {
    run(s, r, z, gate);
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
