// FP32 explicit stages of the IBM3D_MIXED32 step.
//
// The same fractional step as step_kernels.cu (src/ibm3d_fracstep.c:117-487,
// 709-805), with the explicit stencils in FP32 and the momentum solve in
// increment form:
//
//   A u* = b   becomes   A e = c,  c = b - A u^n,  u* = u^n + e.
//
// For a fluid row, with k the Crank-Nicolson coefficients,
//   b   = u_P + sum k (u_nb - u_P) + r,   r = -dt/2 (3 N - N_prev) - dt G_c p + dt f - dt div tau
//   A x = x_P - sum k (x_nb - x_P)
// so c = 2 sum k (u_nb - u_P) + r: the O(1) parts cancel analytically and
// c is O(dt).  Evaluated in FP32, its error is ~1e-7 of |c| plus ~1e-8 of
// |u| (the FP32 neighbour differences), far below the 1e-6 relative
// momentum tolerance, and the FP64 state u^{n+1} = u^n + (e - dt G_c p')
// only ever receives O(dt) increments rounded to FP32.  The solve stops on
// the reference's test ||b - A u*|| < tol ||b|| (||b|| is reduced here).
//
// U* is computed in FP32 and stored widened to FP64; the Poisson right-hand
// side is the FP64 divergence of those stored faces, so the projection
// (FP64) drives div U^{n+1} of the stored faces to the solve's tolerance
// exactly as in the FP64 step.  Every face is computed by both cells that
// share it; the FP32 arithmetic uses explicitly rounded operations so both
// get the same bits.
//
// FP64 fields are read as FP32 with d2f_int / written with f2d_int
// (integer pipe; see common.cuh).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "krylov.h"
#include "ops.cuh"

namespace ibm {

namespace {

constexpr int K32_THREADS = 256;
constexpr int K32_BLOCKS = 1216;  // 8 per SM on 152 SMs; grid-stride
constexpr int UN_TK = 32, UN_TJ = 8, UN_PLANES = 8;

// An FP64 field value in FP32; NaN (solid cells) becomes 0, the value the
// momentum solve gives solid rows.
__device__ __forceinline__ float ld32(const double *__restrict__ a, long long P) {
    const float v = d2f_int(__ldg(a + P));
    return v == v ? v : 0.0f;
}

__device__ __forceinline__ float ldp32(const double *__restrict__ a, long long P) { return d2f_int(__ldg(a + P)); }

// Outer row of the FP32 momentum operator applied to the current velocity
// component (the rows of ops.cuh outer_row, values loaded from FP64).
__device__ __forceinline__ float outer_row_u(const OpT<float> &c, int comp, const double *__restrict__ u, long long P,
                                             int i, int j, int k, int f, int L) {
    const BCRow<float> &F = c.bc[f];
    const int axis = face_axis(f);
    const long long s = axis == 0 ? c.g.sx : axis == 1 ? c.g.sy : 1;
    const long long in = face_low(f) ? s : -s;
    switch (outer_row_kind(OP_MOM, F.type, comp, axis)) {
    case ROW_DIR: return F.dir_o[L - 1] * ld32(u, P) + F.dir_m[L - 1] * ld32(u, P + (2 * L - 1) * in);
    case ROW_NEU: return ld32(u, P) - ld32(u, P + (2 * L - 1) * in);
    case ROW_PER: return ld32(u, P) - ld32(u, periodic_image(c.g, i, j, k));
    default: return F.ext_o[L - 1] * ld32(u, P) - ld32(u, P + in) + F.ext_2[L - 1] * ld32(u, P + 2 * in);
    }
}

}  // namespace

// Tiles of the marching kernels: 32 (k) x 8 (j) columns over up to UN_PLANES
// planes of i, fewer on grids that would leave SMs without a block (a
// 32^3 grid in 8-plane tiles is 16 blocks, each a serial chain of 8 planes:
// the projection took 46 us, U* 43 us; in 1-plane tiles 11 and 18 us).
struct Tiles {
    int tk, tj, planes, nb;
    explicit Tiles(const Grid &g) {
        tk = (g.nz + UN_TK - 1) / UN_TK;
        tj = (g.ny + UN_TJ - 1) / UN_TJ;
        planes = UN_PLANES;
        auto blocks = [&]() { return (long long)tk * tj * ((g.nx + planes - 1) / planes); };
        while (planes > 1 && blocks() < 2 * 152) planes /= 2;
        nb = (int)blocks();
    }
};

// ------------------------------------------------------------------------
// calc_N + momentum right-hand side (src/ibm3d_fracstep.c:117-170,
// 237-352) in FP32, written as the increment system's right-hand side c
// (3 components, w.b32 layout l*n + P) and N (FP32).  The last block
// stores ||b||^2 and ||c||^2 per component in the increment solve's
// scalars (out[l].bnorm2, .rnorm2).
//
// Blocks [0, nb) take tiles of interior columns and march over planes of i;
// the others take the outer rows.  Each FP64 value of u and p is loaded and
// converted once per tile: a plane's values sit in shared memory with a halo
// of one cell (y and z neighbours), the planes before and after in
// registers, and the next plane's loads are in flight while a plane is
// computed.  (One thread per padded cell loading its neighbours converted
// 25 values per cell behind two load latencies: sphere 192x128x128 232 ->
// 148 us, against 47 us of HBM time.)
// ------------------------------------------------------------------------
__global__ void __launch_bounds__(K32_THREADS)
k_conv_rhs32(const Grid g, const AxisF ax, const AxisF ay, const AxisF az, const OpT<float> A, const BCSet bc,
             const uint8_t *__restrict__ flag, const Conv32Args a, const float dt, const float f1, const float f2,
             const float f3, const int les, const Tiles tl, const int *__restrict__ outer, const int nout,
             double *partials, unsigned int *counter, IRScal *out) {
    __shared__ double smem[32 * 6];
    __shared__ float sp[2][4][UN_TJ + 2][UN_TK + 2];   // u1, u2, u3, p of a plane, with halo
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // ||b||^2 (3), ||c||^2 (3)
    const long long n = g.ncell;
    const float NaNf = __int_as_float(0x7fc00000);
    if ((int)blockIdx.x >= tl.nb) {
        const int t = (blockIdx.x - tl.nb) * K32_THREADS + threadIdx.x;
        if (t < nout) {
            // Outer rows: the velocity BC value (VELOCITY faces) or 0.
            const long long P = outer[t];
            int i, j, k;
            cijk_g(g, P, i, j, k);
            int layer;
            const int f = owner_face(g, i, j, k, layer);
            const BCFace &F = bc.f[f];
            const bool vel = F.type == BCT_VELOCITY;
            const double *sv = F.scur ? F.scur + face_line(g, f, i, j, k) : nullptr;
#pragma unroll
            for (int l = 0; l < 3; l++) {
                const float bv = vel ? d2f_int(sv ? sv[l * F.nt] : F.val[l]) : 0.0f;
                const float cv = bv - outer_row_u(A, l, a.u[l], P, i, j, k, f, layer);
                a.c[l * n + P] = cv;
                acc[l] += bv * bv;
                acc[3 + l] += cv * cv;
            }
        }
    } else {
        int b = blockIdx.x;
        const int bk = b % tl.tk;
        b /= tl.tk;
        const int bj = b % tl.tj, bi = b / tl.tj;
        const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
        const int k = bk * UN_TK + tx, j = bj * UN_TJ + ty;
        const int i0 = bi * tl.planes, i1 = min(i0 + tl.planes, g.nx);
        const bool live = j < g.ny && k < g.nz;
        const long long sx = g.sx, sy = g.sy;
        // This thread's column (clamped into the padded box) and its halo
        // cell: 2 x 32 cells above and below, 2 x 8 left and right.
        const int jc = min(j, g.ny + 1), kc = min(k, g.nz + 1);
        const bool halo = t < 2 * UN_TK + 2 * UN_TJ;
        const int hy = t < UN_TK ? 0 : t < 2 * UN_TK ? UN_TJ + 1 : 1 + (t - 2 * UN_TK) % UN_TJ;
        const int hx = t < 2 * UN_TK ? 1 + (t & 31) : t < 2 * UN_TK + UN_TJ ? 0 : UN_TK + 1;
        const int hj = min(bj * UN_TJ + hy - 1, g.ny + 1), hk = min(bk * UN_TK + hx - 1, g.nz + 1);
        long long P = cidx(g, i0, jc, kc), H = cidx(g, i0, hj, hk);
        const double *fld[4] = {a.u[0], a.u[1], a.u[2], a.p};
        const int J = jc + 2, K = kc + 2;
        const float wmy0 = ay.wm[J], wpy0 = ay.wp[J], wmy1 = ay.wm[min(J + 1, g.ny + 3)], wpy1 = ay.wp[min(J + 1, g.ny + 3)];
        const float wmz0 = az.wm[K], wpz0 = az.wp[K], wmz1 = az.wm[min(K + 1, g.nz + 3)], wpz1 = az.wp[min(K + 1, g.nz + 3)];
        const float rdy = ay.rd[J], rdz = az.rd[K], gy = ay.rdcc[J], gz = az.rdcc[K];
        const float kS = ay.km[J], kN = ay.kp[J], kD = az.km[K], kU = az.kp[K];
        const float ff[3] = {f1, f2, f3};
        float vw[4], vc[4];
        double nx[4], nh[4], Uen;   // the next plane: own, halo, high x face
#pragma unroll
        for (int q = 0; q < 4; q++) {
            vw[q] = d2f_int(fld[q][P - sx]);
            vc[q] = d2f_int(fld[q][P]);
            const float hv = halo ? d2f_int(fld[q][H]) : 0.0f;
            if (q < 3) {
                vw[q] = vw[q] == vw[q] ? vw[q] : 0.0f;
                vc[q] = vc[q] == vc[q] ? vc[q] : 0.0f;
            }
            sp[0][q][ty + 1][tx + 1] = vc[q];
            if (halo) sp[0][q][hy][hx] = q < 3 && hv != hv ? 0.0f : hv;
        }
        float Uw = ldp32(a.U[0], P);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            nx[q] = fld[q][P + sx];
            nh[q] = halo ? fld[q][H + sx] : 0.0;
        }
        Uen = a.U[0][P + sx];
        int buf = 0;
        for (int i = i0; i < i1; i++, P += sx, H += sx) {
            const int I = i + 2;
            // Everything else this plane needs, and then the next plane's
            // loads, before the arithmetic.
            const uint8_t fl = flag[P];
            const double Vs64 = a.U[1][P], Vn64 = a.U[1][P + (live ? sy : 0)], Wd64 = a.U[2][P],
                         Wu64 = a.U[2][P + (live ? 1 : 0)];
            float np[3];
#pragma unroll
            for (int l = 0; l < 3; l++) np[l] = a.Np[l][P];
            float ve[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ve[q] = d2f_int(nx[q]);
                if (q < 3) ve[q] = ve[q] == ve[q] ? ve[q] : 0.0f;
                sp[buf ^ 1][q][ty + 1][tx + 1] = ve[q];
                if (halo) {
                    const float hv = d2f_int(nh[q]);
                    sp[buf ^ 1][q][hy][hx] = q < 3 && hv != hv ? 0.0f : hv;
                }
            }
            const float Ue = d2f_int(Uen);
            if (i + 1 < i1) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    nx[q] = fld[q][P + 2 * sx];
                    if (halo) nh[q] = fld[q][H + 2 * sx];
                }
                Uen = a.U[0][P + 2 * sx];
            }
            __syncthreads();   // plane i complete (its stores precede the last barrier), i + 1 being written
            if (live) {
                float bv[3], cv[3];
                if (fl != FLUID) {
                    // Ghost rows (1 + w_self) x_g + sum w x = 0, solid rows x = 0.
                    const int q = fl == GHOST ? A.gid[P] : 0;
#pragma unroll
                    for (int l = 0; l < 3; l++) {
                        a.N[l][P] = NaNf;
                        bv[l] = 0.0f;
                        cv[l] = 0.0f;
                        if (fl == GHOST) {
                            float sum = 0.0f;
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const int m = A.gidx[8 * q + e];
                                if (m >= 0) sum += A.gw[8 * q + e] * ld32(a.u[l], m);
                            }
                            cv[l] = -((1.0f + A.gwself[q]) * vc[l] + sum);
                        }
                    }
                } else {
                    const float wmx0 = ax.wm[I], wpx0 = ax.wp[I], wmx1 = ax.wm[I + 1], wpx1 = ax.wp[I + 1];
                    const float rdx = ax.rd[I], kW = ax.km[I], kE = ax.kp[I], gx = ax.rdcc[I];
                    const float Vs = d2f_int(Vs64), Vn = d2f_int(Vn64), Wd = d2f_int(Wd64), Wu = d2f_int(Wu64);
#pragma unroll
                    for (int l = 0; l < 3; l++) {
                        const float uc = vc[l], uW = vw[l], uE = ve[l];
                        const float uS = sp[buf][l][ty][tx + 1], uN = sp[buf][l][ty + 2][tx + 1];
                        const float uD = sp[buf][l][ty + 1][tx], uU = sp[buf][l][ty + 1][tx + 2];
                        const float fw = uW * wmx0 + uc * wpx0, fe = uc * wmx1 + uE * wpx1;
                        const float fs = uS * wmy0 + uc * wpy0, fn = uc * wmy1 + uN * wpy1;
                        const float fd = uD * wmz0 + uc * wpz0, fu = uc * wmz1 + uU * wpz1;
                        const float Nl = (Ue * fe - Uw * fw) * rdx + (Vn * fn - Vs * fs) * rdy + (Wu * fu - Wd * fd) * rdz;
                        a.N[l][P] = Nl;
                        float dp;
                        if (l == 0) dp = (ve[3] - vw[3]) * gx;
                        else if (l == 1) dp = (sp[buf][3][ty + 2][tx + 1] - sp[buf][3][ty][tx + 1]) * gy;
                        else dp = (sp[buf][3][ty + 1][tx + 2] - sp[buf][3][ty + 1][tx]) * gz;
                        float divtau = 0.0f;
                        if (les) {
                            const int t1 = l == 0 ? 0 : l == 1 ? 1 : 2;
                            const int t2 = l == 0 ? 1 : l == 1 ? 3 : 4;
                            const int t3 = l == 0 ? 2 : l == 1 ? 4 : 5;
                            divtau = (ldp32(a.tau[t1], P + sx) - ldp32(a.tau[t1], P - sx)) * gx +
                                     (ldp32(a.tau[t2], P + sy) - ldp32(a.tau[t2], P - sy)) * gy +
                                     (ldp32(a.tau[t3], P + 1) - ldp32(a.tau[t3], P - 1)) * gz;
                        }
                        const float fl_ = a.force ? ldp32(a.force, l * n + P) : ff[l];
                        const float lap = kW * (uW - uc) + kE * (uE - uc) + kS * (uS - uc) + kN * (uN - uc) +
                                          kD * (uD - uc) + kU * (uU - uc);
                        const float rest = -dt / 2 * (3 * Nl - np[l]) - dt * dp + dt * fl_ - dt * divtau;
                        bv[l] = uc + lap + rest;
                        cv[l] = 2 * lap + rest;
                    }
                }
#pragma unroll
                for (int l = 0; l < 3; l++) {
                    a.c[l * n + P] = cv[l];
                    acc[l] += bv[l] * bv[l];
                    acc[3 + l] += cv[l] * cv[l];
                }
            }
            __syncthreads();   // plane i is read before i + 2 overwrites it
#pragma unroll
            for (int q = 0; q < 4; q++) {
                vw[q] = vc[q];
                vc[q] = ve[q];
            }
            Uw = Ue;
            buf ^= 1;
        }
    }
    double tot[6];
    block_reduce<6, 6, float>(acc, tot, smem);
    if (!publish_partials<6>(tot, partials, counter)) return;
    double all[6];
    reduce_partials<6, 6>(partials, gridDim.x, all, smem);
    if (threadIdx.x == 0) {
        for (int l = 0; l < 3; l++) {
            IRScal &s = out[l];
            s.bnorm2 = all[l];
            s.rnorm2 = all[3 + l];
            s.rmax = 0.0;
            s.divmax = 0.0;
            s.scale = 1.0;
            s.state = all[3 + l] == 0.0 ? KS_DONE : KS_RUN;
            s.outer = 0;
            s.inner = 0;
        }
        *counter = 0;
    }
}

void launch_conv_rhs32(cudaStream_t s, const Grid &g, const AxisF axf[3], const OpT<float> &A, const BCSet &bc,
                       const uint8_t *flag, const Conv32Args &a, double dt, const double f[3], int les,
                       double *partials, unsigned int *counter, IRScal *out) {
    const int no = A.sw.nout, ob = (no + K32_THREADS - 1) / K32_THREADS;
    const Tiles t(g);
    k_conv_rhs32<<<t.nb + ob, K32_THREADS, 0, s>>>(g, axf[0], axf[1], axf[2], A, bc, flag, a, (float)dt, (float)f[0],
                                                   (float)f[1], (float)f[2], les, t, A.sw.outer, no, partials,
                                                   counter, out);
    note_launches(1);
}

// ------------------------------------------------------------------------
// calc_u_tilde + calc_U_star (src/ibm3d_fracstep.c:388-487) in FP32 from
// u* = u^n + e, with the pressure-Poisson right-hand side
// (src/ibm3d_fracstep.c:530-647) in FP64 from the stored faces, in two
// passes: u~ = u* + dt G_c p in FP32 on every cell the faces read (i, j, k
// in [-1, N]), then the faces and the right-hand side over tiles of 32 (k)
// x 8 (j) columns marching over planes of i, each face computed once (x
// faces carried along i, y faces in shared memory, z faces by warp
// shuffle).  Tile-edge threads compute their high faces as well; face32t is
// explicitly rounded, so both computations of such a face give its bits.
// ------------------------------------------------------------------------
namespace {

__device__ __forceinline__ float ustar_of(double u, float e) {
    const float v = d2f_int(u);
    return __fadd_rn(v == v ? v : 0.0f, e);
}
__device__ __forceinline__ float ustar_at(const double *__restrict__ u, const float *__restrict__ e, long long P) {
    return ustar_of(u[P], e[P]);
}

__device__ __forceinline__ bool fg_pair32(uint8_t a, uint8_t b) {
    return (a == FLUID && b == GHOST) || (a == GHOST && b == FLUID);
}

// U* on a face between the cells m and p of an axis (weights wm, wp; rdc
// the reciprocal of their distance): from u~ (utm, utp) and the pressure
// difference, or, across a fluid-ghost pair, from u*.
__device__ __forceinline__ float face32t(float wm, float wp, float rdc, float utm, float utp, float pm, float pp, float dt) {
    const float gf = __fmul_rn(__fsub_rn(pp, pm), rdc);
    return __fsub_rn(__fadd_rn(__fmul_rn(utm, wm), __fmul_rn(utp, wp)), __fmul_rn(dt, gf));
}
__device__ __forceinline__ float face32g(const double *__restrict__ u, const float *__restrict__ e, long long Pm,
                                         long long Pp, float wm, float wp) {
    return __fadd_rn(__fmul_rn(ustar_at(u, e, Pm), wm), __fmul_rn(ustar_at(u, e, Pp), wp));
}

}  // namespace

// Grid (ceil((nz + 2) / 32), ceil((ny + 2) / 8), nx + 2) of 32 x 8 threads,
// no index division.
__global__ void __launch_bounds__(256)
k_utilde32(const Grid g, const AxisF ax, const AxisF ay, const AxisF az, const Ustar32Args a, float *__restrict__ ut,
           const float dt) {
    const int k = blockIdx.x * 32 + threadIdx.x - 1, j = blockIdx.y * 8 + threadIdx.y - 1, i = (int)blockIdx.z - 1;
    if (k > g.nz || j > g.ny) return;
    const long long sx = g.sx, sy = g.sy, P = cidx(g, i, j, k);
    const double pe = a.p[P + sx], pw = a.p[P - sx], pn = a.p[P + sy], ps = a.p[P - sy], pu = a.p[P + 1], pd = a.p[P - 1];
    const double u0 = a.u[0][P], u1 = a.u[1][P], u2 = a.u[2][P];
    const float e0 = a.e[0][P], e1 = a.e[1][P], e2 = a.e[2][P];
    const float gx = (d2f_int(pe) - d2f_int(pw)) * ax.rdcc[i + 2];
    const float gy = (d2f_int(pn) - d2f_int(ps)) * ay.rdcc[j + 2];
    const float gz = (d2f_int(pu) - d2f_int(pd)) * az.rdcc[k + 2];
    ut[P] = ustar_of(u0, e0) + dt * gx;
    ut[g.ncell + P] = ustar_of(u1, e1) + dt * gy;
    ut[2 * g.ncell + P] = ustar_of(u2, e2) + dt * gz;
}

__global__ void __launch_bounds__(UN_TK * UN_TJ, 3)
k_ustar_faces32(const Grid g, const AxisF ax, const AxisF ay, const AxisF az, const Axis ax64, const Axis ay64,
                const Axis az64, const BCSet bc, const uint8_t *__restrict__ flag, const Ustar32Args a,
                const float *__restrict__ ut, const float dt, const double m2re, const Tiles tl) {
    __shared__ float sVs[2][UN_TJ][UN_TK];
    int b = blockIdx.x;
    const int bk = b % tl.tk;
    b /= tl.tk;
    const int bj = b % tl.tj, bi = b / tl.tj;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int k = bk * UN_TK + tx, j = bj * UN_TJ + ty;
    const int i0 = bi * tl.planes, i1 = min(i0 + tl.planes, g.nx);
    const bool live = j < g.ny && k < g.nz;
    const bool own_vn = ty == UN_TJ - 1 || j == g.ny - 1;
    const bool own_wu = tx == UN_TK - 1 || k == g.nz - 1;
    const long long sx = g.sx, sy = g.sy, n = g.ncell;
    const float *ut0 = ut, *ut1 = ut + n, *ut2 = ut + 2 * n;
    // Threads off the grid follow a column inside it and store nothing.
    const int jc = min(j, g.ny - 1), kc = min(k, g.nz - 1), J = jc + 2, K = kc + 2;
    const float wms = ay.wm[J], wps = ay.wp[J], rds = ay.rdc[J], wmn = ay.wm[J + 1], wpn = ay.wp[J + 1], rdn = ay.rdc[J + 1];
    const float wmd = az.wm[K], wpd = az.wp[K], rdd = az.rdc[K], wmu = az.wm[K + 1], wpu = az.wp[K + 1], rdu = az.rdc[K + 1];
    long long P = cidx(g, i0, jc, kc);
    uint8_t fc = flag[P];
    float pc = d2f_int(a.p[P]), u0c = ut0[P];
    float Uw;
    {
        const int I = i0 + 2;
        Uw = fg_pair32(flag[P - sx], fc) ? face32g(a.u[0], a.e[0], P - sx, P, ax.wm[I], ax.wp[I])
                                         : face32t(ax.wm[I], ax.wp[I], ax.rdc[I], ut0[P - sx], u0c, d2f_int(a.p[P - sx]), pc, dt);
    }
    int buf = 0;
    for (int i = i0; i < i1; i++, P += sx) {
        const int I = i + 2;
        // Every load of the plane before its arithmetic.
        const uint8_t fe = flag[P + sx], fs = flag[P - sy], fd = flag[P - 1];
        const float u0e = ut0[P + sx], u1s = ut1[P - sy], u1c = ut1[P], u2d = ut2[P - 1], u2c = ut2[P];
        const double pe64 = a.p[P + sx], ps64 = a.p[P - sy], pd64 = a.p[P - 1];
        const double dinv = a.dinv[P];
        uint8_t fn = SOLID, fu = SOLID;
        float u1n = 0.f, u2u = 0.f;
        double pn64 = 0.0, pu64 = 0.0;
        if (own_vn) {
            fn = flag[P + sy];
            u1n = ut1[P + sy];
            pn64 = a.p[P + sy];
        }
        if (own_wu) {
            fu = flag[P + 1];
            u2u = ut2[P + 1];
            pu64 = a.p[P + 1];
        }
        const float pe = d2f_int(pe64);
        float Ue = face32t(ax.wm[I + 1], ax.wp[I + 1], ax.rdc[I + 1], u0c, u0e, pc, pe, dt);
        float Vs = face32t(wms, wps, rds, u1s, u1c, d2f_int(ps64), pc, dt);
        float Wd = face32t(wmd, wpd, rdd, u2d, u2c, d2f_int(pd64), pc, dt);
        float Vn = 0.f, Wu = 0.f;
        if (own_vn) Vn = face32t(wmn, wpn, rdn, u1c, u1n, pc, d2f_int(pn64), dt);
        if (own_wu) Wu = face32t(wmu, wpu, rdu, u2c, u2u, pc, d2f_int(pu64), dt);
        if (fg_pair32(fc, fe)) Ue = face32g(a.u[0], a.e[0], P, P + sx, ax.wm[I + 1], ax.wp[I + 1]);
        if (fg_pair32(fs, fc)) Vs = face32g(a.u[1], a.e[1], P - sy, P, wms, wps);
        if (fg_pair32(fd, fc)) Wd = face32g(a.u[2], a.e[2], P - 1, P, wmd, wpd);
        if (own_vn && fg_pair32(fc, fn)) Vn = face32g(a.u[1], a.e[1], P, P + sy, wmn, wpn);
        if (own_wu && fg_pair32(fc, fu)) Wu = face32g(a.u[2], a.e[2], P, P + 1, wmu, wpu);
        sVs[buf][ty][tx] = Vs;
        const float wnext = __shfl_down_sync(0xffffffffu, Wd, 1);
        __syncthreads();
        if (!own_vn) Vn = sVs[buf][min(ty + 1, UN_TJ - 1)][tx];
        if (!own_wu) Wu = wnext;
        buf ^= 1;
        if (live) {
            const double Uw64 = f2d_int(Uw), Ue64 = f2d_int(Ue), Vs64 = f2d_int(Vs), Vn64 = f2d_int(Vn);
            const double Wd64 = f2d_int(Wd), Wu64 = f2d_int(Wu);
            a.Us[0][P] = Uw64;
            a.Us[1][P] = Vs64;
            a.Us[2][P] = Wd64;
            if (i == g.nx - 1) a.Us[0][P + sx] = Ue64;
            if (j == g.ny - 1) a.Us[1][P + sy] = Vn64;
            if (k == g.nz - 1) a.Us[2][P + 1] = Wu64;
            double rhs = 0.0;
            if (fc == FLUID && !(bc.p_singular && i == 0 && j == 0 && k == 0)) {
                const double div = (Ue64 - Uw64) * ax64.rd[I] + (Vn64 - Vs64) * ay64.rd[J] + (Wu64 - Wd64) * az64.rd[K];
                rhs = div * m2re * dinv;   // -div / (2 Re coeffsum)
            }
            a.b[P] = rhs;
        }
        Uw = Ue;
        fc = fe;
        pc = pe;
        u0c = u0e;
    }
}

// Outer rows of the Poisson right-hand side: the pressure-BC increments
// p_bc(t + dt) - p_bc(t) (0 for constant values), over the outer-cell list.
__global__ void __launch_bounds__(256)
k_prhs_outer(const Grid g, const BCSet bc, const int *__restrict__ outer, const int nout, double *b) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nout) return;
    const long long P = outer[t];
    int i, j, k;
    cijk_g(g, P, i, j, k);
    int layer;
    const int face = owner_face(g, i, j, k, layer);
    const BCFace &F = bc.f[face];
    double v = 0.0;
    if (F.scur && (F.type == BCT_PRESSURE || F.type == BCT_VELPERIODIC)) {
        const int q = 3 * F.nt + face_line(g, face, i, j, k);
        v = F.snxt[q] - F.scur[q];
    }
    b[P] = v;
}

void launch_ustar_prhs32_tiled(cudaStream_t s, const Grid &g, const AxisF axf[3], const Axis ax64[3],
                               const BCSet &bc, const uint8_t *flag, const Ustar32Args &a, float *ut, double dt,
                               double Re, const int *outer, int nout) {
    k_utilde32<<<dim3((g.nz + 33) / 32, (g.ny + 9) / 8, g.nx + 2), dim3(32, 8), 0, s>>>(g, axf[0], axf[1], axf[2], a, ut,
                                                                                       (float)dt);
    const Tiles t(g);
    k_ustar_faces32<<<t.nb, dim3(UN_TK, UN_TJ), 0, s>>>(g, axf[0], axf[1], axf[2], ax64[0], ax64[1], ax64[2], bc, flag, a,
                                                        ut, (float)dt, -1.0 / (2.0 * Re), t);
    if (nout > 0) k_prhs_outer<<<(nout + 255) / 256, 256, 0, s>>>(g, bc, outer, nout, a.b);
    note_launches(nout > 0 ? 3 : 2);
}

// ------------------------------------------------------------------------
// update_next (src/ibm3d_fracstep.c:709-805) on tiles: each thread owns a
// (j, k) column of a 32 x 8 tile and marches over the planes of i of its
// tile.  The x face between cells i and i+1 is computed once and carried
// to the next plane as its low face; the high y face of a cell is the low
// y face of the thread at j+1 (shared memory, one barrier per plane); the
// high z face is the low z face of the next lane (warp shuffle).  Tile-edge
// threads compute their high faces themselves.  Per fluid cell that is 3
// face updates on the FP64 pipe instead of 6; the maximum runs on the
// integer pipe and a plane's loads go out together (sphere 192x128x128 218
// -> 160 us; its 16 FP64 operations per cell take 96 us).  F32: the increment form of
// the FP32-stage step (the cell velocity takes the FP32 increment
// e - dt G_c p'); otherwise the FP64 step.
// ------------------------------------------------------------------------
template <bool F32>
__global__ void __launch_bounds__(UN_TK * UN_TJ, 3)
k_update_next_tiled(const Grid g, const Axis ax, const Axis ay, const Axis az, const DtAxis dx, const DtAxis dy,
                    const DtAxis dz, const AxisF axf, const AxisF ayf, const AxisF azf, const BCSet bc,
                    const uint8_t *__restrict__ flag, const NextArgs a64, const Next32Args a32, const double dt,
                    const Tiles tl, double *partials, unsigned int *counter, double *maxdiv_out) {
    __shared__ long long smem[32];
    __shared__ double sVs[2][UN_TJ][UN_TK];
    const double NaN = __longlong_as_double(0x7ff8000000000000LL);
    int b = blockIdx.x;
    const int bk = b % tl.tk;
    b /= tl.tk;
    const int bj = b % tl.tj, bi = b / tl.tj;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int k = bk * UN_TK + tx, j = bj * UN_TJ + ty;
    const int i0 = bi * tl.planes, i1 = min(i0 + tl.planes, g.nx);
    const bool live = j < g.ny && k < g.nz;
    const bool own_vn = ty == UN_TJ - 1 || j == g.ny - 1;
    const bool own_wu = tx == UN_TK - 1 || k == g.nz - 1;
    const long long sx = g.sx, sy = g.sy;
    const double *Us0 = F32 ? a32.Us[0] : a64.Us[0], *Us1 = F32 ? a32.Us[1] : a64.Us[1],
                 *Us2 = F32 ? a32.Us[2] : a64.Us[2];
    const double *pp = F32 ? a32.pp : a64.pp, *p = F32 ? a32.p : a64.p;
    double *const *Un = F32 ? a32.Un : a64.Un;
    double *const *un = F32 ? a32.un : a64.un;
    const double *const *uo = F32 ? a32.u : a64.us;   // u^n, or u*
    double *pn = F32 ? a32.pn : a64.pn;
    // Threads off the grid follow a column inside it and store nothing.
    const int jc = min(j, g.ny - 1), kc = min(k, g.nz - 1), J = jc + 2, K = kc + 2;
    const double dys = dy.dtrdc[J], dyn = dy.dtrdc[J + 1], dzd = dz.dtrdc[K], dzu = dz.dtrdc[K + 1];
    const double rdy = ay.rd[J], rdz = az.rd[K];
    long long mdiv = 0;   // max|div U| as the bits of a double >= 0 (ordered as integers; NaN largest)
    long long P = cidx(g, i0, jc, kc);
    uint8_t fc = flag[P];
    double ppc = pp[P], ppw = pp[P - sx];
    double Uw = flag[P - sx] != SOLID && fc != SOLID ? Us0[P] - dx.dtrdc[i0 + 2] * (ppc - ppw) : NaN;
    int buf = 0;
    for (int i = i0; i < i1; i++, P += sx) {
        const int I = i + 2;
        // Every load of the plane before its arithmetic (behind the flags'
        // tests they cost three latencies per plane).
        const uint8_t fe = flag[P + sx], fs = flag[P - sy], fd = flag[P - 1], fn = flag[P + sy], fu = flag[P + 1];
        const double ppe = pp[P + sx], pps = pp[P - sy], ppn = pp[P + sy], ppd = pp[P - 1], ppu = pp[P + 1];
        const double ue = Us0[P + sx], vs = Us1[P], wd = Us2[P], pc = p[P];
        const double o0 = uo[0][P], o1 = uo[1][P], o2 = uo[2][P];
        float e0 = 0.f, e1 = 0.f, e2 = 0.f;
        if (F32) {
            e0 = a32.e[0][P];
            e1 = a32.e[1][P];
            e2 = a32.e[2][P];
        }
        double vn = 0.0, wu = 0.0;
        if (own_vn) vn = Us1[P + sy];
        if (own_wu) wu = Us2[P + 1];
        const bool in = fc != SOLID;
        const double Ue = in && fe != SOLID ? ue - dx.dtrdc[I + 1] * (ppe - ppc) : NaN;
        const double Vs = in && fs != SOLID ? vs - dys * (ppc - pps) : NaN;
        const double Wd = in && fd != SOLID ? wd - dzd * (ppc - ppd) : NaN;
        double Vn = NaN, Wu = NaN;
        if (own_vn && in && fn != SOLID) Vn = vn - dyn * (ppn - ppc);
        if (own_wu && in && fu != SOLID) Wu = wu - dzu * (ppu - ppc);
        sVs[buf][ty][tx] = Vs;
        const double wnext = __shfl_down_sync(0xffffffffu, Wd, 1);
        __syncthreads();
        if (!own_vn) Vn = sVs[buf][min(ty + 1, UN_TJ - 1)][tx];
        if (!own_wu) Wu = wnext;
        buf ^= 1;
        if (live) {
            Un[0][P] = Uw;
            Un[1][P] = Vs;
            Un[2][P] = Wd;
            if (i == g.nx - 1) Un[0][P + sx] = Ue;
            if (j == g.ny - 1) Un[1][P + sy] = Vn;
            if (k == g.nz - 1) Un[2][P + 1] = Wu;
            pn[P] = (fc == FLUID || fc == GHOST) ? pc + ppc : NaN;
            if (fc == FLUID) {
                if (F32) {
                    const float gx = (d2f_int(ppe) - d2f_int(ppw)) * axf.rdcc[I];
                    const float gy = (d2f_int(ppn) - d2f_int(pps)) * ayf.rdcc[J];
                    const float gz = (d2f_int(ppu) - d2f_int(ppd)) * azf.rdcc[K];
                    const float dtf = (float)dt;
                    un[0][P] = o0 + f2d_int(e0 - dtf * gx);
                    un[1][P] = o1 + f2d_int(e1 - dtf * gy);
                    un[2][P] = o2 + f2d_int(e2 - dtf * gz);
                } else {
                    un[0][P] = o0 - dx.dtrdcc[I] * (ppe - ppw);
                    un[1][P] = o1 - dy.dtrdcc[J] * (ppn - pps);
                    un[2][P] = o2 - dz.dtrdcc[K] * (ppu - ppd);
                }
                if (!(bc.p_singular && i == 0 && j == 0 && k == 0)) {
                    const double div = (Ue - Uw) * ax.rd[I] + (Vn - Vs) * rdy + (Wu - Wd) * rdz;
                    mdiv = max(mdiv, __double_as_longlong(div) & 0x7fffffffffffffffLL);
                }
            } else if (fc == SOLID) {
                un[0][P] = un[1][P] = un[2][P] = NaN;
            }
        }
        Uw = Ue;
        fc = fe;
        ppw = ppc;
        ppc = ppe;
    }
    // Maximum over the block, then over the blocks (the last block to
    // finish reduces every block's value).  Integer maxima of the bits keep
    // the FP64 pipe free and NaN largest.
    const int t = ty * UN_TK + tx, lane = t & 31, warp = t >> 5;
    auto block_max = [&](long long x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_down_sync(0xffffffffu, x, o));
        __syncthreads();
        if (lane == 0) smem[warp] = x;
        __syncthreads();
        for (int w = 0; w < (UN_TK * UN_TJ) / 32; w++) x = max(x, smem[w]);
        return x;   // of the whole block in thread 0
    };
    long long m = block_max(mdiv);
    __shared__ bool last;
    if (t == 0) {
        partials[blockIdx.x] = __longlong_as_double(m);
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    m = 0;
    for (int q = t; q < (int)gridDim.x; q += UN_TK * UN_TJ) m = max(m, __double_as_longlong(__ldcg(partials + q)));
    m = block_max(m);
    if (t == 0) {
        *maxdiv_out = __longlong_as_double(m);
        *counter = 0;
    }
}

void launch_update_next_tiled(cudaStream_t s, const Grid &g, const Axis ax64[3], const DtAxis dta[3],
                              const AxisF axf[3], const BCSet &bc, const uint8_t *flag, const NextArgs *a64,
                              const Next32Args *a32, double dt, double *partials, unsigned int *counter,
                              double *maxdiv_out) {
    const Tiles t(g);
    const dim3 blk(UN_TK, UN_TJ);
    if (a32)
        k_update_next_tiled<true><<<t.nb, blk, 0, s>>>(g, ax64[0], ax64[1], ax64[2], dta[0], dta[1], dta[2], axf[0],
                                                      axf[1], axf[2], bc, flag, NextArgs{}, *a32, dt, t, partials,
                                                      counter, maxdiv_out);
    else
        k_update_next_tiled<false><<<t.nb, blk, 0, s>>>(g, ax64[0], ax64[1], ax64[2], dta[0], dta[1], dta[2], axf[0],
                                                       axf[1], axf[2], bc, flag, *a64, Next32Args{}, dt, t, partials,
                                                       counter, maxdiv_out);
    note_launches(1);
}

// ------------------------------------------------------------------------
// FP32 N read back as FP64 (field export of the mixed FP32 step).
// ------------------------------------------------------------------------
__global__ void k_widen_f32(const long long n, const float *__restrict__ x, double *__restrict__ y) {
    for (long long P = blockIdx.x * (long long)blockDim.x + threadIdx.x; P < n;
         P += (long long)gridDim.x * blockDim.x)
        y[P] = (double)x[P];
}

void launch_widen_f32(cudaStream_t s, long long n, const float *x, double *y) {
    k_widen_f32<<<K32_BLOCKS, 256, 0, s>>>(n, x, y);
    note_launches(1);
}

// u* = u^n + e (NaN in u^n, solid cells, counts as 0), for read-back.
__global__ void k_ustar_from_increment(const long long n, const double *__restrict__ u, const float *__restrict__ e,
                                       double *__restrict__ y) {
    for (long long P = blockIdx.x * (long long)blockDim.x + threadIdx.x; P < n;
         P += (long long)gridDim.x * blockDim.x) {
        const double v = u[P];
        y[P] = (v == v ? v : 0.0) + (double)e[P];
    }
}

void launch_ustar_from_increment(cudaStream_t s, long long n, const double *u, const float *e, double *y) {
    k_ustar_from_increment<<<K32_BLOCKS, 256, 0, s>>>(n, u, e, y);
    note_launches(1);
}

// ------------------------------------------------------------------------
// Self-test of the integer-pipe conversions against the hardware ones:
// x[q] for q < n is converted both ways; mismatches are counted (ties of
// the rounding, where d2f_int rounds away from zero and the hardware to
// even, and float subnormals are excluded by the caller's values).
// ------------------------------------------------------------------------
__global__ void k_conversion_check(const long long n, const double *__restrict__ x, unsigned long long *bad) {
    unsigned long long nb = 0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const double v = x[q];
        const float a = d2f_int(v), b = __double2float_rn(v);
        const bool same_f = __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
        const double c = f2d_int(b), d = (double)b;
        const bool same_d = __double_as_longlong(c) == __double_as_longlong(d) || (c != c && d != d);
        nb += (!same_f) + (!same_d);
    }
    atomicAdd(bad, nb);
}

int conversion_check(long long n, const double *x_host, unsigned long long *mismatches) {
    double *x = nullptr;
    unsigned long long *bad = nullptr;
    int rc = -1;
    if (cudaMalloc(&x, sizeof(double) * n) == cudaSuccess && cudaMalloc(&bad, sizeof *bad) == cudaSuccess &&
        cudaMemcpy(x, x_host, sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess &&
        cudaMemset(bad, 0, sizeof *bad) == cudaSuccess) {
        k_conversion_check<<<K32_BLOCKS, 256>>>(n, x, bad);
        if (cudaGetLastError() == cudaSuccess &&
            cudaMemcpy(mismatches, bad, sizeof *bad, cudaMemcpyDeviceToHost) == cudaSuccess)
            rc = 0;
    }
    cudaFree(x);
    cudaFree(bad);
    return rc;
}

}  // namespace ibm
