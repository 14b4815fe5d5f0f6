// Fast diagonalisation, FP32: the two ends of an application as one kernel
// each, for grids whose slices (z and the other densely transformed axis)
// fit one block.  Included by fastpoisson.cu.
//
// Both axes' transforms act within a slice, and a mirror-symmetric axis
// splits its modes by parity.  k_fp_front takes the padded residual to the
// modes of a slice (one block per slice and row parity): the source of every
// cell, the mirrored cells' sums and differences on both axes, the product
// with the z modes, and, from shared memory, with the row modes.  k_fp_rear
// goes back: a block expands the row modes into a set of rows and their
// mirror images, keeps those in shared memory, and expands the z modes into
// the padded array.  The axis matrices are loaded before the kernel waits for
// its predecessor.
//
// Bound by latency: two launches in place of five, each a chain of loads, a
// product, a barrier and a product.  Boxes 95x61x47, cold: 22.9 -> 17.3 us
// (gather, two forward transforms) and 12.3 -> 11.2 (two backward); the step
// with its 9 applications 1.40 -> 1.33 ms.
#pragma once

namespace ibm {

// For slices of at most 64 rows (32 where the rows' axis is not
// mirror-symmetric) by 64 columns.
constexpr int FPP_THREADS = 256, FPP_ROWS = 32, FPP_COLS = 64;
constexpr int FPP_PITCH = FPP_ROWS + 4;   // length of a shared-memory row along the slice's rows

struct FpPlane {
    int o;                       // the rows' axis: 1 (y, slices along x) or 0 (x, slices along y)
    int nr, nz;                  // rows, cells along z
    int fo, he, ho;              // rows: folded, even and odd modes
    int fz, ne, no, off, ld;     // z: the same, first odd column, row length
    const float *mz[2], *mr[2];  // matrices of z and of the rows, per parity
    int lz[2], lr[2];            // their row lengths
    long long sr, sb;            // compact strides: row modes, slices
    int s2, s3;                  // shared-memory offsets (floats) of the second and third region
};

// ---------------------------------------------------------------- front --
// 2 rows by 4 columns per thread (ty, tx 16 x 16), the whole slice in one
// tile.  Shared memory: G (column k of both parities, rows contiguous),
// replaced by Z (row, z mode); the z matrices (k, column); the row matrix
// (row, mode).
template <typename S>
__global__ void __launch_bounds__(FPP_THREADS, 2)
k_fp_front(const OpT<float> c, const S *__restrict__ r, float *__restrict__ out, const FpPlane p, const int body,
           const float *__restrict__ gscale, const int *gate) {
    constexpr int RT = 2, TR = FPP_ROWS, TC = FPP_COLS, PG = FPP_PITCH;
    using Row = FpVec<float, RT>;
    using Col = FpVec<float, 4>;
    extern __shared__ __align__(16) float sm[];
    float *G = sm, *FZ = sm + p.s2, *FR = sm + p.s3;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
    const int b = blockIdx.x, par = blockIdx.y, H = par ? p.ho : p.he;
    const float *mr = par ? p.mr[1] : p.mr[0];
    const int lr = par ? p.lr[1] : p.lr[0];
    for (int e = t; e < p.ne * (TC / 4); e += FPP_THREADS) {
        const int k = e / (TC / 4), q = e % (TC / 4) * 4, h = p.fz && q >= p.off, m = q - (h ? p.off : 0);
        Col v{};
        const int lz = h ? p.lz[1] : p.lz[0];
        if (m < lz && k < (h ? p.no : p.ne)) v = *reinterpret_cast<const Col *>((h ? p.mz[1] : p.mz[0]) + k * lz + m);
        *reinterpret_cast<Col *>(FZ + k * TC + q) = v;
    }
    for (int e = t; e < H * (TR / 4); e += FPP_THREADS) {
        const int q = e / (TR / 4), m = e % (TR / 4) * 4;
        Col v{};
        if (m < lr) v = *reinterpret_cast<const Col *>(mr + q * lr + m);
        *reinterpret_cast<Col *>(FR + q * TR + m) = v;
    }
    FP_GATE(gate);
    // Sources, folded on both axes.
    const Grid &g = c.g;
    const int ob = 1 - p.o, nb = p.o ? g.nx : g.ny;
    const int fb0 = p.o ? F_W : F_S, fb1 = p.o ? F_E : F_N, fr0 = p.o ? F_S : F_W, fr1 = p.o ? F_N : F_E;
    const long long sb = p.o ? g.sx : g.sy, sr = p.o ? g.sy : g.sx;
    const long long base = cidx(g, 0, 0, 0) + b * sb;
    const float ksb = c.ks[ob][b + 2];
    // The outer rows beside the slice's own edges: thread t takes row t's two
    // ends (t < 128) or the first and last row's cell t - 128, here, with the
    // gather's loads, and adds them when it is done.
    const bool ends = t < 128;
    const int et = ends ? t : t - 128, ea = ends ? 2 : p.o, en = ends ? p.nz : p.nr;
    const long long es = ends ? 1 : sr, er = ends ? sr : 1, ez = (ends ? p.nz - 1 : p.nr - 1) * es;
    const int em = (ends ? p.fo : p.fz) ? (ends ? p.nr : p.nz) - 1 - et : et;
    const bool edge = et < (ends ? H : p.ne), mirror = edge && em != et;
    const long long E0 = base + et * er, E1 = base + em * er;
    S eo[4];
    bool ef[4];
    auto counts = [&](long long P) { return !(body && c.flag[P] != FLUID) && !(c.p_singular && P == c.pinned); };
    if (edge) {
        eo[0] = r[E0 - es], eo[1] = r[E0 + ez + es];
        ef[0] = counts(E0), ef[1] = counts(E0 + ez);
        if (mirror) {
            eo[2] = r[E1 - es], eo[3] = r[E1 + ez + es];
            ef[2] = counts(E1), ef[3] = counts(E1 + ez);
        }
    }
    // pass 0: the cells' own residuals; 1 and 2: those of the outer rows
    // beside the first and the last slice.
    for (int pass = 0; pass < 3; pass++) {
        if ((pass == 1 && b > 0) || (pass == 2 && b < nb - 1)) continue;
        const long long from = pass == 0 ? 0 : pass == 1 ? -sb : sb;
        const float ko = pass == 1 ? c.km[ob][2] : pass == 2 ? c.kp[ob][b + 2] : 0.0f;
        auto source = [&](long long P, S x, uint8_t fl, float ks) {
            float v = fp_value<float, S>(x);
            if (pass > 0) {
                v = fl == FLUID ? ko * fp_outer(c.bc[pass == 1 ? fb0 : fb1], v) : 0.0f;
            } else {
                v *= ks;
                if (fl == GHOST) v *= gscale[c.gid[P]];
                else if (fl != FLUID) v = 0;
            }
            return c.p_singular && P == c.pinned ? 0.0f : v;
        };
        for (int k = lane; k < p.ne; k += 32) {
            const int kz = p.fz ? p.nz - 1 - k : k;
            const float s1 = c.ks[2][k + 2], s2 = c.ks[2][kz + 2];
            for (int q0 = warp; q0 < H; q0 += 16) {
                S x[2][4];
                uint8_t fl[2][4];
                float kr[2][2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int q = min(q0 + 8 * u, H - 1), qm = p.fo ? p.nr - 1 - q : q;
                    const long long P = base + q * sr, M = base + qm * sr;
                    x[u][0] = r[P + from + k];
                    if (p.fz) x[u][1] = r[P + from + kz];
                    if (p.fo) x[u][2] = r[M + from + k];
                    if (p.fo && p.fz) x[u][3] = r[M + from + kz];
                    kr[u][0] = c.ks[p.o][q + 2];
                    kr[u][1] = c.ks[p.o][qm + 2];
#pragma unroll
                    for (int w = 0; w < 4; w++) fl[u][w] = FLUID;
                    if (body) {
                        fl[u][0] = c.flag[P + k];
                        if (p.fz) fl[u][1] = c.flag[P + kz];
                        if (p.fo) fl[u][2] = c.flag[M + k];
                        if (p.fo && p.fz) fl[u][3] = c.flag[M + kz];
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int q = q0 + 8 * u, qm = p.fo ? p.nr - 1 - q : q;
                    if (q >= H) break;
                    const long long P = base + q * sr, M = base + qm * sr;
                    const float k0 = ksb + kr[u][0], k1 = ksb + kr[u][1];
                    float v = source(P + k, x[u][0], fl[u][0], k0 + s1), w = 0;
                    if (kz != k) w = source(P + kz, x[u][1], fl[u][1], k0 + s2);
                    if (qm != q) {
                        const float a = source(M + k, x[u][2], fl[u][2], k1 + s1);
                        float d = 0;
                        if (kz != k) d = source(M + kz, x[u][3], fl[u][3], k1 + s2);
                        v += par ? -a : a;
                        w += par ? -d : d;
                    }
                    float *ge = G + k * PG + q, *go = G + (p.off + k) * PG + q;
                    *ge = (pass ? *ge : 0.0f) + (v + w);
                    if (p.fz) *go = (pass ? *go : 0.0f) + (kz != k ? v - w : 0.0f);
                }
            }
        }
    }
    // First and last value beside the edge: of cell (row) et and of its mirror image.
    auto outer = [&](int w) {
        const int f = w & 1 ? (ends ? F_U : fr1) : (ends ? F_D : fr0);
        return ef[w] ? (w & 1 ? c.kp[ea][en + 1] : c.km[ea][2]) * fp_outer(c.bc[f], fp_value<float, S>(eo[w])) : 0.0f;
    };
    float a = 0, d = 0, am = 0, dm = 0;
    if (edge) a = outer(0), d = outer(1);
    if (mirror) am = outer(2), dm = outer(3);
    __syncthreads();
    if (edge && ends) {
        a += par ? -am : am;
        d += par ? -dm : dm;
        if (p.fz) {
            G[et] += a + d;
            G[p.off * PG + et] += a - d;
        } else {
            G[et] += a;
            G[(p.nz - 1) * PG + et] += d;
        }
    }
    __syncthreads();
    if (edge && !ends) {
        float *e = G + et * PG, *o = G + (p.off + et) * PG;
        if (p.fo) {
            a += par ? -d : d;
            am += par ? -dm : dm;
            e[0] += a + am;
            if (mirror) o[0] += a - am;
        } else {
            e[0] += a + am;
            e[p.nr - 1] += d + dm;
            if (mirror) {
                o[0] += a - am;
                o[p.nr - 1] += d - dm;
            }
        }
    }
    __syncthreads();
    float acc[RT][4];
    auto step = [&](const float *rows, const float *cols) {
        const Row x = *reinterpret_cast<const Row *>(rows + ty * RT);
        const Col y = *reinterpret_cast<const Col *>(cols + tx * 4);
#pragma unroll
        for (int i = 0; i < RT; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] += x.v[i] * y.v[j];
    };
    auto store = [&](float *row, int i) {
        Col o;
#pragma unroll
        for (int j = 0; j < 4; j++) o.v[j] = acc[i][j];
        *reinterpret_cast<Col *>(row + tx * 4) = o;
    };
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0;
    // z: Z(row, mode) = sum over k of G(k, row) FZ(k, mode).
    const bool odd = p.fz && tx * 4 >= p.off;
    const int kn = odd ? p.no : p.ne;
    const float *gk = G + (odd ? p.off : 0) * PG;
#pragma unroll 8
    for (int k = 0; k < kn; k++) step(gk + k * PG, FZ + k * TC);
    __syncthreads();
    float *Z = G;
#pragma unroll
    for (int i = 0; i < RT; i++)
        if (ty * RT + i < H) store(Z + (ty * RT + i) * TC, i);
    __syncthreads();
    // Rows: out(mode, column) = sum over rows q of FR(q, mode) Z(q, column).
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0;
#pragma unroll 8
    for (int q = 0; q < H; q++) step(FR + q * TR, Z + q * TC);
    if (tx * 4 >= p.ld) return;
#pragma unroll
    for (int i = 0; i < RT; i++)
        if (ty * RT + i < H) store(out + b * p.sb + (par * p.he + ty * RT + i) * p.sr, i);
}

// ----------------------------------------------------------------- rear --
// A block takes 16 rows of a slice's first half and their mirror images.
// Shared memory: X (row mode, column), replaced by U (column, row); the row
// matrices (mode, row); the z matrices (mode, cell), even modes first.  2 x 2
// values of both parities per thread: of 8 x 32 threads in the first product,
// of 16 x 16 in the second.
constexpr int FPP_HALF = 16;

template <typename S>
__global__ void __launch_bounds__(FPP_THREADS, 3)
k_fp_rear(const Grid g, const S *__restrict__ r, const float *__restrict__ in, float *__restrict__ z, const FpPlane p,
          const float *__restrict__ v0, const int singular, const long long pinned, const int *gate) {
    constexpr int RT = 2, TH = FPP_HALF, TC = FPP_COLS, PU = FPP_PITCH, TK = FPP_ROWS;
    using Vec = FpVec<float, RT>;
    using Col = FpVec<float, 4>;
    static_assert(2 * TH + 4 == PU && 16 * RT == TK && 32 * RT == TC, "tiles");
    extern __shared__ __align__(16) float sm[];
    __shared__ float red[FPP_THREADS / 32];
    float *X = sm, *BR = sm + p.s2, *BZ = sm + p.s3;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int b = blockIdx.x, r0 = blockIdx.y * TH;
    const int nkz = (p.ne + TK - 1) / TK * TK;   // cells of the z matrices' rows, padded to the tile
    for (int e = t; e < (p.he + p.ho) * TH; e += FPP_THREADS) {
        const int m = e / TH, q = r0 + e % TH, h = m >= p.he, mm = m - (h ? p.he : 0);
        BR[e] = q < (h ? p.ho : p.he) ? (h ? p.mr[1] : p.mr[0])[mm * (h ? p.lr[1] : p.lr[0]) + q] : 0.0f;
    }
    for (int e = t; e < (p.ne + p.no) * nkz; e += FPP_THREADS) {
        const int m = e / nkz, k = e % nkz, h = m >= p.ne, mm = m - (h ? p.ne : 0);
        const int lz = h ? p.lz[1] : p.lz[0];
        BZ[e] = k < lz ? (h ? p.mz[1] : p.mz[0])[mm * lz + k] : 0.0f;
    }
    FP_GATE(gate);
    // Rows: E and O.
    const int wx = lane & 7, wy = lane >> 3;
    const int ax = (warp & 3) * 8 + wx, ay = (warp >> 2) * 4 + wy;
    for (int e = t; e < (p.he + p.ho) * (TC / 4); e += FPP_THREADS) {
        const int m = e / (TC / 4), q = e % (TC / 4) * 4;
        if (q < p.ld)
            *reinterpret_cast<Col *>(X + m * TC + q) = *reinterpret_cast<const Col *>(in + b * p.sb + m * p.sr + q);
    }
    float shift = 0;
    if (singular) {
        // z(0,0,0) of the unshifted solution, by every block for itself.
        float s = 0;
        for (int m = warp; m < p.he + p.ho; m += FPP_THREADS / 32) {
            const int h = m >= p.he;
            float l = 0;
            for (int q = lane; q < p.ld; q += 32) l += in[m * p.sr + q] * v0[q];
            s += (h ? p.mr[1] : p.mr[0])[(m - (h ? p.he : 0)) * (h ? p.lr[1] : p.lr[0])] * l;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[warp] = s;
    }
    __syncthreads();
    if (singular) {
        float s = 0;
#pragma unroll
        for (int w = 0; w < FPP_THREADS / 32; w++) s += red[w];
        shift = fp_value<float, S>(r[pinned]) - s;
    }
    float ea[RT][RT], oa[RT][RT];
#pragma unroll
    for (int x = 0; x < RT; x++)
#pragma unroll
        for (int y = 0; y < RT; y++) ea[x][y] = oa[x][y] = 0;
    auto r_step = [&](float (&acc)[RT][RT], const float *bm, const float *xm) {
        const Vec a = *reinterpret_cast<const Vec *>(bm + ay * RT);
        const Vec q = *reinterpret_cast<const Vec *>(xm + ax * RT);
#pragma unroll
        for (int x = 0; x < RT; x++)
#pragma unroll
            for (int y = 0; y < RT; y++) acc[x][y] += a.v[x] * q.v[y];
    };
#pragma unroll 4
    for (int m = 0; m < p.he; m++) r_step(ea, BR + m * TH, X + m * TC);
#pragma unroll 4
    for (int m = p.he; m < p.he + p.ho; m++) r_step(oa, BR + m * TH, X + m * TC);
    __syncthreads();
    float *U = X;
#pragma unroll
    for (int y = 0; y < RT; y++) {
        const int q = ax * RT + y;
        if (q >= p.ld) break;
        Vec e, o;
#pragma unroll
        for (int x = 0; x < RT; x++) {
            e.v[x] = ea[x][y] + oa[x][y];
            o.v[x] = ea[x][y] - oa[x][y];
        }
        *reinterpret_cast<Vec *>(U + q * PU + ay * RT) = e;
        *reinterpret_cast<Vec *>(U + q * PU + TH + ay * RT) = o;
    }
    __syncthreads();
    // z, into the padded array.
    const int tx = (warp & 1) * 8 + wx, ty = (warp >> 1) * 4 + wy;
    for (int k0 = 0; k0 < p.ne; k0 += TK) {
#pragma unroll
        for (int x = 0; x < RT; x++)
#pragma unroll
            for (int y = 0; y < RT; y++) ea[x][y] = oa[x][y] = 0;
        auto z_step = [&](float (&acc)[RT][RT], const float *um, const float *bm) {
            const Vec a = *reinterpret_cast<const Vec *>(um + ty * RT);
            const Vec q = *reinterpret_cast<const Vec *>(bm + k0 + tx * RT);
#pragma unroll
            for (int x = 0; x < RT; x++)
#pragma unroll
                for (int y = 0; y < RT; y++) acc[x][y] += a.v[x] * q.v[y];
        };
#pragma unroll 2
        for (int m = 0; m < p.no; m++) {
            z_step(ea, U + m * PU, BZ + m * nkz);
            z_step(oa, U + (p.off + m) * PU, BZ + (p.ne + m) * nkz);
        }
#pragma unroll 4
        for (int m = p.no; m < p.ne; m++) z_step(ea, U + m * PU, BZ + m * nkz);
#pragma unroll
        for (int x = 0; x < RT; x++) {
            const int rho = ty * RT + x, up = rho >= TH, q = r0 + rho - (up ? TH : 0);
            if (q >= (up ? p.ho : p.he)) continue;
            const int row = up ? p.nr - 1 - q : q;
            float *line = z + (p.o ? cidx(g, b, row, 0) : cidx(g, row, b, 0));
#pragma unroll
            for (int y = 0; y < RT; y++) {
                const int k = k0 + tx * RT + y;
                if (k >= p.ne) break;
                const float e = ea[x][y] + shift, o = oa[x][y];
                line[k] = e + o;
                if (p.fz && k < p.no) line[p.nz - 1 - k] = e - o;
            }
        }
    }
}

}  // namespace ibm
