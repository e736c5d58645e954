// FP64 species and heat transport solves, compute_C (tse.py:783-916) and
// compute_T (tse.py:919-1081), plus the dispersion coefficients
// (dispersivity, tse.py:460-644).
//
// Within a solve the upwind/diffusive/dispersive neighbour coefficients, the
// explicit (1-omega) part, R*Xn, the source and the IMBLFLO term are fixed,
// so one assembly pass computes them in the reference's operation order and
// the persistent red-black loop evaluates
//   X = (1-SOR) X + SOR (omega (Mnew+Nnew+Onew+Pnew+Qnew+Rnew)
//                        + (1-omega) (...) + R Xn + W - E) / (R - omega M)
// (tse.py:870-875, 1038-1043) term by term.  Compiled with --fmad=false.
#include <algorithm>
#include <cmath>

#include "tse_dc.cuh"
#include "tse_forms.cuh"
#include "tse_rbsolve.cuh"
#include "tse_rbsolve_res.cuh"
#include "tse_rbsolve_tma.cuh"

namespace tse {

// dispersivity (tse.py:460-644); D = {xl, yl, zl, xr, yr, zr}
__device__ void dispersivity_dev(const double* qx, const double* qy, const double* qz,
                                 const double* l_l, const double* l_t, const double* B, int i,
                                 int j, int k, int nx, int ny, int nz, double* D) {
    const long long sx = (long long)ny * nz, sy = nz;
    const long long c = ((long long)i * ny + j) * nz + k;
#define IX3(ii, jj, kk) (c + (long long)((ii) - i) * sx + (long long)((jj) - j) * sy + ((kk) - k))
    double qxl = 0, qyl = 0, qzl = 0, qxr = 0, qyr = 0, qzr = 0;
    double qxyl = 0, qxzl = 0, qyxl = 0, qyzl = 0, qzxl = 0, qzyl = 0;
    double qxyr = 0, qxzr = 0, qyxr = 0, qyzr = 0, qzxr = 0, qzyr = 0;
    // cnt: 1/2 or 1/4 -- dividing by 2 or 4 and multiplying by 0.5 or 0.25
    // round the same exact quotient, so the results are identical
    double q1, q2, q3, q4, cnt;
    if (i != 0) {
        qxl = qx[IX3(i - 1, j, k)];
        q1 = qy[IX3(i - 1, j, k)]; q2 = qy[c]; q3 = q4 = 0; cnt = 0.5;
        if (j != 0) { q3 = qy[IX3(i, j - 1, k)]; q4 = qy[IX3(i - 1, j - 1, k)]; cnt = 0.25; }
        if (!(B[IX3(i - 1, j, k)] != 0)) qxyl = (q1 + q2 + q3 + q4) * cnt;
        q1 = qz[IX3(i - 1, j, k)]; q2 = qz[c]; q3 = q4 = 0; cnt = 0.5;
        if (k != 0) { q3 = qz[IX3(i, j, k - 1)]; q4 = qz[IX3(i - 1, j, k - 1)]; cnt = 0.25; }
        if (!(B[IX3(i - 1, j, k)] != 0)) qxzl = (q1 + q2 + q3 + q4) * cnt;
    }
    if (i != nx - 1) {
        qxr = qx[c];
        q1 = qy[c]; q2 = qy[IX3(i + 1, j, k)]; q3 = q4 = 0; cnt = 0.5;
        if (j != 0) { q3 = qy[IX3(i + 1, j - 1, k)]; q4 = qy[IX3(i, j - 1, k)]; cnt = 0.25; }
        if (!(B[IX3(i + 1, j, k)] != 0)) qxyr = (q1 + q2 + q3 + q4) * cnt;
        q1 = qz[c]; q2 = qz[IX3(i + 1, j, k)]; q3 = q4 = 0; cnt = 0.5;
        if (k != 0) { q3 = qz[IX3(i + 1, j, k - 1)]; q4 = qz[IX3(i, j, k - 1)]; cnt = 0.25; }
        if (!(B[IX3(i + 1, j, k)] != 0)) qxzr = (q1 + q2 + q3 + q4) * cnt;
    }
    if (j != 0) {
        qyl = qy[IX3(i, j - 1, k)];
        q1 = qx[c]; q2 = qx[IX3(i, j - 1, k)]; q3 = q4 = 0; cnt = 0.5;
        if (i != 0) { q3 = qx[IX3(i - 1, j - 1, k)]; q4 = qx[IX3(i - 1, j, k)]; cnt = 0.25; }
        if (!(B[IX3(i, j - 1, k)] != 0)) qyxl = (q1 + q2 + q3 + q4) * cnt;
        q1 = qz[IX3(i, j - 1, k)]; q2 = qz[c]; q3 = q4 = 0; cnt = 0.5;
        if (k != 0) { q3 = qz[IX3(i, j, k - 1)]; q4 = qz[IX3(i, j - 1, k - 1)]; cnt = 0.25; }
        if (!(B[IX3(i, j - 1, k)] != 0)) qyzl = (q1 + q2 + q3 + q4) * cnt;
    }
    if (j != ny - 1) {
        qyr = qy[c];
        q1 = qx[IX3(i, j + 1, k)]; q2 = qx[c]; q3 = q4 = 0; cnt = 0.5;
        if (i != 0) { q3 = qx[IX3(i - 1, j, k)]; q4 = qx[IX3(i - 1, j + 1, k)]; cnt = 0.25; }
        if (!(B[IX3(i, j + 1, k)] != 0)) qyxr = (q1 + q2 + q3 + q4) * cnt;
        q1 = qz[c]; q2 = qz[IX3(i, j + 1, k)]; q3 = q4 = 0; cnt = 0.5;
        if (k != 0) { q3 = qz[IX3(i, j + 1, k - 1)]; q4 = qz[IX3(i, j, k - 1)]; cnt = 0.25; }
        if (!(B[IX3(i, j + 1, k)] != 0)) qyzr = (q1 + q2 + q3 + q4) * cnt;
    }
    if (k != 0) {
        qzl = qz[IX3(i, j, k - 1)];
        q1 = qx[c]; q2 = qx[IX3(i, j, k - 1)]; q3 = q4 = 0; cnt = 0.5;
        if (i != 0) { q3 = qx[IX3(i - 1, j, k - 1)]; q4 = qx[IX3(i - 1, j, k)]; cnt = 0.25; }
        if (!(B[IX3(i, j, k - 1)] != 0)) qzxl = (q1 + q2 + q3 + q4) * cnt;
        q1 = qy[c]; q2 = qy[IX3(i, j, k - 1)]; q3 = q4 = 0; cnt = 0.5;
        if (j != 0) { q3 = qy[IX3(i, j - 1, k - 1)]; q4 = qy[IX3(i, j - 1, k)]; cnt = 0.25; }
        if (!(B[IX3(i, j, k - 1)] != 0)) qzyl = (q1 + q2 + q3 + q4) * cnt;
    }
    if (k != nz - 1) {
        qzr = qz[c];
        q1 = qx[IX3(i, j, k + 1)]; q2 = qx[c]; q3 = q4 = 0; cnt = 0.5;
        if (i != 0) { q3 = qx[IX3(i - 1, j, k)]; q4 = qx[IX3(i - 1, j, k + 1)]; cnt = 0.25; }
        if (!(B[IX3(i, j, k + 1)] != 0)) qzxr = (q1 + q2 + q3 + q4) * cnt;
        q1 = qy[IX3(i, j, k + 1)]; q2 = qy[c]; q3 = q4 = 0; cnt = 0.5;
        if (j != 0) { q3 = qy[IX3(i, j - 1, k)]; q4 = qy[IX3(i, j - 1, k + 1)]; cnt = 0.25; }
        if (!(B[IX3(i, j, k + 1)] != 0)) qzyr = (q1 + q2 + q3 + q4) * cnt;
    }
#undef IX3
    const double ll = l_l[c], lt = l_t[c];
    D[0] = ll * fabs(qxl) + lt * (fabs(qxyl) + fabs(qxzl));
    D[1] = ll * fabs(qyl) + lt * (fabs(qyxl) + fabs(qyzl));
    D[2] = ll * fabs(qzl) + lt * (fabs(qzxl) + fabs(qzyl));
    D[3] = ll * fabs(qxr) + lt * (fabs(qxyr) + fabs(qxzr));
    D[4] = ll * fabs(qyr) + lt * (fabs(qyxr) + fabs(qyzr));
    D[5] = ll * fabs(qzr) + lt * (fabs(qzxr) + fabs(qzyr));
}

struct CellIdx {
    int i, j, k, col;
    long long m, c;
    bool pad;
};

__device__ __forceinline__ bool decode_padded(long long t, const Layout& L, CellIdx& x) {
    const long long total = (long long)L.nx * L.ny * L.nzp;
    if (t >= total) return false;
    long long row;
    grid_coords(t, L.ny, L.nzp, x.i, x.j, x.k, row);
    x.m = t >> 1;
    x.col = (x.i + x.j + x.k) & 1;
    x.pad = x.k >= L.nz;
    x.c = row * L.nz + x.k;
    return true;
}

// The assemblies below keep the reference's operations and their order for
// every value they produce, and drop only work whose result is already
// known:
//  - each face's means are formed once, by the face pass, rather than by
//    both cells that share the face (see species_face);
//  - min0(q) / d and max0(q) / d: one of the two is 0 / d, so q / d is formed
//    once and 0 / d (+0 for d > 0) is selected for the other.
// harm2w is harm2(H1, H2, d1, d2) = (d1 + d2) / (d1 / H1 + d2 / H2) with the
// quotients w1 = d1 / H1, w2 = d2 / H2 passed in.
__device__ __forceinline__ double harm2w(double H1, double H2, double d1, double d2, double w1,
                                         double w2) {
    if (H1 != 0.0 && H2 != 0.0) return (d1 + d2) / (w1 + w2);
    return 0.0;
}
__device__ __forceinline__ double zero_over(double d) { return d > 0.0 ? 0.0 : 0.0 / d; }

// One axis of a transport assembly: the + face (toward the next cell along
// the axis) and the - face.  dP/dM: diffusive (and dispersive) coefficients,
// minP/maxP: min0/max0 of the cell's own face flux (scaled), maxM/minM: the
// same for the - neighbour's face flux, coP/coM: upwinded neighbour
// coefficients, oldP/oldM: coP * Xn(+ neighbour), coM * Xn(- neighbour).
struct AxisTerms {
    double dP, dM, minP, maxP, maxM, minM, coP, coM, oldP, oldM;
};

// The means both cells of a face form alike, computed once a face by a pass
// before the assembly (faces_kernel): for a species harm2(D) * amean2(phi),
// the face's value of A (tse.py:811-861); for heat the conductivity mix
// (1 - por) lr + por lf and the mean of rho_f times that of cp_f
// (tse.py:952-1027).  The cell on the + side forms them with the operands
// swapped -- (d1 + d2) / (d1/H1 + d2/H2) and (X1 d1 + X2 d2) / (d1 + d2) --
// and IEEE addition and multiplication commute, so the values are the ones
// each cell would form itself, bit for bit.  Stored per axis for the face
// toward the + neighbour (0 where there is none).
__device__ __forceinline__ void species_face(const double* __restrict__ Df, const double* __restrict__ phi,
                                             const double* __restrict__ d, long long c, long long st,
                                             int ii, bool hp, double phic, double* __restrict__ out) {
    double v = 0.0;
    if (hp) {
        const long long o = c + st;
        const double dd = d[ii], dp = d[ii + 1];
        const double Dc = Df[c], Dp = Df[o];
        v = harm2w(Dp, Dc, dp, dd, dp / Dp, dd / Dc) * amean2(phi[o], phic, dp, dd);
    }
    out[c] = v;
}

__device__ __forceinline__ void heat_face(const TseHeatArgs& a, const double* __restrict__ d, long long c,
                                          long long st, int ii, bool hp, double* __restrict__ k1_out,
                                          double* __restrict__ rc_out) {
    double k1 = 0.0, rc = 0.0;
    if (hp) {
        const long long o = c + st;
        const double dd = d[ii], dp = d[ii + 1];
        const double phic = a.phi[c], lfc = a.l_f[c], lrc = a.l_r[c], cpc = a.cp_f[c], rhc = a.rho_f[c];
        const double php = a.phi[o], lfp = a.l_f[o], lrp = a.l_r[o], cpp = a.cp_f[o], rhp = a.rho_f[o];
        const double por = amean2(phic, php, dd, dp);
        const double lf = harm2w(lfc, lfp, dd, dp, dd / lfc, dp / lfp);
        const double lr = harm2w(lrc, lrp, dd, dp, dd / lrc, dp / lrp);
        const double cpf = harm2w(cpc, cpp, dd, dp, dd / cpc, dp / cpp);
        rc = harm2w(rhc, rhp, dd, dp, dd / rhc, dp / rhp) * cpf;
        k1 = (1 - por) * lr + por * lf;
    }
    k1_out[c] = k1;
    rc_out[c] = rc;
}

// compute_C, one axis (tse.py:811-861): x -> (A, B, N, H, M, G), y -> (C, D,
// P, J, O, I), z -> (E, F, R, L, Q, K); Pf: this axis's face values
__device__ __forceinline__ AxisTerms species_axis(const double* __restrict__ Pf,
                                                  const double* __restrict__ Xn,
                                                  const double* __restrict__ q,
                                                  const double* __restrict__ d, long long c,
                                                  long long st, int ii, bool hp, bool hm,
                                                  double DdP, double DdM) {
    AxisTerms r = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const long long op = hp ? c + st : c, om = hm ? c - st : c;
    const double dd = d[ii], dp = d[hp ? ii + 1 : ii], dm = d[hm ? ii - 1 : ii];
    const double xp = Xn[op], xm = Xn[om];
    const double qc = q[c], qm = q[om];
    const double fp = Pf[c], fm = Pf[om];
    const double z = zero_over(dd);
    if (hp) {
        const double dd2 = (0.5 * (dp + dd)) * dd;
        r.dP = (fp + DdP) / dd2;
        const double qd = qc / dd;
        r.minP = (0.0 < qc) ? z : qd;
        r.maxP = (0.0 > qc) ? z : qd;
        r.coP = r.dP - r.minP;
        r.oldP = r.coP * xp;
    }
    if (hm) {
        const double dd2 = (0.5 * (dm + dd)) * dd;
        r.dM = (fm + DdM) / dd2;
        const double qd = qm / dd;
        r.maxM = (0.0 > qm) ? z : qd;
        r.minM = (0.0 < qm) ? z : qd;
        r.coM = r.dM + r.maxM;
        r.oldM = r.coM * xm;
    }
    return r;
}

// compute_T, one axis (tse.py:952-1027); K1, RC: this axis's face values
// (conductivity mix, rho_f cp_f mean)
__device__ __forceinline__ AxisTerms heat_axis(const double* __restrict__ K1, const double* __restrict__ RC,
                                               const double* __restrict__ Xn,
                                               const double* __restrict__ q,
                                               const double* __restrict__ d, long long c,
                                               long long st, int ii, bool hp, bool hm,
                                               double DdP, double DdM) {
    AxisTerms r = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const long long op = hp ? c + st : c, om = hm ? c - st : c;
    const double dd = d[ii], dp = d[hp ? ii + 1 : ii], dm = d[hm ? ii - 1 : ii];
    const double qc = q[c], qm = q[om];
    if (hp) {
        const double dd2 = (0.5 * (dp + dd)) * dd;
        const double rhocpf = RC[c];
        r.dP = (K1[c] + DdP * rhocpf) / dd2;
        const double S = rhocpf / dd;
        r.minP = min0(qc) * S;
        r.maxP = max0(qc) * S;
        r.coP = r.dP - r.minP;
        r.oldP = r.coP * Xn[op];
    }
    if (hm) {
        const double dd2 = (0.5 * (dm + dd)) * dd;
        const double rhocpf = RC[om];
        r.dM = (K1[om] + DdM * rhocpf) / dd2;
        const double S = rhocpf / dd;
        r.maxM = max0(qm) * S;
        r.minM = min0(qm) * S;
        r.coM = r.dM + r.maxM;
        r.oldM = r.coM * Xn[om];
    }
    return r;
}

// The per-cell terms of a transport solve: the six neighbour coefficients
// (x+, x-, y+, y-, z+, z-), M, (1-omega)-part Mo, R and its numerator, source
// and IMBLFLO term.
struct TransportTerms {
    double co[6];
    double Mo, Xn, Rnum, R, M, W, EX;
    bool active;
};

__device__ __forceinline__ void combine_axes(const AxisTerms& X, const AxisTerms& Y,
                                             const AxisTerms& Z, double Xn, TransportTerms& T) {
    T.co[0] = X.coP;
    T.co[1] = X.coM;
    T.co[2] = Y.coP;
    T.co[3] = Y.coM;
    T.co[4] = Z.coP;
    T.co[5] = Z.coM;
    // M = -A - B - C - D - E - F + G - H + I - J + K - L (tse.py:863, 1029)
    T.M = -X.dP - X.dM - Y.dP - Y.dM - Z.dP - Z.dM + X.minM - X.maxP + Y.minM - Y.maxP + Z.minM -
          Z.maxP;
    T.Xn = Xn;
    T.Mo = Xn * T.M + X.oldP + X.oldM + Y.oldP + Y.oldM + Z.oldP + Z.oldM;
}

// coefficient part of compute_C.solve (tse.py:795-868)
__device__ __forceinline__ void species_terms(const TseGrid& g, const TseSpeciesArgs& a,
                                              const CellIdx& x, const Layout& L,
                                              const double* __restrict__ faces, TransportTerms& T) {
    const int nx = L.nx, ny = L.ny, nz = L.nz, i = x.i, j = x.j, k = x.k;
    const long long c = x.c;
    double Dd[6] = {0, 0, 0, 0, 0, 0};
    if (a.l_l[c] != 0 || a.l_t[c] != 0)
        dispersivity_dev(a.qx, a.qy, a.qz, a.l_l, a.l_t, a.BC, i, j, k, nx, ny, nz, Dd);
    const long long n = (long long)nx * ny * nz;
    const AxisTerms X = species_axis(faces, a.C, a.qx, g.dx, c, (long long)ny * nz, i, i != nx - 1,
                                     i != 0, Dd[3], Dd[0]);
    const AxisTerms Y = species_axis(faces + n, a.C, a.qy, g.dy, c, nz, j, j != ny - 1, j != 0,
                                     Dd[4], Dd[1]);
    const AxisTerms Z = species_axis(faces + 2 * n, a.C, a.qz, g.dz, c, 1, k, k != nz - 1, k != 0,
                                     Dd[5], Dd[2]);
    const double phic = a.phi[c];
    const double Xn = a.C[c];
    combine_axes(X, Y, Z, Xn, T);
    T.Rnum = a.RC[c] * phic;
    T.R = T.Rnum / a.dt;
    T.EX = a.imblflo ? Xn / a.rho_f[c] * a.e[c] : 0.0;
    T.W = a.WC[c];
    T.active = !(a.BC[c] != 0.0);
}

// coefficient part of compute_T.solve (tse.py:930-1036)
__device__ __forceinline__ void heat_terms(const TseGrid& g, const TseHeatArgs& a, const CellIdx& x,
                                           const Layout& L, const double* __restrict__ faces,
                                           TransportTerms& T) {
    const int nx = L.nx, ny = L.ny, nz = L.nz, i = x.i, j = x.j, k = x.k;
    const long long c = x.c;
    double Dd[6] = {0, 0, 0, 0, 0, 0};
    if (a.l_l[c] != 0 || a.l_t[c] != 0)
        dispersivity_dev(a.qx, a.qy, a.qz, a.l_l, a.l_t, a.BT, i, j, k, nx, ny, nz, Dd);
    const long long n = (long long)nx * ny * nz;
    const AxisTerms X = heat_axis(faces, faces + 3 * n, a.T, a.qx, g.dx, c, (long long)ny * nz, i,
                                  i != nx - 1, i != 0, Dd[3], Dd[0]);
    const AxisTerms Y = heat_axis(faces + n, faces + 4 * n, a.T, a.qy, g.dy, c, nz, j, j != ny - 1,
                                  j != 0, Dd[4], Dd[1]);
    const AxisTerms Z = heat_axis(faces + 2 * n, faces + 5 * n, a.T, a.qz, g.dz, c, 1, k, k != nz - 1,
                                  k != 0, Dd[5], Dd[2]);
    const double Xn = a.T[c];
    combine_axes(X, Y, Z, Xn, T);
    const double por_ = a.phi[c];
    T.Rnum = por_ * a.rho_f[c] * a.cp_f[c] + (1 - por_) * a.rho_r[c] * a.cp_r[c];
    T.R = T.Rnum / a.dt;
    T.EX = a.imblflo ? a.cp_f[c] * Xn * a.e[c] : 0.0;
    T.W = a.WT[c];
    T.active = !(a.BT[c] != 0.0);
}

// The exact form's per-cell arrays (TransportForm) and the flag byte.
__device__ __forceinline__ void store_terms(const TransportForm& F, uint8_t* msk, const CellIdx& x,
                                            const TransportTerms& T, int nx, int ny, int nz) {
    double* b = F.arr[x.col];
    const long long N = F.Ncal, m = x.m;
    const double omega = F.omega;
    for (int q = 0; q < 6; ++q) b[q * N + m] = T.co[q];
    // the (1-omega) part and the IMBLFLO term are read only where the form
    // uses them (TransportForm::useY / useEX)
    if (F.useY) b[TA_Y * N + m] = (1 - omega) * T.Mo;
    b[TA_RXN * N + m] = T.R * T.Xn;
    b[TA_W * N + m] = T.W;
    if (F.useEX) b[TA_EX * N + m] = T.EX;
    b[TA_DEN * N + m] = T.R - omega * T.M;
    b[TA_RNUM * N + m] = T.Rnum;
    b[TA_M * N + m] = T.M;
    b[TA_XN * N + m] = T.Xn;
    b[TA_X * N + m] = T.Xn;
    uint8_t f = neighbour_flags(x.i, x.j, x.k, nx, ny, nz);
    if (T.active) f |= F_ACTIVE;
    msk[m] = f;
}

__device__ __forceinline__ void store_padding(const TransportForm& F, uint8_t* msk, const CellIdx& x) {
    double* b = F.arr[x.col];
    for (int q = 0; q < TA_COUNT; ++q) b[q * F.Ncal + x.m] = 0.0;
    msk[x.m] = 0;
}

struct SpeciesKind {
    using Args = TseSpeciesArgs;
    static __device__ __forceinline__ void terms(const TseGrid& g, const Args& a, const CellIdx& x,
                                                 const Layout& L, const double* faces,
                                                 TransportTerms& T) {
        species_terms(g, a, x, L, faces, T);
    }
    // the face pass, one cell (natural order)
    static __device__ __forceinline__ void faces(const TseGrid& g, const Args& a, const Layout& L,
                                                 long long c, int i, int j, int k, double* out) {
        const long long n = (long long)L.nx * L.ny * L.nz;
        const double phic = a.phi[c];
        species_face(a.D_fx, a.phi, g.dx, c, (long long)L.ny * L.nz, i, i != L.nx - 1, phic, out);
        species_face(a.D_fy, a.phi, g.dy, c, L.nz, j, j != L.ny - 1, phic, out + n);
        species_face(a.D_fz, a.phi, g.dz, c, 1, k, k != L.nz - 1, phic, out + 2 * n);
    }
};
struct HeatKind {
    using Args = TseHeatArgs;
    static __device__ __forceinline__ void terms(const TseGrid& g, const Args& a, const CellIdx& x,
                                                 const Layout& L, const double* faces,
                                                 TransportTerms& T) {
        heat_terms(g, a, x, L, faces, T);
    }
    static __device__ __forceinline__ void faces(const TseGrid& g, const Args& a, const Layout& L,
                                                 long long c, int i, int j, int k, double* out) {
        const long long n = (long long)L.nx * L.ny * L.nz;
        heat_face(a, g.dx, c, (long long)L.ny * L.nz, i, i != L.nx - 1, out, out + 3 * n);
        heat_face(a, g.dy, c, L.nz, j, j != L.ny - 1, out + n, out + 4 * n);
        heat_face(a, g.dz, c, 1, k, k != L.nz - 1, out + 2 * n, out + 5 * n);
    }
};

// The exact form's assemblies are bound by the latency of their loads (15 input
// arrays, neighbours included).  Four 256-thread blocks per SM (64 registers,
// some spilled): with the face values read from the face pass, measured on the
// 256 x 256 x 128 reservoir (whole mixed-precision calls, which shared these
// kernels), a species
// solve of 5 iterations took 1.65 ms at four blocks, 1.89 at three and 2.09 at
// two (heat, 3 iterations: 1.39, 1.51, 1.65 ms).
#ifndef TSE_ASM_MINB
#define TSE_ASM_MINB 4
#endif
constexpr int kAssembleMinBlocks = TSE_ASM_MINB;

// One thread per cell of the padded natural order.
template <class Kind>
__device__ __forceinline__ void assemble_body(const TseGrid& g, const typename Kind::Args& a,
                                              const TransportForm& F, uint8_t* mask0, uint8_t* mask1,
                                              const Layout& L, const double* __restrict__ faces) {
    CellIdx x;
    if (!decode_padded((long long)blockIdx.x * kBlock + threadIdx.x, L, x)) return;
    uint8_t* msk = x.col ? mask1 : mask0;
    if (x.pad) {
        store_padding(F, msk, x);
        return;
    }
    TransportTerms T;
    Kind::terms(g, a, x, L, faces, T);
    store_terms(F, msk, x, T, L.nx, L.ny, L.nz);
}

// coefficient part of compute_C.solve (tse.py:795-868)
__global__ void __launch_bounds__(kBlock, kAssembleMinBlocks)
    assemble_c_kernel(TseGrid g, TseSpeciesArgs a, TransportForm F, uint8_t* mask0, uint8_t* mask1, Layout L,
                      const double* faces) {
    assemble_body<SpeciesKind>(g, a, F, mask0, mask1, L, faces);
}

// coefficient part of compute_T.solve (tse.py:930-1036)
__global__ void __launch_bounds__(kBlock, kAssembleMinBlocks)
    assemble_t_kernel(TseGrid g, TseHeatArgs a, TransportForm F, uint8_t* mask0, uint8_t* mask1, Layout L,
                      const double* faces) {
    assemble_body<HeatKind>(g, a, F, mask0, mask1, L, faces);
}

// ---------------------------------------------- the mixed-precision assembly
// One pass from the inputs to the first correction cycle (DcFuse): records
// K'_q = omega co_q / Den, r' of the initial iterate, flags, x^2 partials, and
// the FP64 arrays later cycles read.  The same terms as the exact form's, with
// each cell forming its own six faces' means: a face pass's 24 or 48 bytes a
// cell to write and read again cost more than the means.
//
// What bounded it were instructions, FP64 divisions above all (an SM finishes
// 3.7 a clock against 63 additions, and each is some 20 instructions), then the
// latency of its loads, then its 15 stored arrays.  So:
//  - quotients by a spacing, by a product or sum of two spacings or by dt take
//    the divisor's reciprocal from a table {b, 1 / b} (axis_tables_kernel) and
//    one correction step with fused operations, q = a r, q + r (a - b q) (the
//    closing step of a division by Newton's method, Markstein 1990): the
//    rounded quotient but for rare cases one unit in the last place off;
//  - a harmonic mean is (d1 + d2) H1 H2 / (d1 H2 + d2 H1), one division, and
//    heat's two products of means share one each;
//  - with `lean` (a solve that streams its grid and runs alone) the terms only
//    later cycles' sums need are stored, nine words instead of fifteen; a dt
//    halving runs this pass again.
__device__ __forceinline__ double qdiv(double a, double2 b) {
    const double q = a * b.y;
    const double r = __fma_rn(__fma_rn(-b.x, q, a), b.y, q);
    return (__double2hiint(q) & 0x7ff00000) == 0x7ff00000 ? q : r;   // inf, NaN
}
// An infinite divisor (a steady state's dt, a product of spacings) goes along as
// {0, 0}: the correction is then 0, where -inf 0 + a would be NaN, and the
// quotient a 0.
// |v| far from both ends of the exponent range (and not 0, inf or NaN)
__device__ __forceinline__ bool mid_range(double v) {
    const unsigned e = ((unsigned)__double2hiint(v) >> 20) & 0x7ffu;
    return e - 64u < 1920u;
}

// Per axis and index i four pairs {b, 1 / b}: b = d[i], the + face's and the -
// face's (0.5 (d[i] + d[i +- 1])) d[i], and d[i] + d[i + 1] ({1, 1} where the
// axis has no such neighbour); all indices' first pairs (x, y, z axes in turn),
// then all second pairs ...: along z a warp's loads are contiguous.
constexpr int kTabPairs = 4;
__global__ void axis_tables_kernel(TseGrid g, double2* tab) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.nx + g.ny + g.nz) return;
    double2* t = tab + i;
    const int st = g.nx + g.ny + g.nz;
    const double* d = g.dx;
    int n = g.nx;
    if (i >= g.nx + g.ny) {
        i -= g.nx + g.ny;
        d = g.dz;
        n = g.nz;
    } else if (i >= g.nx) {
        i -= g.nx;
        d = g.dy;
        n = g.ny;
    }
    const double dd = d[i];
    double b[kTabPairs] = {dd, 1.0, 1.0, 1.0};
    if (i + 1 < n) {
        b[1] = (0.5 * (d[i + 1] + dd)) * dd;
        b[3] = d[i + 1] + dd;
    }
    if (i > 0) b[2] = (0.5 * (d[i - 1] + dd)) * dd;
    // an infinite product as {0, 0}, see qdiv; the others are spacings too
    for (int q = 0; q < kTabPairs; ++q) {
        const double r = 1.0 / b[q];
        t[q * st] = make_double2(r == 0.0 && (q == 1 || q == 2) ? 0.0 : b[q], r);
    }
}
static size_t axis_table_bytes(const Layout& L) {
    return align256((size_t)(L.nx + L.ny + L.nz) * kTabPairs * sizeof(double2));
}

// the dispersion terms as a call: cells without dispersivity leave its
// registers to the rest of the pass
__device__ __noinline__ void dispersivity_call(const double* qx, const double* qy, const double* qz,
                                               const double* l_l, const double* l_t, const double* B, int i,
                                               int j, int k, int nx, int ny, int nz, double* D) {
    dispersivity_dev(qx, qy, qz, l_l, l_t, B, i, j, k, nx, ny, nz, D);
}

// axis(): one axis of a cell, added to M, to the neighbour sum s of the initial
// iterate and into the two coefficients.  A face is always formed with its +
// cell's values first, so both its cells get the same bits.
struct SpeciesFast {
    using Args = TseSpeciesArgs;
    static constexpr int kBlocks = 5;   // resident on a SM
    static __device__ __forceinline__ const double* X(const Args& a) { return a.C; }
    static __device__ __forceinline__ const double* B(const Args& a) { return a.BC; }
    static __device__ __forceinline__ const double* W(const Args& a) { return a.WC; }
    static __device__ __forceinline__ const double* field(const Args& a, int axis) {
        return axis == 0 ? a.D_fx : axis == 1 ? a.D_fy : a.D_fz;
    }
    // harm2(D) amean2(phi) of the face between cells p (+) and m (-)
    static __device__ __forceinline__ double mean(const double* D, const double* phi, long long p, long long m,
                                                  double dp, double dm, double2 s) {
        const double H1 = D[p], H2 = D[m];
        const double por = qdiv(phi[p] * dp + phi[m] * dm, s);
        if (!(H1 != 0.0 && H2 != 0.0)) return 0.0 * por;
        const double n = s.x * (H1 * H2), t = __fma_rn(dp, H2, dm * H1);
        if (mid_range(H1 * H2) && mid_range(n) && mid_range(t)) return n / t * por;
        return (dp + dm) / (dp / H1 + dm / H2) * por;
    }
    static __device__ __forceinline__ void axis(const Args& a, int ax, const double* q, const double2* t,
                                                int ts, long long c, long long st, bool hp, bool hm, double DdP,
                                                double DdM, double& M, double& s, double& coP, double& coM) {
        const double* D = field(a, ax);
        const double2 b = t[0];
        const double z = 0.0 * b.y;
        coP = coM = 0.0;
        if (hp) {
            const double qc = q[c];
            const double f = mean(D, a.phi, c + st, c, t[1].x, b.x, t[3 * ts]);
            const double d = qdiv(f + DdP, t[ts]), qd = qdiv(qc, b);
            coP = d - ((0.0 < qc) ? z : qd);
            M = M - d - ((0.0 > qc) ? z : qd);
            s = s + coP * a.C[c + st];
        }
        if (hm) {
            const double qm = q[c - st];
            const double f = mean(D, a.phi, c, c - st, b.x, t[-1].x, t[3 * ts - 1]);
            const double d = qdiv(f + DdM, t[2 * ts]), qd = qdiv(qm, b);
            coM = d + ((0.0 > qm) ? z : qd);
            M = M - d + ((0.0 < qm) ? z : qd);
            s = s + coM * a.C[c - st];
        }
    }
    static __device__ __forceinline__ void rest(const Args& a, long long c, double Xn, double& Rnum, double& EX) {
        Rnum = a.RC[c] * a.phi[c];
        EX = a.imblflo ? Xn / a.rho_f[c] * a.e[c] : 0.0;
    }
};
struct HeatFast {
    using Args = TseHeatArgs;
    static constexpr int kBlocks = 4;
    static __device__ __forceinline__ const double* X(const Args& a) { return a.T; }
    static __device__ __forceinline__ const double* B(const Args& a) { return a.BT; }
    static __device__ __forceinline__ const double* W(const Args& a) { return a.WT; }
    // the conductivity mix and the mean of rho_f times that of cp_f
    static __device__ __forceinline__ void means(const Args& a, long long p, long long m, double dp, double dm,
                                                 double2 s, double& k1, double& rc) {
        const double por = qdiv(a.phi[p] * dp + a.phi[m] * dm, s);
        const double f1 = a.l_f[p], f2 = a.l_f[m], r1 = a.l_r[p], r2 = a.l_r[m];
        const double c1 = a.cp_f[p], c2 = a.cp_f[m], h1 = a.rho_f[p], h2 = a.rho_f[m];
        // numerators and denominators of the four harmonic means, less the
        // common factor dp + dm
        const double nf = f1 * f2, tf = __fma_rn(dp, f2, dm * f1), nr = r1 * r2, tr = __fma_rn(dp, r2, dm * r1);
        const double nc = c1 * c2, tc = __fma_rn(dp, c2, dm * c1), nh = h1 * h2, th = __fma_rn(dp, h2, dm * h1);
        const double nk = s.x * __fma_rn((1 - por) * nr, tf, por * nf * tr), tk = tf * tr;
        const double n2 = (s.x * nc) * (s.x * nh), t2 = tc * th;
        if (mid_range(nf) && mid_range(nr) && mid_range(nc) && mid_range(nh) && mid_range(tk) &&
            mid_range(t2) && mid_range(nk) && mid_range(n2)) {
            k1 = nk / tk;
            rc = n2 / t2;
        } else {
            rc = harm2(h1, h2, dp, dm) * harm2(c1, c2, dp, dm);
            k1 = (1 - por) * harm2(r1, r2, dp, dm) + por * harm2(f1, f2, dp, dm);
        }
    }
    static __device__ __forceinline__ void axis(const Args& a, int, const double* q, const double2* t, int ts,
                                                long long c, long long st, bool hp, bool hm, double DdP,
                                                double DdM, double& M, double& s, double& coP, double& coM) {
        const double2 b = t[0];
        coP = coM = 0.0;
        if (hp) {
            const double qc = q[c];
            double k1, rc;
            means(a, c + st, c, t[1].x, b.x, t[3 * ts], k1, rc);
            const double d = qdiv(k1 + DdP * rc, t[ts]), S = qdiv(rc, b);
            coP = d - min0(qc) * S;
            M = M - d - max0(qc) * S;
            s = s + coP * a.T[c + st];
        }
        if (hm) {
            const double qm = q[c - st];
            double k1, rc;
            means(a, c, c - st, b.x, t[-1].x, t[3 * ts - 1], k1, rc);
            const double d = qdiv(k1 + DdM * rc, t[2 * ts]), S = qdiv(rc, b);
            coM = d + max0(qm) * S;
            M = M - d + min0(qm) * S;
            s = s + coM * a.T[c - st];
        }
    }
    static __device__ __forceinline__ void rest(const Args& a, long long c, double Xn, double& Rnum, double& EX) {
        const double por = a.phi[c];
        Rnum = por * a.rho_f[c] * a.cp_f[c] + (1 - por) * a.rho_r[c] * a.cp_r[c];
        EX = a.imblflo ? a.cp_f[c] * Xn * a.e[c] : 0.0;
    }
};

// Measured at 256 x 256 x 128 (B200), dispersivity 0, with the first cycle's
// records: species 582 us (face pass and assembly took 963), heat 747 (1089).
// It waits for its loads most of the time (1.7 of 4 instructions a clock): more
// blocks a SM help as long as registers last (species 630 us with 4 blocks, heat
// 858 with 5), loads gathered ahead of the arithmetic cost more registers than
// they hide (species 640 and more).
// STEADY: a.dt is infinite (an instance of its own costs the others nothing; a
// test of dt in the kernel 1 % of a call).
template <class Kind, bool LEAN, bool STEADY>
__global__ void __launch_bounds__(kBlock, Kind::kBlocks)
    assemble_fast_kernel(TseGrid g, typename Kind::Args a, TransportForm F, uint8_t* mask0, uint8_t* mask1,
                         Layout L, const double2* __restrict__ tab, DcFuse fz) {
    __shared__ double sh[kBlock / 32];
    const double2 dt = STEADY ? make_double2(0.0, 0.0) : make_double2(a.dt, 1.0 / a.dt);
    const double omega = F.omega;
    const long long N = F.Ncal;
    const int ts = L.nx + L.ny + L.nz;
    double x2 = 0.0;
    for (int rep = 0; rep < fz.per_thread; ++rep) {
        CellIdx x;
        const long long t = ((long long)blockIdx.x * fz.per_thread + rep) * kBlock + threadIdx.x;
        if (!decode_padded(t, L, x)) break;
        uint8_t* msk = x.col ? mask1 : mask0;
        double* b = (x.col ? F.arr[1] : F.arr[0]) + x.m;
        float* Kc = x.col ? fz.K[1] : fz.K[0];
        float2* rec = k_rec(Kc, fz.ks, x.m);
        if (x.pad) {
            for (int q = 0; q < TA_COUNT; ++q) b[q * N] = 0.0;
            msk[x.m] = 0;
            for (int q = 0; q < 3; ++q) rec[q] = make_float2(0.0f, 0.0f);
            *k_rp(Kc, fz.ks, x.m) = 0.0f;
            *k_flag(Kc, fz.ks, x.m) = 0;
            continue;
        }
        const int i = x.i, j = x.j, k = x.k;
        const long long c = x.c;
        double Dd[6] = {0, 0, 0, 0, 0, 0};
        if (a.l_l[c] != 0 || a.l_t[c] != 0)
            dispersivity_call(a.qx, a.qy, a.qz, a.l_l, a.l_t, Kind::B(a), i, j, k, L.nx, L.ny, L.nz, Dd);
        double M = 0.0, s = 0.0, co[6];
        Kind::axis(a, 0, a.qx, tab + i, ts, c, (long long)L.ny * L.nz, i != L.nx - 1, i != 0, Dd[3],
                   Dd[0], M, s, co[0], co[1]);
        Kind::axis(a, 1, a.qy, tab + L.nx + j, ts, c, L.nz, j != L.ny - 1, j != 0, Dd[4], Dd[1], M, s,
                   co[2], co[3]);
        Kind::axis(a, 2, a.qz, tab + L.nx + L.ny + k, ts, c, 1, k != L.nz - 1, k != 0, Dd[5], Dd[2], M,
                   s, co[4], co[5]);
        const double Xn = Kind::X(a)[c], W = Kind::W(a)[c];
        const bool active = !(Kind::B(a)[c] != 0.0);
        double Rnum, EX;
        Kind::rest(a, c, Xn, Rnum, EX);
        const double R = qdiv(Rnum, dt), den = R - omega * M;
#pragma unroll
        for (int q = 0; q < 6; ++q) b[q * N] = co[q];
        // the terms that stay fixed during the solve, in sum()'s order
        double num = omega * s, fix;
        const double Y = F.useY ? (1 - omega) * (Xn * M + s) : 0.0;
        fix = R * Xn;
        if (F.useY) fix = Y + fix;
        fix = fix + W;
        if (F.useEX) fix = fix - EX;
        num = num + fix;
        b[TA_DEN * N] = den;
        b[TA_X * N] = Xn;
        if (LEAN) {
            b[TA_RXN * N] = fix;
        } else {
            b[TA_RXN * N] = R * Xn;
            b[TA_W * N] = W;
            if (F.useY) b[TA_Y * N] = Y;
            if (F.useEX) b[TA_EX * N] = EX;
            b[TA_RNUM * N] = Rnum;
            b[TA_M * N] = M;
            b[TA_XN * N] = Xn;
        }
        uint8_t f = neighbour_flags(i, j, k, L.nx, L.ny, L.nz);
        if (active) f |= F_ACTIVE;
        msk[x.m] = f;
        *k_flag(Kc, fz.ks, x.m) = f;
        float rp = 0.0f;
        if (active) {
            const double rden = 1.0 / den, w = omega * rden;
#pragma unroll
            for (int q = 0; q < 3; ++q)
                rec[q] = make_float2((float)(co[2 * q] * w), (float)(co[2 * q + 1] * w));
            rp = (float)((num - den * Xn) * rden);
        } else {
#pragma unroll
            for (int q = 0; q < 3; ++q) rec[q] = make_float2(0.0f, 0.0f);
        }
        *k_rp(Kc, fz.ks, x.m) = rp;
        x2 = x2 + Xn * Xn;
    }
    const double bs = block_sum<kBlock>(x2, sh);
    if (threadIdx.x == 0) fz.partials[blockIdx.x] = bs;
}

// the face pass before an assembly: one thread per cell, natural order
template <class Kind>
__global__ void faces_kernel(TseGrid g, typename Kind::Args a, Layout L, double* faces) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= (long long)L.nx * L.ny * L.nz) return;
    int i, j, k;
    long long row;
    grid_coords(c, L.ny, L.nz, i, j, k, row);
    Kind::faces(g, a, L, c, i, j, k, faces);
}

__global__ void unpack_t_kernel(double* out, const double* X0, const double* X1, Layout L) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)L.nx * L.ny * L.nz;
    if (t >= total) return;
    int i, j, k;
    long long row;
    grid_coords(t, L.ny, L.nz, i, j, k, row);
    const long long m = (row * L.nzp + k) >> 1;
    out[t] = ((i + j + k) & 1) ? X1[m] : X0[m];
}

// face values a cell: 3 for a species, 6 for heat
constexpr int kTransportFaceWords = 6;

size_t transport_ws_bytes(const Layout& L, long long* Ncal_out) {
    long long Ncal = (L.Nc + 31) & ~31LL;
    if (Ncal_out) *Ncal_out = Ncal;
    size_t b = 0;
    b += align256(sizeof(GridBarrier));
    b += align256((size_t)2 * kMaxBlocks * sizeof(double));
    b += 2 * align256((size_t)Ncal);
    b += 2 * (size_t)TA_COUNT * Ncal * sizeof(double);
    // the exact form's face pass, or the mixed-precision form's axis tables
    b += std::max(align256((size_t)kTransportFaceWords * L.nx * L.ny * L.nz * sizeof(double)), axis_table_bytes(L));
    return b;
}

// Carve the workspace (shared by the exact and the defect-correction
// transport solves) and reset the grid barrier.
template <class Args>
static int carve_transport(const TseGrid* grid, const Args* a, void* d_ws, size_t ws_bytes,
                           cudaStream_t stream, int imbl, TransportSetup& S) {
    S.L = make_layout(grid->nx, grid->ny, grid->nz);
    const size_t need = transport_ws_bytes(S.L, &S.Ncal);
    if (need > ws_bytes) return TSE_ERR_WORKSPACE;
    char* p = (char*)d_ws;
    S.bar = (GridBarrier*)p;
    p += align256(sizeof(GridBarrier));
    S.partials = (double*)p;
    p += align256((size_t)2 * kMaxBlocks * sizeof(double));
    S.mask[0] = (uint8_t*)p;
    p += align256((size_t)S.Ncal);
    S.mask[1] = (uint8_t*)p;
    p += align256((size_t)S.Ncal);
    S.F.arr[0] = (double*)p;
    S.F.arr[1] = S.F.arr[0] + (size_t)TA_COUNT * S.Ncal;
    S.faces = S.F.arr[1] + (size_t)TA_COUNT * S.Ncal;
    S.F.Ncal = S.Ncal;
    S.F.SX = S.L.SX;
    S.F.H = S.L.H;
    S.F.omega = a->omega;
    S.F.SOR = a->SOR;
    S.F.useY = a->omega != 1.0;
    S.F.useEX = imbl != 0;
    S.F.useW = 1;
    S.tail = (char*)d_ws + need;
    S.tail_bytes = ws_bytes - need;
    if (cudaMemsetAsync(S.bar, 0, sizeof(GridBarrier), stream) != cudaSuccess) return TSE_ERR_LAUNCH;
    return TSE_OK;
}

// the face pass of an exact setup
template <class Args, class FacesK>
static void launch_faces(const TseGrid* grid, const Args* a, const TransportSetup& S, FacesK fk,
                         cudaStream_t stream) {
    const long long n = (long long)S.L.nx * S.L.ny * S.L.nz;
    fk<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock, 0, stream>>>(*grid, *a, S.L, S.faces);
}

// carve + the face pass + the exact form's assembly
template <class Args, class FacesK, class AssembleK>
static int setup_transport(const TseGrid* grid, const Args* a, void* d_ws, size_t ws_bytes,
                           cudaStream_t stream, FacesK fk, AssembleK kernel, int imbl,
                           TransportSetup& S) {
    int rc = carve_transport(grid, a, d_ws, ws_bytes, stream, imbl, S);
    if (rc != TSE_OK) return rc;
    launch_faces(grid, a, S, fk, stream);
    const long long total = (long long)S.L.nx * S.L.ny * S.L.nzp;
    kernel<<<(unsigned)((total + kBlock - 1) / kBlock), kBlock, 0, stream>>>(
        *grid, *a, S.F, S.mask[0], S.mask[1], S.L, S.faces);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

// the mixed-precision form's assembly of a carved setup, for the given dt
template <class Kind>
static int assemble_fast(const TseGrid* grid, const typename Kind::Args* a, TransportSetup& S, int* nparts,
                         cudaStream_t stream) {
    DcCtl c;
    dc_carve(S, c, TA_X);
    long long per, nb;
    dc_fuse_grid(S.L, per, nb);
    DcFuse fz;
    fz.K[0] = c.K[0];
    fz.K[1] = c.K[1];
    fz.ks = c.ks;
    fz.partials = S.partials;
    fz.per_thread = (int)per;
    double2* tab = (double2*)S.faces;
    const int nt = S.L.nx + S.L.ny + S.L.nz;
    axis_tables_kernel<<<(unsigned)((nt + 127) / 128), 128, 0, stream>>>(*grid, tab);
    // the form as the assembly fills it: with `lean` its later sums read one
    // fixed term (setup_transport_dc), its own switches say what goes in
    TransportForm F = S.F;
    F.useY = a->omega != 1.0;
    F.useEX = a->imblflo != 0;
    const bool steady = std::isinf(a->dt);
    auto kernel = S.lean ? (steady ? assemble_fast_kernel<Kind, true, true> : assemble_fast_kernel<Kind, true, false>)
                         : (steady ? assemble_fast_kernel<Kind, false, true> : assemble_fast_kernel<Kind, false, false>);
    kernel<<<(unsigned)nb, kBlock, 0, stream>>>(*grid, *a, F, S.mask[0], S.mask[1], S.L, tab, fz);
    *nparts = (int)nb;
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

// carve + the mixed-precision form's assembly; *nparts: the number of x^2
// partials.  S.lean: see SolveSetup.
template <class Kind>
static int setup_transport_dc(const TseGrid* grid, const typename Kind::Args* a, void* d_ws, size_t ws_bytes,
                              cudaStream_t stream, TransportSetup& S, int* nparts) {
    int rc = carve_transport(grid, a, d_ws, ws_bytes, stream, a->imblflo, S);
    if (rc != TSE_OK) return rc;
    if (S.tail_bytes < dc_extra_bytes(S.L)) return TSE_ERR_WORKSPACE;
    if (S.lean) S.F.useY = S.F.useEX = S.F.useW = 0;
    return assemble_fast<Kind>(grid, a, S, nparts, stream);
}

int setup_species(const TseGrid* grid, const TseSpeciesArgs* a, void* d_ws, size_t ws_bytes,
                  cudaStream_t stream, TransportSetup& S) {
    return setup_transport(grid, a, d_ws, ws_bytes, stream, faces_kernel<SpeciesKind>,
                           assemble_c_kernel, a->imblflo, S);
}

int setup_heat(const TseGrid* grid, const TseHeatArgs* a, void* d_ws, size_t ws_bytes,
               cudaStream_t stream, TransportSetup& S) {
    return setup_transport(grid, a, d_ws, ws_bytes, stream, faces_kernel<HeatKind>,
                           assemble_t_kernel, a->imblflo, S);
}

int setup_species_dc(const TseGrid* grid, const TseSpeciesArgs* a, void* d_ws, size_t ws_bytes,
                     cudaStream_t stream, TransportSetup& S, int* nparts) {
    return setup_transport_dc<SpeciesFast>(grid, a, d_ws, ws_bytes, stream, S, nparts);
}

int setup_heat_dc(const TseGrid* grid, const TseHeatArgs* a, void* d_ws, size_t ws_bytes,
                  cudaStream_t stream, TransportSetup& S, int* nparts) {
    return setup_transport_dc<HeatFast>(grid, a, d_ws, ws_bytes, stream, S, nparts);
}

int again_species_dc(const TseGrid* grid, const TseSpeciesArgs* a, cudaStream_t stream, TransportSetup& S,
                     int* nparts) {
    return assemble_fast<SpeciesFast>(grid, a, S, nparts, stream);
}

int again_heat_dc(const TseGrid* grid, const TseHeatArgs* a, cudaStream_t stream, TransportSetup& S,
                  int* nparts) {
    return assemble_fast<HeatFast>(grid, a, S, nparts, stream);
}

template <class Args, class FacesK, class AssembleK>
static int run_transport(const TseGrid* grid, const Args* a, double* X, TseSolveStatus* d_status,
                         void* d_ws, size_t ws_bytes, void* stream_, FacesK fk, AssembleK kernel,
                         int imbl) {
    cudaStream_t stream = (cudaStream_t)stream_;
    TransportSetup S;
    int rc = setup_transport(grid, a, d_ws, ws_bytes, stream, fk, kernel, imbl, S);
    if (rc != TSE_OK) return rc;
    const Layout L = S.L;
    TransportForm F = S.F;
    struct {
        GridBarrier* bar;
        double* partials;
        uint8_t* mask[2];
        double* arr[2];
        long long Ncal;
    } w = {S.bar, S.partials, {S.mask[0], S.mask[1]}, {S.F.arr[0], S.F.arr[1]}, S.Ncal};
    SolveCtl ctl;
    ctl.L = L;
    ctl.Ncal = w.Ncal;
    ctl.plain_sweep = plain_sweep(a->sweep, ctl.L);
    ctl.dt = a->dt;
    ctl.inc_it = a->inc_it;
    ctl.max_dt = a->max_dt;
    ctl.min_dt = a->min_dt;
    ctl.conv = a->conv;
    ctl.max_it = a->max_it;
    ctl.pressure_schedule = 0;
    ctl.stop_on_first = a->omega == 0.0;
    ctl.X[0] = w.arr[0] + (size_t)TA_X * w.Ncal;
    ctl.X[1] = w.arr[1] + (size_t)TA_X * w.Ncal;
    ctl.mask[0] = w.mask[0];
    ctl.mask[1] = w.mask[1];
    ctl.partials = w.partials;
    ctl.bar = w.bar;
    ctl.status = d_status;
    if (a->sweep != 1 && a->sweep != 2) {
        rc = launch_rb_resident(F, ctl, S.tail, S.tail_bytes, X, stream);
        if (rc != 1) return rc;
    }
    rc = launch_rb_solve_tma(F, ctl, stream);
    if (rc == 1) rc = launch_rb_solve(F, ctl, stream);
    if (rc != TSE_OK) return rc;
    const long long nat = (long long)L.nx * L.ny * L.nz;
    unpack_t_kernel<<<(unsigned)((nat + kBlock - 1) / kBlock), kBlock, 0, stream>>>(X, ctl.X[0],
                                                                                     ctl.X[1], L);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    return TSE_OK;
}

// smolarkiewicz (tse.py:1083-1116)
__global__ void smolarkiewicz_kernel(TseGrid g, const double* C, const double* qx, const double* qy,
                                     const double* qz, double* vx, double* vy, double* vz,
                                     double dt, double eps, double Sc) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const long long total = (long long)nx * ny * nz;
    if (t >= total) return;
    int i, j, k;
    long long row;
    grid_coords(t, ny, nz, i, j, k, row);
    const double c0 = C[t];
    if (c0 > 0) {
        double dd;
        if (i < nx - 1) {
            const double c1 = C[t + (long long)ny * nz];
            const double q = qx[t];
            dd = 0.5 * (g.dx[i + 1] + g.dx[i]);
            vx[t] = (Sc * (fabs(q) * dd - dt * (q * q)) * (c1 - c0) / ((c0 + c1 + eps) * dd));
        }
        if (j < ny - 1) {
            const double c1 = C[t + nz];
            const double q = qy[t];
            dd = 0.5 * (g.dy[j + 1] + g.dy[j]);
            vy[t] = (Sc * (fabs(q) * dd - dt * (q * q)) * (c1 - c0) / ((c0 + c1 + eps) * dd));
        }
        if (k < nz - 1) {
            const double c1 = C[t + 1];
            const double q = qz[t];
            dd = 0.5 * (g.dz[k + 1] + g.dz[k]);
            vz[t] = (Sc * (fabs(q) * dd - dt * (q * q)) * (c1 - c0) / ((c0 + c1 + eps) * dd));
        }
    } else {
        vx[t] = 0.0;
        vy[t] = 0.0;
        vz[t] = 0.0;
    }
}

}  // namespace tse

using namespace tse;

extern "C" int32_t tse_compute_C(const TseGrid* grid, const TseSpeciesArgs* a,
                                 TseSolveStatus* d_status, void* d_ws, size_t ws_bytes,
                                 void* stream) {
    if (!grid || !a || !d_status || !d_ws) return TSE_ERR_ARG;
    if (grid->nx < 1 || grid->ny < 1 || grid->nz < 1 || a->max_it < 1) return TSE_ERR_ARG;
    if (!a->C || !a->D_fx || !a->D_fy || !a->D_fz || !a->phi || !a->rho_f || !a->qx || !a->qy ||
        !a->qz || !a->BC || !a->WC || !a->RC || !a->e || !a->l_l || !a->l_t)
        return TSE_ERR_ARG;
    return run_transport(grid, a, a->C, d_status, d_ws, ws_bytes, stream, faces_kernel<SpeciesKind>,
                         assemble_c_kernel, a->imblflo);
}

extern "C" int32_t tse_compute_T(const TseGrid* grid, const TseHeatArgs* a,
                                 TseSolveStatus* d_status, void* d_ws, size_t ws_bytes,
                                 void* stream) {
    if (!grid || !a || !d_status || !d_ws) return TSE_ERR_ARG;
    if (grid->nx < 1 || grid->ny < 1 || grid->nz < 1 || a->max_it < 1) return TSE_ERR_ARG;
    if (!a->T || !a->l_f || !a->cp_f || !a->rho_f || !a->phi || !a->qx || !a->qy || !a->qz ||
        !a->BT || !a->WT || !a->e || !a->l_r || !a->rho_r || !a->cp_r || !a->l_l || !a->l_t)
        return TSE_ERR_ARG;
    return run_transport(grid, a, a->T, d_status, d_ws, ws_bytes, stream, faces_kernel<HeatKind>,
                         assemble_t_kernel, a->imblflo);
}

extern "C" int32_t tse_smolarkiewicz(const TseGrid* grid, const double* C, const double* qx,
                                     const double* qy, const double* qz, double* vx, double* vy,
                                     double* vz, double dt, double eps, double Sc, void* stream) {
    if (!grid || !C || !qx || !qy || !qz || !vx || !vy || !vz) return TSE_ERR_ARG;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    if (n <= 0) return TSE_ERR_ARG;
    smolarkiewicz_kernel<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock, 0, (cudaStream_t)stream>>>(
        *grid, C, qx, qy, qz, vx, vy, vz, dt, eps, Sc);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}
