// Darcy fluxes, flow-balance error, CFL / Neumann limits, L2 norm, field
// statistics, Peclet diagnostics and the declared linear EOS.
// FP64, reference operation order, compiled with --fmad=false.
#include <algorithm>
#include <cmath>

#include "tse_common.cuh"
#include "tse_quotient.cuh"

namespace tse {

constexpr int kRedBlocks = 1024;   // fixed partial count: deterministic reductions

__device__ __forceinline__ void decode(long long t, int ny, int nz, int& i, int& j, int& k) {
    long long row;
    grid_coords(t, ny, nz, i, j, k, row);
}

// The flux kernels walk along x with a warp on 32 consecutive cells of the
// (y, z) plane: the x face and its quotients stay in registers, a z face's come
// from the next lane (rows need no alignment: a row's last cell has no + face),
// and reciprocals of spacings are formed once a walk.  Lanes at a warp's ends
// repeat cells of the next one.
constexpr int kWalkMax = 16;
// From these grid sizes on; below, a thread a cell keeps the SMs fuller (us,
// thread a cell against walks: fluxes 36 / 39 at 96^3, 74 / 57 at 112^3, 156 / 111
// at 160 x 192 x 101; flow error 5.2 / 6.5 at 48^3, 18.5 / 16.6 at 80^3, 101 / 85).
// On a plane (ny = 1) a thread a cell skips the y faces that a walk forms all the
// same: flow error 14.4 / 18.5 at 1000 x 1 x 500, 53 / 60 at 2000 x 1 x 1000.
constexpr long long kWalkCellsQ = 1200000, kWalkCellsE = 400000;
// Blocks resident on a SM.  Flow error: 3 below kWalkCellsE4 cells, where another
// block's shorter walks start over more often, else 4 (us with 3 / 4: 22.5 / 24.9
// at 90^3, 47 / 49 at 128 x 128 x 100, 62 / 58 at 128^3, 231 / 221 at 255 x 256 x
// 127, launched alone).
constexpr int kWalkBlocksQ = 4;
constexpr long long kWalkCellsE4 = 2000000;
constexpr int kWalkWarps = kBlock / 32;
struct Walk {
    int steps;                // cells of a walk
    unsigned tiles, blocks;   // blocks across the plane, and of all walks
};
// The length whose waves of resident blocks take the fewest steps in all, one
// more a walk for its start (a last wave that is nearly empty costs a full one).
static bool walk_of(const TseGrid& g, int out_lanes, int blocks_per_sm, Walk& w) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
        return false;
    const long long plane = (long long)g.ny * g.nz;
    const long long warps = (plane + out_lanes - 1) / out_lanes, slots = (long long)sms * blocks_per_sm;
    w = {1, (unsigned)((warps + kWalkWarps - 1) / kWalkWarps), 0};
    long long best = 0;
    for (int s = kWalkMax; s >= 1; --s) {
        const long long blocks = (long long)w.tiles * ((g.nx + s - 1) / s);
        const long long cost = (blocks + slots - 1) / slots * (s + 1);
        if (best == 0 || cost < best) {
            best = cost;
            w.steps = s;
            w.blocks = (unsigned)blocks;
        }
    }
    return true;
}
// along x: spacings dx[i0 - 1 .. i0 + steps] and the divisors dx[i] and
// dx[i] + dx[i + 1] of cells i0 - 1 .. (spacing 1 beside the grid, unused)
struct WalkX {
    double d[kWalkMax + 2];
    Divisor own[kWalkMax + 1], sum[kWalkMax + 1];
    // false in every thread if a divisor is not plain
    __device__ __forceinline__ bool fill(const TseGrid& g, int i0) {
        bool ok = true;
        for (int q = threadIdx.x; q < kWalkMax + 2; q += blockDim.x) {
            const int i = i0 - 1 + q;
            const double a = i >= 0 && i < g.nx ? g.dx[i] : 1.0;
            d[q] = a;
            ok = ok && plain_positive(a);
            if (q < kWalkMax + 1) {
                const double b = i + 1 < g.nx ? g.dx[i + 1] : 1.0;
                own[q] = divisor(a);
                sum[q] = divisor(b + a);
                ok = ok && plain_positive(b + a);
            }
        }
        return __syncthreads_and(ok);
    }
};

// compute_q (tse.py:744-780); q on the last plane of each axis is not written
__device__ __forceinline__ void darcy_cell(const TseGrid& g, long long t, int i, int j, int k, const double* P,
                                           const double* BP, const double* Kx, const double* Ky,
                                           const double* Kz, double* qx, double* qy, double* qz,
                                           const double* nue, const double* rho) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const double *dx = g.dx, *dy = g.dy, *dz = g.dz;
    if (i < nx - 1) {
        const long long o = t + (long long)ny * nz;
        if (!(BP[t] != 0 && BP[o] != 0))
            qx[t] = (-harm2(Kx[o], Kx[t], dx[i + 1], dx[i]) / harm2(nue[o], nue[t], dx[i + 1], dx[i]) *
                     ((P[o] - P[t]) / (0.5 * (dx[i + 1] + dx[i])) +
                      amean2(rho[o], rho[t], dx[i + 1], dx[i]) * g.g * g.sin_beta));
        else
            qx[t] = 0.0;
    }
    if (j < ny - 1) {
        const long long o = t + nz;
        if (!(BP[t] != 0 && BP[o] != 0))
            qy[t] = (-harm2(Ky[o], Ky[t], dy[j + 1], dy[j]) / harm2(nue[o], nue[t], dy[j + 1], dy[j]) *
                     (P[o] - P[t]) / (0.5 * (dy[j + 1] + dy[j])));
        else
            qy[t] = 0.0;
    }
    if (k < nz - 1) {
        const long long o = t + 1;
        if (!(BP[t] != 0 && BP[o] != 0))
            qz[t] = (-harm2(Kz[o], Kz[t], dz[k + 1], dz[k]) / harm2(nue[o], nue[t], dz[k + 1], dz[k]) *
                     ((P[o] - P[t]) / (0.5 * (dz[k + 1] + dz[k])) +
                      amean2(rho[o], rho[t], dz[k + 1], dz[k]) * g.g * g.cos_beta));
        else
            qz[t] = 0.0;
    }
}

__device__ __noinline__ void compute_q_cell(const TseGrid& g, long long t, int i, int j, int k, const double* P,
                                            const double* BP, const double* Kx, const double* Ky,
                                            const double* Kz, double* qx, double* qy, double* qz,
                                            const double* nue, const double* rho) {
    darcy_cell(g, t, i, j, k, P, BP, Kx, Ky, Kz, qx, qy, qz, nue, rho);
}
__global__ void compute_q_cells_kernel(TseGrid g, const double* P, const double* BP, const double* Kx,
                                       const double* Ky, const double* Kz, double* qx, double* qy, double* qz,
                                       const double* nue, const double* rho) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)g.nx * g.ny * g.nz) return;
    int i, j, k;
    decode(t, g.ny, g.nz, i, j, k);
    darcy_cell(g, t, i, j, k, P, BP, Kx, Ky, Kz, qx, qy, qz, nue, rho);
}

// A K of zero (harm2 is then 0) goes along as 1 and a flag.
struct Perm {
    double a;   // d / K
    bool zero;
};
__device__ __forceinline__ Perm perm(double K, double d, bool& ok) {
    const bool z = K == 0.0;
    const double s = z ? 1.0 : K;
    ok = ok && plain_positive(s);
    return {quotient(d, divisor(s)), z};
}
// -harm2(K) / harm2(nue) of a face
__device__ __forceinline__ double mobility(double dsum, const Perm& a, const Perm& b, double n1, double n2) {
    const double sk = a.a + b.a, sn = n1 + n2;
    const double hk = quotient(dsum, divisor(sk)), hn = quotient(dsum, divisor(sn));
    return quotient_0(a.zero || b.zero ? -0.0 : -hk, divisor(hn));
}

// 255 x 256 x 127 (B200): 418 us with a thread a cell and the operator's
// divisions, 286 now (10 arrays, 101 us); 302 with 3 blocks a SM, 318 with 5.  Bound: 15 reciprocals and 23 quotients a cell and the loads' latency
// (FP64 pipe 42 % busy, 28 warps a SM, DRAM 30 %).
__global__ void __launch_bounds__(kBlock, kWalkBlocksQ)
    compute_q_kernel(TseGrid g, Walk w, const double* P, const double* BP, const double* Kx, const double* Ky,
                     const double* Kz, double* qx, double* qy, double* qz, const double* nue,
                     const double* rho) {
    __shared__ WalkX X;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const long long plane = (long long)ny * nz;
    const int i0 = (int)(blockIdx.x / w.tiles) * w.steps, tile = (int)(blockIdx.x % w.tiles);
    bool okd = X.fill(g, i0);
    const int lane = threadIdx.x & 31;
    const long long u = ((long long)tile * kWalkWarps + (threadIdx.x >> 5)) * 31 + lane;
    if (u - lane >= plane) return;   // whole warps only: the others exchange
    const bool out = u < plane && lane < 31;
    const long long c0 = u < plane ? u : plane - 1;
    const int j = (int)(c0 / nz), k = (int)(c0 - (long long)j * nz);
    const bool hy = j < ny - 1, hz = k < nz - 1;
    const double dy0 = g.dy[j], dy1 = hy ? g.dy[j + 1] : 1.0, dz0 = g.dz[k], dz1 = hz ? g.dz[k + 1] : 1.0;
    const Divisor sy = divisor(dy1 + dy0), sz = divisor(dz1 + dz0);
    okd = okd && plain_positive(dy0) && plain_positive(dy1) && plain_positive(dz0) && plain_positive(dz1) &&
          plain_positive(sy.b) && plain_positive(sz.b);
    long long t = (long long)i0 * plane + c0;
    double p = P[t], r = rho[t], n = nue[t], bp = BP[t];
    bool ok0 = okd && plain_positive(n) && plain_positive(r);   // the cell's own values
    Divisor nd = divisor(n);
    Perm ax = perm(Kx[t], X.d[1], ok0);
    double an = quotient(X.d[1], nd);
    const int steps = min(w.steps, nx - i0);
    for (int s = 0; s < steps; ++s, t += plane) {
        const bool hx = i0 + s < nx - 1;
        const long long tx = hx ? t + plane : t, ty = hy ? t + nz : t, tz = hz ? t + 1 : t;
        // the next cell along x, and this cell's + neighbours along y and z
        const double p1 = P[tx], r1 = rho[tx], n1 = nue[tx], kx1 = Kx[tx], b1 = BP[tx];
        const double ky = Ky[t], kz = Kz[t], kyo = Ky[ty], no = nue[ty], po = P[ty], bo = BP[ty];
        const double pz = P[tz], rz = rho[tz], bz = BP[tz];
        const Divisor nd1 = divisor(n1);
        bool ok1 = okd && plain_positive(n1) && plain_positive(r1);
        const Perm ax1 = perm(kx1, X.d[s + 2], ok1);
        const double an1 = quotient(X.d[s + 2], nd1);
        bool ok = ok0 && ok1 && plain_positive(no) && plain_positive(rz);
        Perm zk = perm(kz, dz0, ok);
        const double zn = quotient(dz0, nd);
        const unsigned good = __ballot_sync(0xffffffffu, ok), zero = __ballot_sync(0xffffffffu, zk.zero);
        const Perm zk1 = {__shfl_down_sync(0xffffffffu, zk.a, 1), (zero >> ((lane + 1) & 31) & 1u) != 0};
        const double zn1 = __shfl_down_sync(0xffffffffu, zn, 1);
        ok = ok && (!hz || (good >> ((lane + 1) & 31) & 1u));
        const double px = p1 - p, py = po - p, pu = pz - p;
        ok = ok && plain_signed(px) && plain_signed(py) && plain_signed(pu);
        const Divisor sx = X.sum[s + 1];
        const double vx = mobility(sx.b, ax1, ax, an1, an) *
                          (quotient_0(px, half(sx)) + quotient(r1 * X.d[s + 2] + r * X.d[s + 1], sx) * g.g * g.sin_beta);
        const double vy = quotient_0(mobility(sy.b, perm(kyo, dy1, ok), perm(ky, dy0, ok), quotient(dy1, divisor(no)),
                                              quotient(dy0, nd)) * py,
                                     half(sy));
        const double vz = mobility(sz.b, zk1, zk, zn1, zn) *
                          (quotient_0(pu, half(sz)) + quotient(rz * dz1 + r * dz0, sz) * g.g * g.cos_beta);
        if (out) {
            if (ok) {
                const bool in = bp != 0;
                if (hx) qx[t] = in && b1 != 0 ? 0.0 : vx;
                if (hy) qy[t] = in && bo != 0 ? 0.0 : vy;
                if (hz) qz[t] = in && bz != 0 ? 0.0 : vz;
            } else {
                compute_q_cell(g, t, i0 + s, j, k, P, BP, Kx, Ky, Kz, qx, qy, qz, nue, rho);
            }
        }
        p = p1;
        r = r1;
        bp = b1;
        nd = nd1;
        ax = ax1;
        an = an1;
        ok0 = ok1;
    }
}

// flow_error (tse.py:409-446)
__device__ __forceinline__ double balance_cell(const TseGrid& g, long long t, int i, int j, int k, const double* P,
                                               const double* Pn, const double* qx, const double* qy,
                                               const double* qz, const double* WP, const double* phi,
                                               const double* c_f, const double* c_r, const double* rho,
                                               double dt_P) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const double *dx = g.dx, *dy = g.dy, *dz = g.dz;
    const long long sx = (long long)ny * nz;
    double v = 0.0;
    if (i != nx - 1) v -= (qx[t] / dx[i] * harm2(rho[t + sx], rho[t], dx[i + 1], dx[i]));
    if (i != 0) v += (qx[t - sx] / dx[i] * harm2(rho[t - sx], rho[t], dx[i - 1], dx[i]));
    if (j != ny - 1) v -= (qy[t] / dy[j] * harm2(rho[t + nz], rho[t], dy[j + 1], dy[j]));
    if (j != 0) v += (qy[t - nz] / dy[j] * harm2(rho[t - nz], rho[t], dy[j - 1], dy[j]));
    if (k != nz - 1) v -= (qz[t] / dz[k] * harm2(rho[t + 1], rho[t], dz[k + 1], dz[k]));
    if (k != 0) v += (qz[t - 1] / dz[k] * harm2(rho[t - 1], rho[t], dz[k - 1], dz[k]));
    const double por = phi[t];
    v += (WP[t] + ((1 - por) * c_r[t] + por * c_f[t]) * (P[t] - Pn[t]) * rho[t] / dt_P);
    return v;
}

__device__ __noinline__ double flow_error_cell(const TseGrid& g, long long t, int i, int j, int k, const double* P,
                                               const double* Pn, const double* qx, const double* qy,
                                               const double* qz, const double* WP, const double* phi,
                                               const double* c_f, const double* c_r, const double* rho,
                                               double dt_P) {
    return balance_cell(g, t, i, j, k, P, Pn, qx, qy, qz, WP, phi, c_f, c_r, rho, dt_P);
}
__global__ void flow_error_cells_kernel(TseGrid g, const double* P, const double* Pn, const double* qx,
                                        const double* qy, const double* qz, const double* WP, const double* phi,
                                        const double* c_f, const double* c_r, const double* rho, double dt_P,
                                        double* e) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)g.nx * g.ny * g.nz) return;
    int i, j, k;
    decode(t, g.ny, g.nz, i, j, k);
    e[t] = balance_cell(g, t, i, j, k, P, Pn, qx, qy, qz, WP, phi, c_f, c_r, rho, dt_P);
}

// harm2 from its two quotients
__device__ __forceinline__ double harm_of(double dsum, double a1, double a2) {
    return quotient(dsum, divisor(a1 + a2));
}

// A face's mean density is the same bits from either side.  255 x 256 x 127
// (B200): 305 us with a thread a cell, 221 now (11 arrays, 112 us).  Bound: 7 reciprocals and 18 quotients a cell and the loads'
// latency (FP64 pipe 41 % busy, 21 warps a SM, DRAM 45 %).
template <int BLOCKS>
__global__ void __launch_bounds__(kBlock, BLOCKS)
    flow_error_kernel(TseGrid g, Walk w, const double* P, const double* Pn, const double* qx, const double* qy,
                      const double* qz, const double* WP, const double* phi, const double* c_f,
                      const double* c_r, const double* rho, double dt_P, double* e) {
    __shared__ WalkX X;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const long long plane = (long long)ny * nz;
    const int i0 = (int)(blockIdx.x / w.tiles) * w.steps, tile = (int)(blockIdx.x % w.tiles);
    bool okd = X.fill(g, i0);
    const int lane = threadIdx.x & 31;
    const long long u = ((long long)tile * kWalkWarps + (threadIdx.x >> 5)) * 30 + lane - 1;
    if (u - lane + 1 >= plane) return;   // whole warps only: the others exchange
    const bool out = u >= 0 && u < plane && lane > 0 && lane < 31;
    const long long c0 = u < 0 ? 0 : u < plane ? u : plane - 1;
    const int j = (int)(c0 / nz), k = (int)(c0 - (long long)j * nz);
    const bool hy = j < ny - 1, ly = j != 0, hz = k < nz - 1, lz = k != 0;
    const double dy1 = hy ? g.dy[j + 1] : 1.0, dy2 = ly ? g.dy[j - 1] : 1.0;
    const double dz1 = hz ? g.dz[k + 1] : 1.0;
    const Divisor dy = divisor(g.dy[j]), dz = divisor(g.dz[k]), dt = divisor(dt_P);
    okd = okd && plain_positive(dy.b) && plain_positive(dz.b) && plain_positive(dt_P) && plain_positive(dy1) &&
          plain_positive(dy2) && plain_positive(dz1);
    long long t = (long long)i0 * plane + c0;
    double r = rho[t];
    bool ok0 = okd && plain_positive(r), okm = true;   // this cell's density; the face before
    Divisor rd = divisor(r);
    double ar = quotient(X.d[1], rd), q0 = 0.0, fx = 0.0;
    if (i0 != 0) {
        const double rm = rho[t - plane];
        q0 = qx[t - plane];
        okm = ok0 && plain_positive(rm) && plain_signed(q0);
        fx = harm_of(X.d[0] + X.d[1], quotient(X.d[0], divisor(rm)), ar);
    }
    const int steps = min(w.steps, nx - i0);
    for (int s = 0; s < steps; ++s, t += plane) {
        const bool hx = i0 + s < nx - 1, lx = i0 + s != 0;
        const double r1 = rho[hx ? t + plane : t], ra = rho[hy ? t + nz : t], rb = rho[ly ? t - nz : t];
        const double fm = fx, qm = q0, qa = qy[t], qb = qy[ly ? t - nz : t], qu = qz[t], qd = qz[lz ? t - 1 : t];
        q0 = qx[t];
        const double por = phi[t], cr = c_r[t], cf = c_f[t], dp = P[t] - Pn[t], W = WP[t];
        // the z face above, of this lane and of the one before
        const double zr = quotient(dz.b, rd);
        bool ok = ok0;
        const double zr1 = __shfl_down_sync(0xffffffffu, zr, 1);
        const double fz = harm_of(dz1 + dz.b, zr1, zr);
        const double fz0 = __shfl_up_sync(0xffffffffu, fz, 1);
        // the lanes beside: their densities (and the face of the one before)
        const unsigned good = __ballot_sync(0xffffffffu, ok);
        ok = ok && (!hz || (good >> ((lane + 1) & 31) & 1u)) && (!lz || (good >> ((lane + 31) & 31) & 1u));
        // the next x face
        const Divisor rd1 = divisor(r1);
        const bool ok1 = okd && plain_positive(r1);
        const double ar1 = quotient(X.d[s + 2], rd1);
        bool okx = ok0 && ok1 && plain_signed(q0);
        fx = harm_of(X.sum[s + 1].b, ar1, ar);
        ok = ok && okx && okm && plain_positive(ra) && plain_positive(rb) && plain_signed(qa) && plain_signed(qb) &&
             plain_signed(qu) && plain_signed(qd);
        const Divisor dx = X.own[s + 1];
        const double yr = quotient(dy.b, rd);
        const double fa = harm_of(dy1 + dy.b, quotient(dy1, divisor(ra)), yr);
        const double fb = harm_of(dy2 + dy.b, quotient(dy2, divisor(rb)), yr);
        double v = 0.0;
        if (hx) v -= (quotient_0(q0, dx) * fx);
        if (lx) v += (quotient_0(qm, dx) * fm);
        if (hy) v -= (quotient_0(qa, dy) * fa);
        if (ly) v += (quotient_0(qb, dy) * fb);
        if (hz) v -= (quotient_0(qu, dz) * fz);
        if (lz) v += (quotient_0(qd, dz) * fz0);
        const double st = ((1 - por) * cr + por * cf) * dp * r;
        ok = ok && plain_signed(st);
        v += (W + quotient_0(st, dt));
        if (out) e[t] = ok ? v : flow_error_cell(g, t, i0 + s, j, k, P, Pn, qx, qy, qz, WP, phi, c_f, c_r, rho, dt_P);
        okm = okx;
        r = r1;
        rd = rd1;
        ar = ar1;
        ok0 = ok1;
    }
}

// ---------------------------------------------------------------- reduces
enum RedOp { R_SUM = 0, R_MAX = 1, R_MIN = 2 };

__device__ __forceinline__ double red_init(int op) {
    return op == R_SUM ? 0.0 : (op == R_MAX ? -__longlong_as_double(0x7ff0000000000000LL)
                                            : __longlong_as_double(0x7ff0000000000000LL));
}
__device__ __forceinline__ double red_combine(int op, double a, double b) {
    return op == R_SUM ? a + b : (op == R_MAX ? nmax(a, b) : nmin(a, b));
}

template <int NT>
__device__ __forceinline__ double block_red(int op, double v, double* sh) {
    if (op == R_SUM) return block_sum<NT>(v, sh);
    if (op == R_MAX) return block_nmax<NT>(v, sh);
    return block_nmin<NT>(v, sh);
}

struct Ops {
    int op[4];
};

// Final pass: one block folds `nparts` partials per output (fixed order).
__global__ void finish_kernel(const double* parts, int nparts, int nout, Ops ops, double* out,
                              int post) {
    __shared__ double sh[kBlock / 32];
    // every output's loads before the first reduction
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[q] = red_init(ops.op[q]);
        if (q < nout)
#pragma unroll 4
            for (int b = threadIdx.x; b < nparts; b += kBlock) v[q] = red_combine(ops.op[q], v[q], parts[q * nparts + b]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q >= nout) break;
        double r = block_red<kBlock>(ops.op[q], v[q], sh);
        if (threadIdx.x == 0) out[q] = r;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (post == 1) {          // l2_norm: out = {sum d^2, sum old^2} -> l2
            double l2 = sqrt(out[0]) / sqrt(out[1] + 1e-200);
            out[0] = (l2 != l2) ? 1.0 : l2;
        } else if (post == 2) {   // CFL: out = {max x, max y, max z} -> dt_CFL
            out[0] = 0.9 / (out[0] + out[1] + out[2]);
        }
    }
}

__global__ void l2_partial_kernel(const double* New, const double* Old, long long n, double* parts) {
    __shared__ double sh[kBlock / 32];
    double s1 = 0.0, s2 = 0.0;
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < n;
         f += (long long)gridDim.x * blockDim.x) {
        const double d = New[f] - Old[f];
        s1 = s1 + d * d;
        s2 = s2 + Old[f] * Old[f];
    }
    double r1 = block_sum<kBlock>(s1, sh);
    double r2 = block_sum<kBlock>(s2, sh);
    if (threadIdx.x == 0) {
        parts[blockIdx.x] = r1;
        parts[gridDim.x + blockIdx.x] = r2;
    }
}

// dt_CFL (tse.py:1241-1246): element f of reshape(|qx|/phi, (ny,nz,nx)) / dx
// is divided by dx[f % nx]; likewise dy[f % ny]; qz uses dz[k].
// Bound: the divisions, then DRAM.  On large grids |q| / p / d is formed only
// where it can exceed the warp's maximum so far.  A product tells, with a margin
// for its rounding, where the maximum, p and d are positive and far from the ends
// of the exponent range (|q| / p may then round to nothing without reaching the
// maximum); with any other, and with NaN, the quotient is formed.  Of 160 us at
// 255 x 256 x 127 the arrays take 41; six divisions and two 64-bit remainders a
// cell took the rest.  Now 92.  Below kCflDirect cells a thread has too few cells
// for a maximum to save much, and the warp's agreement on it costs more (us,
// direct and not: 23 / 27 at 90^3, 29 / 34 at 128 x 128 x 100, 47 / 50 at 160 x
// 192 x 101, 56 / 59 at 200 x 190 x 101; 106 / 92-104 at 255 x 256 x 127).
constexpr long long kCflDirect = 4000000;
template <bool DIRECT>
struct CflMax {
    double m = -HUGE_VAL;   // the warp's, or the thread's
    __device__ __forceinline__ bool below(double q, double p, double d) const {
        return plain_positive(m) && plain_positive(p) && plain_positive(d) && q * (1.0 + 1e-12) < m * p * d;
    }
    __device__ __forceinline__ void take(double q, double p, double d, bool in) {
        if (DIRECT) {
            if (in) m = nmax(m, q / p / d);
            return;
        }
        const bool cand = in && !below(q, p, d);
        if (!__any_sync(0xffffffffu, cand)) return;
        double v = cand ? q / p / d : m;
        for (int o = 16; o > 0; o >>= 1) v = nmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        m = nmax(m, v);
    }
};
template <bool DIRECT>
__global__ void cfl_partial_kernel(TseGrid g, const double* qx, const double* qy, const double* qz,
                                   const double* phi, double* parts) {
    __shared__ double sh[kBlock / 32];
    const long long n = (long long)g.nx * g.ny * g.nz;
    const long long st = (long long)gridDim.x * blockDim.x, f0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    // f % nx, f % ny, f % nz, stepped along (st and f0 are below 2^32)
    const unsigned u = (unsigned)st, v = (unsigned)f0;
    const int ax = (int)(u % (unsigned)g.nx), ay = (int)(u % (unsigned)g.ny), az = (int)(u % (unsigned)g.nz);
    int ix = (int)(v % (unsigned)g.nx), iy = (int)(v % (unsigned)g.ny), iz = (int)(v % (unsigned)g.nz);
    CflMax<DIRECT> a, b, c;
    for (long long w0 = f0 - (threadIdx.x & 31), f = f0; w0 < n; w0 += st, f += st) {
        const bool in = f < n;
        const long long h = in ? f : n - 1;
        const double p = phi[h], x = fabs(qx[h]), y = fabs(qy[h]), z = fabs(qz[h]);
        a.take(x, p, g.dx[ix], in);
        b.take(y, p, g.dy[iy], in);
        c.take(z, p, g.dz[iz], in);
        ix += ax;
        iy += ay;
        iz += az;
        if (ix >= g.nx) ix -= g.nx;
        if (iy >= g.ny) iy -= g.ny;
        if (iz >= g.nz) iz -= g.nz;
    }
    double ra = block_nmax<kBlock>(a.m, sh);
    double rb = block_nmax<kBlock>(b.m, sh);
    double rc = block_nmax<kBlock>(c.m, sh);
    if (threadIdx.x == 0) {
        parts[blockIdx.x] = ra;
        parts[gridDim.x + blockIdx.x] = rb;
        parts[2 * gridDim.x + blockIdx.x] = rc;
    }
}

// explicit_C (tse.py:385-396); per-cell max over species, NaN propagating
struct SpeciesPtrs {
    const double* p[8];
};

__global__ void explicit_c_partial_kernel(TseGrid g, SpeciesPtrs D, int ns, const double* phi,
                                          double* parts) {
    __shared__ double sh[kBlock / 32];
    const long long n = (long long)g.nx * g.ny * g.nz;
    double m = 1e100;
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < n;
         f += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        decode(f, g.ny, g.nz, i, j, k);
        double dmax = D.p[0][f];
        for (int s = 1; s < ns; ++s) dmax = nmax(dmax, D.p[s][f]);
        const double dxi = g.dx[i], dyj = g.dy[j], dzk = g.dz[k];
        const double v = 0.45 * dmax / phi[f] / (1 / (dxi * dxi) + 1 / (dyj * dyj) + 1 / (dzk * dzk));
        m = pymin(m, v);
    }
    double r = block_nmin<kBlock>(m, sh);
    if (threadIdx.x == 0) parts[blockIdx.x] = r;
}

__global__ void stats_partial_kernel(const double* x, long long n, double* parts) {
    __shared__ double sh[kBlock / 32];
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    double s = 0.0, mx = -inf, mn = inf;
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < n;
         f += (long long)gridDim.x * blockDim.x) {
        const double v = x[f];
        s = s + v;
        mx = nmax(mx, v);
        mn = nmin(mn, v);
    }
    double r1 = block_sum<kBlock>(s, sh);
    double r2 = block_nmax<kBlock>(mx, sh);
    double r3 = block_nmin<kBlock>(mn, sh);
    if (threadIdx.x == 0) {
        parts[blockIdx.x] = r1;
        parts[gridDim.x + blockIdx.x] = r2;
        parts[2 * gridDim.x + blockIdx.x] = r3;
    }
}

// peclet_C (tse.py:331-354): non-boundary cells get |q| / max_s D * d (NaN
// when max_s D == 0); boundary cells keep the zero the reference's PeC array
// was initialised with.
__global__ void peclet_c_partial_kernel(TseGrid g, const double* qx, const double* qy,
                                        const double* qz, SpeciesPtrs Dx, SpeciesPtrs Dy,
                                        SpeciesPtrs Dz, int ns, const double* BC, double* parts) {
    __shared__ double sh[kBlock / 32];
    const long long n = (long long)g.nx * g.ny * g.nz;
    double a = 0.0, b = 0.0, c = 0.0;   // max over a zero-initialised array
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < n;
         f += (long long)gridDim.x * blockDim.x) {
        if (BC[f] == 0) {
            int i, j, k;
            decode(f, g.ny, g.nz, i, j, k);
            double mx = Dx.p[0][f], my = Dy.p[0][f], mz = Dz.p[0][f];
            for (int s = 1; s < ns; ++s) {
                mx = nmax(mx, Dx.p[s][f]);
                my = nmax(my, Dy.p[s][f]);
                mz = nmax(mz, Dz.p[s][f]);
            }
            a = nmax(a, mx != 0 ? fabs(qx[f]) / mx * g.dx[i] : nan);
            b = nmax(b, my != 0 ? fabs(qy[f]) / my * g.dy[j] : nan);
            c = nmax(c, mz != 0 ? fabs(qz[f]) / mz * g.dz[k] : nan);
        }
    }
    double ra = block_nmax<kBlock>(a, sh);
    double rb = block_nmax<kBlock>(b, sh);
    double rc = block_nmax<kBlock>(c, sh);
    if (threadIdx.x == 0) {
        parts[blockIdx.x] = ra;
        parts[gridDim.x + blockIdx.x] = rb;
        parts[2 * gridDim.x + blockIdx.x] = rc;
    }
}

// peclet_T (tse.py:357-383)
__global__ void peclet_t_partial_kernel(TseGrid g, const double* qx, const double* qy,
                                        const double* qz, const double* rho, const double* cp,
                                        const double* phi, const double* l_r, const double* l_f,
                                        const double* BT, double* parts) {
    __shared__ double sh[kBlock / 32];
    const long long n = (long long)g.nx * g.ny * g.nz;
    double a = 0.0, b = 0.0, c = 0.0;
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < n;
         f += (long long)gridDim.x * blockDim.x) {
        if (BT[f] == 0) {
            int i, j, k;
            decode(f, g.ny, g.nz, i, j, k);
            const double den = (1 - phi[f]) * l_r[f] + phi[f] * l_f[f];
            a = nmax(a, fabs(qx[f]) * rho[f] * cp[f] / den * g.dx[i]);
            b = nmax(b, fabs(qy[f]) * rho[f] * cp[f] / den * g.dy[j]);
            c = nmax(c, fabs(qz[f]) * rho[f] * cp[f] / den * g.dz[k]);
        }
    }
    double ra = block_nmax<kBlock>(a, sh);
    double rb = block_nmax<kBlock>(b, sh);
    double rc = block_nmax<kBlock>(c, sh);
    if (threadIdx.x == 0) {
        parts[blockIdx.x] = ra;
        parts[gridDim.x + blockIdx.x] = rb;
        parts[2 * gridDim.x + blockIdx.x] = rc;
    }
}

// Mass-balance totals in FP64 (cell volume V = dx dy dz):
//   water  sum phi rho V             species s  sum RC phi C_s V
//   heat   sum (phi rho cp_f + (1-phi) rho_r cp_r) T V
//   source rates  sum WP V, sum WC_s V, sum WT V
// out (per block partial q): 0 water, 1..ns species, ns+1 heat, ns+2 WP,
// ns+3..2ns+2 WC, 2ns+3 WT
struct MassArgs {
    const double *phi, *rho, *RC, *T, *cp_f, *rho_r, *cp_r, *WP, *WT;
    const double* C[8];
    const double* WC[8];
};

// Bound: DRAM.  One instance a species count, so the sums are registers: with
// a run-time count they were local memory, 431 us at 255 x 256 x 127 and two
// species, 141 now (13 arrays, 132 us).
template <int NS>
__global__ void __launch_bounds__(kBlock, 2) mass_partial_kernel(TseGrid g, MassArgs a, double* parts) {
    __shared__ double sh[kBlock / 32];
    const long long n = (long long)g.nx * g.ny * g.nz;
    constexpr int nq = 2 * NS + 4;
    double acc[nq];
#pragma unroll
    for (int q = 0; q < nq; ++q) acc[q] = 0.0;
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < n;
         f += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        decode(f, g.ny, g.nz, i, j, k);
        const double ph = a.phi[f], rho = a.rho[f], RC = a.RC[f], cf = a.cp_f[f], rr = a.rho_r[f], cr = a.cp_r[f],
                     T = a.T[f], WP = a.WP[f], WT = a.WT[f];
        double C[NS + 1], WC[NS + 1];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            C[s] = a.C[s][f];
            WC[s] = a.WC[s][f];
        }
        const double V = g.dx[i] * g.dy[j] * g.dz[k];
        acc[0] += ph * rho * V;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            acc[1 + s] += RC * ph * C[s] * V;
            acc[NS + 3 + s] += WC[s] * V;
        }
        acc[NS + 1] += (ph * rho * cf + (1 - ph) * rr * cr) * T * V;
        acc[NS + 2] += WP * V;
        acc[2 * NS + 3] += WT * V;
    }
#pragma unroll
    for (int q = 0; q < nq; ++q) {
        const double r = block_sum<kBlock>(acc[q], sh);
        if (threadIdx.x == 0) parts[q * gridDim.x + blockIdx.x] = r;
    }
}

// one block an output
__global__ void mass_finish_kernel(const double* parts, int nparts, double* out) {
    __shared__ double sh[kBlock / 32];
    double v = 0.0;
    for (int b = threadIdx.x; b < nparts; b += kBlock) v = v + parts[(size_t)blockIdx.x * nparts + b];
    const double r = block_sum<kBlock>(v, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = r;
}

// Declared linear EOS: rho = rho0 + a0*C[s0] + ... - tcoef*(T - T0)
struct EosLinear {
    const double* C[8];
    double a[8];
    int m;
    double rho0, tcoef, T0;
};

__global__ void eos_linear_kernel(EosLinear E, const double* T, double* rho, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double r = E.rho0;
    for (int q = 0; q < E.m; ++q) r = r + E.a[q] * E.C[q][t];
    r = r - E.tcoef * (T[t] - E.T0);
    rho[t] = r;
}

// Declared per-cell property forms (constant, fourth-order polynomial in T),
// optionally guarded: cells whose guard species equals guard_value keep their
// value, as `if C[s] != v:` in a config callback does.
struct EosForm {
    int kind;
    const double* guard;
    double guard_value;
    double c[5];
};

__global__ void eos_form_kernel(EosForm E, const double* T, double* out, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    if (E.guard && !(E.guard[t] != E.guard_value)) return;
    double r;
    if (E.kind == TSE_EOS_CONSTANT) {
        r = E.c[0];
    } else {
        // c[4] + c[3]*T + c[2]*T**2 + c[1]*T**3 + c[0]*T**4, left to right,
        // powers by repeated squaring: T**3 = T*(T*T), T**4 = (T*T)*(T*T) --
        // the products numba emits for a literal integer exponent
        const double x = T[t];
        const double x2 = x * x;
        const double x3 = x * x2;
        const double x4 = x2 * x2;
        r = E.c[4] + E.c[3] * x;
        r = r + E.c[2] * x2;
        r = r + E.c[1] * x3;
        r = r + E.c[0] * x4;
    }
    out[t] = r;
}

inline unsigned grid_for(long long n) {
    long long b = (n + kBlock - 1) / kBlock;
    return (unsigned)(b < 1 ? 1 : b);
}

inline unsigned red_blocks(long long n) {
    long long b = (n + kBlock - 1) / kBlock;
    if (b > kRedBlocks) b = kRedBlocks;
    return (unsigned)(b < 1 ? 1 : b);
}

// reduce workspace: up to 8 outputs x kRedBlocks partials
size_t reduce_ws_bytes() { return align256(sizeof(double) * 8 * kRedBlocks); }

static int finish(double* parts, unsigned nparts, int nout, const int* h_ops, double* out, int post,
                  void*, cudaStream_t s) {
    Ops ops;
    for (int q = 0; q < 4; ++q) ops.op[q] = q < nout ? h_ops[q] : 0;
    finish_kernel<<<1, kBlock, 0, s>>>(parts, (int)nparts, nout, ops, out, post);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

}  // namespace tse

using namespace tse;

extern "C" int32_t tse_compute_q(const TseGrid* grid, const double* P, const double* BP,
                                 const double* Kx, const double* Ky, const double* Kz, double* qx,
                                 double* qy, double* qz, const double* nue, const double* rho_f,
                                 void* stream) {
    if (!grid || !P || !BP || !Kx || !Ky || !Kz || !qx || !qy || !qz || !nue || !rho_f) return TSE_ERR_ARG;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    if (n <= 0) return TSE_ERR_ARG;
    if (n < kWalkCellsQ) {
        compute_q_cells_kernel<<<grid_for(n), kBlock, 0, (cudaStream_t)stream>>>(*grid, P, BP, Kx, Ky, Kz, qx,
                                                                                 qy, qz, nue, rho_f);
        return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
    }
    Walk w;
    if (!walk_of(*grid, 31, kWalkBlocksQ, w)) return TSE_ERR_LAUNCH;
    compute_q_kernel<<<w.blocks, kBlock, 0, (cudaStream_t)stream>>>(*grid, w, P, BP, Kx, Ky, Kz, qx, qy, qz,
                                                                  nue, rho_f);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

extern "C" int32_t tse_flow_error(const TseGrid* grid, const double* P, const double* Pn,
                                  const double* qx, const double* qy, const double* qz,
                                  const double* WP, const double* phi, const double* c_f,
                                  const double* c_r, const double* rho_f, double dt_P, double* e,
                                  void* stream) {
    if (!grid || !P || !Pn || !qx || !qy || !qz || !WP || !phi || !c_f || !c_r || !rho_f || !e)
        return TSE_ERR_ARG;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    if (n <= 0) return TSE_ERR_ARG;
    if (n < kWalkCellsE || grid->ny == 1) {
        flow_error_cells_kernel<<<grid_for(n), kBlock, 0, (cudaStream_t)stream>>>(
            *grid, P, Pn, qx, qy, qz, WP, phi, c_f, c_r, rho_f, dt_P, e);
        return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
    }
    const bool four = n >= kWalkCellsE4;
    Walk w;
    if (!walk_of(*grid, 30, four ? 4 : 3, w)) return TSE_ERR_LAUNCH;
    (four ? flow_error_kernel<4> : flow_error_kernel<3>)<<<w.blocks, kBlock, 0, (cudaStream_t)stream>>>(
        *grid, w, P, Pn, qx, qy, qz, WP, phi, c_f, c_r, rho_f, dt_P, e);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

extern "C" int32_t tse_l2_norm(const double* New, const double* Old, int64_t n, double* d_out,
                               void* ws, size_t ws_bytes, void* stream) {
    if (!New || !Old || !d_out || !ws || n <= 0) return TSE_ERR_ARG;
    if (ws_bytes < reduce_ws_bytes()) return TSE_ERR_WORKSPACE;
    cudaStream_t s = (cudaStream_t)stream;
    double* parts = (double*)ws;
    const unsigned nb = red_blocks(n);
    l2_partial_kernel<<<nb, kBlock, 0, s>>>(New, Old, n, parts);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    static const int ops[2] = {R_SUM, R_SUM};
    return finish(parts, nb, 2, ops, d_out, 1, ws, s);
}

extern "C" int32_t tse_dt_cfl(const TseGrid* grid, const double* qx, const double* qy,
                              const double* qz, const double* phi, double* d_out, void* ws,
                              size_t ws_bytes, void* stream) {
    if (!grid || !qx || !qy || !qz || !phi || !d_out || !ws) return TSE_ERR_ARG;
    if (ws_bytes < reduce_ws_bytes()) return TSE_ERR_WORKSPACE;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    if (n <= 0) return TSE_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    double* parts = (double*)ws;
    const unsigned nb = red_blocks(n);
    if (n < kCflDirect)
        cfl_partial_kernel<true><<<nb, kBlock, 0, s>>>(*grid, qx, qy, qz, phi, parts);
    else
        cfl_partial_kernel<false><<<nb, kBlock, 0, s>>>(*grid, qx, qy, qz, phi, parts);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    static const int ops[3] = {R_MAX, R_MAX, R_MAX};
    return finish(parts, nb, 3, ops, d_out, 2, ws, s);
}

extern "C" int32_t tse_explicit_C(const TseGrid* grid, const double* const* h_D, int32_t nspec,
                                  const double* phi, double* d_out, void* ws, size_t ws_bytes,
                                  void* stream) {
    if (!grid || !h_D || nspec < 1 || nspec > 8 || !phi || !d_out || !ws) return TSE_ERR_ARG;
    if (ws_bytes < reduce_ws_bytes()) return TSE_ERR_WORKSPACE;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    cudaStream_t s = (cudaStream_t)stream;
    SpeciesPtrs D;
    for (int q = 0; q < 8; ++q) D.p[q] = q < nspec ? h_D[q] : nullptr;
    double* parts = (double*)ws;
    const unsigned nb = red_blocks(n);
    explicit_c_partial_kernel<<<nb, kBlock, 0, s>>>(*grid, D, nspec, phi, parts);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    static const int ops[1] = {R_MIN};
    return finish(parts, nb, 1, ops, d_out, 0, ws, s);
}

extern "C" int32_t tse_field_stats(const double* x, int64_t n, double* d_out, void* ws,
                                   size_t ws_bytes, void* stream) {
    if (!x || n <= 0 || !d_out || !ws) return TSE_ERR_ARG;
    if (ws_bytes < reduce_ws_bytes()) return TSE_ERR_WORKSPACE;
    cudaStream_t s = (cudaStream_t)stream;
    double* parts = (double*)ws;
    const unsigned nb = red_blocks(n);
    stats_partial_kernel<<<nb, kBlock, 0, s>>>(x, n, parts);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    static const int ops[3] = {R_SUM, R_MAX, R_MIN};
    return finish(parts, nb, 3, ops, d_out, 0, ws, s);
}

extern "C" int32_t tse_peclet_C(const TseGrid* grid, const double* qx, const double* qy,
                                const double* qz, const double* const* h_Dx,
                                const double* const* h_Dy, const double* const* h_Dz, int32_t ns,
                                const double* BC, double* d_out, void* ws, size_t ws_bytes,
                                void* stream) {
    if (!grid || !qx || !qy || !qz || !h_Dx || !h_Dy || !h_Dz || ns < 1 || ns > 8 || !BC || !d_out || !ws)
        return TSE_ERR_ARG;
    if (ws_bytes < reduce_ws_bytes()) return TSE_ERR_WORKSPACE;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    cudaStream_t s = (cudaStream_t)stream;
    SpeciesPtrs X, Y, Z;
    for (int q = 0; q < 8; ++q) {
        X.p[q] = q < ns ? h_Dx[q] : nullptr;
        Y.p[q] = q < ns ? h_Dy[q] : nullptr;
        Z.p[q] = q < ns ? h_Dz[q] : nullptr;
    }
    double* parts = (double*)ws;
    const unsigned nb = red_blocks(n);
    peclet_c_partial_kernel<<<nb, kBlock, 0, s>>>(*grid, qx, qy, qz, X, Y, Z, ns, BC, parts);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    static const int ops[3] = {R_MAX, R_MAX, R_MAX};
    return finish(parts, nb, 3, ops, d_out, 0, ws, s);
}

extern "C" int32_t tse_peclet_T(const TseGrid* grid, const double* qx, const double* qy,
                                const double* qz, const double* rho_f, const double* cp_f,
                                const double* phi, const double* l_r, const double* l_f,
                                const double* BT, double* d_out, void* ws, size_t ws_bytes,
                                void* stream) {
    if (!grid || !qx || !qy || !qz || !rho_f || !cp_f || !phi || !l_r || !l_f || !BT || !d_out || !ws)
        return TSE_ERR_ARG;
    if (ws_bytes < reduce_ws_bytes()) return TSE_ERR_WORKSPACE;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    cudaStream_t s = (cudaStream_t)stream;
    double* parts = (double*)ws;
    const unsigned nb = red_blocks(n);
    peclet_t_partial_kernel<<<nb, kBlock, 0, s>>>(*grid, qx, qy, qz, rho_f, cp_f, phi, l_r, l_f, BT,
                                                 parts);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    static const int ops[3] = {R_MAX, R_MAX, R_MAX};
    return finish(parts, nb, 3, ops, d_out, 0, ws, s);
}

extern "C" int32_t tse_mass_totals(const TseGrid* grid, const double* phi, const double* rho_f,
                                   const double* RC, const double* const* h_C,
                                   const double* const* h_WC, int32_t nspec, const double* T,
                                   const double* cp_f, const double* rho_r, const double* cp_r,
                                   const double* WP, const double* WT, double* d_out, void* ws,
                                   size_t ws_bytes, void* stream) {
    if (!grid || !phi || !rho_f || !RC || !T || !cp_f || !rho_r || !cp_r || !WP || !WT || !d_out ||
        !ws || nspec < 0 || nspec > 8 || (nspec > 0 && (!h_C || !h_WC)))
        return TSE_ERR_ARG;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    const int nq = 2 * nspec + 4;
    const unsigned nb = std::min(red_blocks(n), 256u);   // nq nb partials fit the workspace
    if (ws_bytes < reduce_ws_bytes()) return TSE_ERR_WORKSPACE;
    MassArgs a;
    a.phi = phi;
    a.rho = rho_f;
    a.RC = RC;
    a.T = T;
    a.cp_f = cp_f;
    a.rho_r = rho_r;
    a.cp_r = cp_r;
    a.WP = WP;
    a.WT = WT;
    for (int s = 0; s < 8; ++s) {
        a.C[s] = s < nspec ? h_C[s] : nullptr;
        a.WC[s] = s < nspec ? h_WC[s] : nullptr;
    }
    cudaStream_t s = (cudaStream_t)stream;
    double* parts = (double*)ws;
    using Kernel = void (*)(TseGrid, MassArgs, double*);
    static const Kernel kernels[9] = {mass_partial_kernel<0>, mass_partial_kernel<1>, mass_partial_kernel<2>,
                                      mass_partial_kernel<3>, mass_partial_kernel<4>, mass_partial_kernel<5>,
                                      mass_partial_kernel<6>, mass_partial_kernel<7>, mass_partial_kernel<8>};
    kernels[nspec]<<<nb, kBlock, 0, s>>>(*grid, a, parts);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    mass_finish_kernel<<<nq, kBlock, 0, s>>>(parts, (int)nb, d_out);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

extern "C" int32_t tse_eos_linear(const TseGrid* grid, const double* const* h_C,
                                  const int32_t* h_sidx, const double* h_coef, int32_t m,
                                  const double* T, double rho0, double tcoef, double T0,
                                  double* rho_f, void* stream) {
    if (!grid || !T || !rho_f || m < 0 || m > 8 || (m > 0 && (!h_C || !h_sidx || !h_coef)))
        return TSE_ERR_ARG;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    EosLinear E;
    for (int q = 0; q < 8; ++q) {
        E.C[q] = q < m ? h_C[h_sidx[q]] : nullptr;
        E.a[q] = q < m ? h_coef[q] : 0.0;
    }
    E.m = m;
    E.rho0 = rho0;
    E.tcoef = tcoef;
    E.T0 = T0;
    eos_linear_kernel<<<grid_for(n), kBlock, 0, (cudaStream_t)stream>>>(E, T, rho_f, n);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

extern "C" int32_t tse_eos_form(const TseGrid* grid, const TseEosForm* form, const double* T,
                                const double* guard, double* out, void* stream) {
    if (!grid || !form || !out) return TSE_ERR_ARG;
    if (form->kind != TSE_EOS_CONSTANT && form->kind != TSE_EOS_POLY4_T) return TSE_ERR_ARG;
    if (form->kind == TSE_EOS_POLY4_T && !T) return TSE_ERR_ARG;
    const long long n = (long long)grid->nx * grid->ny * grid->nz;
    if (n <= 0) return TSE_ERR_ARG;
    EosForm E;
    E.kind = form->kind;
    E.guard = guard;
    E.guard_value = form->guard_value;
    for (int q = 0; q < 5; ++q) E.c[q] = form->coef[q];
    eos_form_kernel<<<grid_for(n), kBlock, 0, (cudaStream_t)stream>>>(E, T, out, n);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}
