// The FP64 persistent solve of a grid whose solver state fits in shared
// memory: rb_solve_kernel's loop -- same checks, dt growth and halving, same
// per-cell arithmetic operation for operation (the forms' update_with) -- with
// a block's coefficients, flags and both colours of the solution in shared
// memory for the whole solve (tse_resident.cuh has the tiling and the edge
// exchange).  The per-cell values are identical to rb_solve_kernel's; only the
// grouping of the L2 sums of the convergence check differs.  The last act of
// the kernel is the natural-layout result.
//
// Bound: an iteration is two exchanges (about 1,200 clocks each through L2,
// 500 in a cluster) and two passes over the tile, whose vector loads from
// shared memory (19 16-byte ones for two cells) and divisions set the time of
// larger tiles.  Measured against the staged kernel, us per iteration of whole
// pressure solves (B200): 60 x 1 x 30 9.2 -> 1.9, 16^3 13-15 -> 2.2, 24^3
// 13-15 -> 2.4, 48^3 15.9 -> 3.5, 63 x 57 x 41 15.7 -> 4.4, 60^3 15.9 -> 4.5.
// A group's arrays lie side by side (immediate offsets; compile-time switches):
// with one array after another, 24^3 took 2.9 and 63 x 57 x 41 4.8.
#pragma once

#include "tse_resident.cuh"
#include "tse_rbsolve.cuh"

namespace tse {

constexpr int kXResVals = 2;        // doubles a group
constexpr int kXResThreads = 512;
struct XResCtl {
    ResMem mem;
    double* out;   // natural layout
};

// shared memory: two colours of padded groups; per colour and group its nst
// arrays, side by side; a group word and a flag word a group; the edge groups'
// records and places
inline int x_res_smem(const ResPlan& P, int nst) {
    const long long b = 2LL * P.pad * 16 + (long long)P.groups * (32LL * nst + 8) + ((P.halo * 6 + 15) & ~15);
    return b > (1 << 30) ? (1 << 30) : (int)b;
}

template <class Form, bool G1, bool G2, int COL, int MODE>
__device__ __forceinline__ void x_res_sweep(const Form& F, int groups, const double2* __restrict__ sa,
                                            const unsigned* sf,
                                            const unsigned* sw_word, double2* sw, const double2* sq,
                                            uint64_t* recs, int plane, int rrow, int rbase, unsigned tag,
                                            const ResPeers& peers, int dxp, int dyp, bool check, double& d2,
                                            double& o2) {
    for (int u = threadIdx.x; u < groups; u += kXResThreads) {
        const unsigned f = sw_word[u];
        const unsigned fl = sf[u] >> (16 * COL);
        const int p = f & 0xffffu;
        const bool odd = (((f >> 16) & 1u) ^ COL) != 0;
        constexpr int kNst = Form::template res_arrays<G1, G2>();
        const double2* a = sa + u * kNst;
        double2 v[Form::kCoef];
#pragma unroll
        for (int k = 0; k < Form::kCoef; ++k) {
            const int at = Form::template res_slot<G1, G2>(k);
            v[k] = at >= 0 ? a[at] : make_double2(0.0, 0.0);
        }
        const double2 old = sw[p];
        const double2 xp = sq[p + dxp], xm = sq[p - dxp], yp = sq[p + dyp], ym = sq[p - dyp], o = sq[p];
        // odd cells have k + 1 a place further and k - 1 at their own, even
        // cells k + 1 at their own and k - 1 a place before
        const double e = reinterpret_cast<const double*>(sq + p)[odd ? 2 : -1];
        const double z0 = odd ? o.x : e, z1 = odd ? o.y : o.x, z2 = odd ? e : o.y;
        // both cells' chains of dependent operations run side by side; an
        // inactive cell's result is dropped (it is kept as 1 / 1: a division
        // of or by zero would take its slow path)
        const double ux = F.update_with([&](int k) { return v[k].x; },
                                        [&](int q) {
                                            return q == 0 ? xp.x : q == 1 ? xm.x : q == 2 ? yp.x
                                                 : q == 3 ? ym.x : q == 4 ? z1 : z0;
                                        },
                                        (uint8_t)(fl & 0xffu), old.x);
        const double uy = F.update_with([&](int k) { return v[k].y; },
                                        [&](int q) {
                                            return q == 0 ? xp.y : q == 1 ? xm.y : q == 2 ? yp.y
                                                 : q == 3 ? ym.y : q == 4 ? z2 : z1;
                                        },
                                        (uint8_t)((fl >> 8) & 0xffu), old.y);
        const double2 xn = make_double2((fl & F_ACTIVE) ? ux : old.x, ((fl >> 8) & F_ACTIVE) ? uy : old.y);
        sw[p] = xn;
        if (f & RS_SHARED) {
            const uint64_t a = __double_as_longlong(xn.x), b = __double_as_longlong(xn.y);
            if (MODE == RES_CLUSTER)
                peers.publish(f, sw + p, (unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
            else
                res_publish(recs, plane, p + (int)(f >> 24) * rrow + rbase, (unsigned)a, (unsigned)(a >> 32),
                            (unsigned)b, (unsigned)(b >> 32), tag);
        }
        if (check) {
            o2 = o2 + old.x * old.x;
            o2 = o2 + old.y * old.y;
            // an inactive cell's difference is 0
            const double dx = xn.x - old.x, dy = xn.y - old.y;
            if (fl & F_ACTIVE) d2 = d2 + dx * dx;
            if ((fl >> 8) & F_ACTIVE) d2 = d2 + dy * dy;
        }
    }
}

template <class Form, bool G1, bool G2, int MODE>
__global__ void __launch_bounds__(kXResThreads, 1)
    rb_resident_kernel(Form Fr, SolveCtl c, ResPlan P, XResCtl w) {
    constexpr int NT = kXResThreads;
    constexpr int kNst = Form::template res_arrays<G1, G2>();
    const Form F = Fr.template res_form<G1, G2>();
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ ResSumShared sum;
    __shared__ int s_err;
    const unsigned nb = gridDim.x, b = blockIdx.x;
    const int tid = threadIdx.x;
    const int nx = c.L.nx, ny = c.L.ny, nz = c.L.nz, H = c.L.H;
    ResTile T;
    T.init(c.L, P, (int)b);
    const int groups = T.groups;
    double2* s0 = reinterpret_cast<double2*>(res_smem);
    double2* s1 = s0 + P.pad;
    double2* sa = s1 + P.pad;                       // colour 0's arrays, then colour 1's
    double2* sb = sa + (size_t)kNst * P.groups;
    unsigned* word = reinterpret_cast<unsigned*>(sb + (size_t)kNst * P.groups);
    unsigned* flag = word + P.groups;
    int* hrec = reinterpret_cast<int*>(flag + P.groups);
    unsigned short* hp = reinterpret_cast<unsigned short*>(hrec + P.halo);
    volatile int* err = &s_err;
    const int nh = nb > 1 ? T.halo_groups(nx) : 0;
    for (int h = tid; h < nh; h += NT) {
        int rec, pp;
        T.halo(h, nx, rec, pp);
        hrec[h] = rec;
        hp[h] = (unsigned short)pp;
    }
    if (tid == 0) s_err = 0;
    const int rrow = T.rec_row(), rbase = T.rec_base();
    const int dxp = T.pitch * T.Hg, dyp = T.Hg;
    ResPeers peers = {0u, 0u, 0u, 0u};
    if (MODE == RES_CLUSTER) peers.init(T, c.L, P, (int)b, res_smem);
    for (int q = tid; q < 2 * P.pad; q += NT) s0[q] = make_double2(0.0, 0.0);
    for (int u = tid; u < groups; u += NT) word[u] = res_group_word(T, u, nx, nb > 1);

    unsigned tag = 0, sums = 0, bars = 0;
    double t = 0.0, dt = c.dt, diff = 1e100;
    int converged = 0, num_it = 0, num_sub_it = 0, halvings = 0, fail = 0, nev = 0;
    const bool leader = b == 0 && tid == 0;

    for (;;) {
        __syncthreads();   // the group words and edge lists
        // ---- the tile's state from the workspace (at the start and after a
        // dt halving); the rings too, so the first half-sweeps need no exchange
        for (int u = tid; u < 2 * groups; u += NT) {
            const int col = u >= groups, v = u - col * groups;
            int ci, cj, g;
            T.decode(v, ci, cj, g);
            const long long m = (long long)T.column(ci, cj) * H + 2 * g;
            const bool two = 2 * g + 1 < H;
            const double* arr = col ? F.arr[1] : F.arr[0];
            const double* x = (col ? c.X[1] : c.X[0]) + m;
            (col ? s1 : s0)[T.p(ci, cj, g)] = make_double2(__ldcg(x), two ? __ldcg(x + 1) : 0.0);
            const uint8_t* f = (col ? c.mask[1] : c.mask[0]) + m;
            const unsigned bits = (unsigned)f[0] | (two ? (unsigned)f[1] << 8 : 0u);
            reinterpret_cast<unsigned short*>(flag + v)[col] = (unsigned short)bits;
#pragma unroll
            for (int k = 0; k < Form::kCoef; ++k) {
                const int at = Form::template res_slot<G1, G2>(k);
                if (at < 0) continue;
                const double* a = arr + (long long)k * c.Ncal + m;
                double2 d = make_double2(__ldcg(a), two ? __ldcg(a + 1) : 0.0);
                if (k == Form::kDen || k == Form::kRhs) {
                    if (!(bits & F_ACTIVE)) d.x = 1.0;
                    if (!((bits >> 8) & F_ACTIVE)) d.y = 1.0;
                }
                (col ? sb : sa)[v * kNst + at] = d;
            }
        }
        for (int h = tid; h < nh; h += NT) {
            const int column = hrec[h] / T.Hg, g = hrec[h] - column * T.Hg;
            const long long m = (long long)column * H + 2 * g;
            const bool two = 2 * g + 1 < H;
            for (int col = 0; col < 2; ++col) {
                const double* x = (col ? c.X[1] : c.X[0]) + m;
                (col ? s1 : s0)[hp[h]] = make_double2(__ldcg(x), two ? __ldcg(x + 1) : 0.0);
            }
        }
        bool fresh = true, halved = false, ok = true;
        while (!converged) {
            num_it += 1;
            num_sub_it += 1;
            double d2 = 0.0, o2 = 0.0;
            const bool check = c.pressure_schedule ? (num_it < 50 || num_it % 10 == 0) : true;
            if (MODE == RES_CLUSTER) {
                cluster_sync();
            } else {
                if (!fresh)
                    res_poll<NT>(w.mem.recs[1], w.mem.plane, tag, reinterpret_cast<uint4*>(s1), hrec, hp, nh,
                                 c.bar, err);
                __syncthreads();
            }
            fresh = false;
            x_res_sweep<Form, G1, G2, 0, MODE>(F, groups, sa, flag, word, s0, s1, w.mem.recs[0], w.mem.plane, rrow,
                                       rbase, ++tag, peers, dxp, dyp, check, d2, o2);
            if (MODE == RES_CLUSTER) {
                cluster_sync();
            } else {
                res_poll<NT>(w.mem.recs[0], w.mem.plane, tag, reinterpret_cast<uint4*>(s0), hrec, hp, nh, c.bar,
                             err);
                __syncthreads();
            }
            x_res_sweep<Form, G1, G2, 1, MODE>(F, groups, sb, flag, word, s1, s0, w.mem.recs[1], w.mem.plane, rrow,
                                       rbase, ++tag, peers, dxp, dyp, check, d2, o2);
            diff = 1e100;
            if (check) {
                // a poll of this block that ran out shows here
                ok = res_team_sum<NT, MODE>(d2, o2, sum, w.mem.slots, nb, b, sums++, c.bar, err);
                if (!ok) break;
                const double l2 = sqrt(d2) / sqrt(o2 + 1e-200);
                diff = (l2 != l2) ? 1.0 : l2;
            }
            if (diff < c.conv || c.stop_on_first) {
                converged = 1;
                t += dt;
                if (num_sub_it < c.max_it / 2.0) dt = pymin(dt * c.inc_it, c.max_dt);
            } else {
                if (num_sub_it >= c.max_it) {
                    if (leader && nev < 8) {
                        c.status->ev_it[nev] = num_it;
                        c.status->ev_dt[nev] = dt;
                        c.status->ev_diff[nev] = diff;
                    }
                    nev += 1;
                    dt = dt / 2;
                    num_sub_it = 0;
                    halvings += 1;
                    halved = true;
                }
                if (halved || dt <= c.min_dt) break;
            }
        }
        // the block's values are in shared memory, and no block still writes
        // into another's rings
        if (MODE == RES_CLUSTER)
            cluster_sync();
        else
            __syncthreads();
        if (!ok || *err) { fail = 1; break; }
        const bool last = converged || dt <= c.min_dt;
        if (halved || last) {
            for (int u = tid; u < 2 * groups; u += NT) {
                const int col = u >= groups;
                int ci, cj, g;
                T.decode(u - col * groups, ci, cj, g);
                const double2 s = (col ? s1 : s0)[T.p(ci, cj, g)];
                const int i = T.i0 + ci, j = T.j0 + cj;
                for (int q = 0; q < 2 && 2 * g + q < H; ++q) {
                    const long long m = (long long)T.column(ci, cj) * H + 2 * g + q;
                    double x = q ? s.y : s.x;
                    if (halved) {
                        F.reassemble(col, m, dt);
                        x = (col ? c.X[1] : c.X[0])[m];
                    }
                    const int z = 2 * (2 * g + q) + ((i + j + col) & 1);
                    if (last && z < nz) w.out[((long long)i * ny + j) * nz + z] = x;
                }
            }
        }
        if (last) break;
        // the reset values are read by the neighbours' rings
        if (MODE == RES_CLUSTER) {
            cluster_sync();
        } else if (nb > 1) {
            if (!count_sync(w.mem.counter, ++bars * nb, c.bar)) { fail = 1; break; }
        }
    }
    bool failed = fail != 0;
    if (res_last<MODE>(w.mem.leavers, nb, b, failed)) {
        TseSolveStatus* s = c.status;
        s->t = t;
        s->dt = dt;
        s->diff = diff;
        s->converged = converged && !failed;
        s->num_it = num_it;
        s->num_sub_it = num_sub_it;
        s->halvings = halvings;
        s->error = failed ? TSE_STATUS_BARRIER_TIMEOUT : TSE_STATUS_OK;
        s->n_events = nev < 8 ? nev : 8;
        s->cycles = 0;
        s->sweep = TSE_SWEEP_RESIDENT;
    }
}

constexpr int kXResCluster = 16;
// Groups one block takes by itself.  Measured, us per iteration in one block
// and in a cluster of 16: 128 groups 1.67 and 2.08, 256 and 480 groups the same
// (2.15, 1.87 both ways); a block leaves the other SMs to other streams.
constexpr int kXResSingle = 480;
// the largest grid (cells per colour) a workspace carries exchange memory for
constexpr long long kXResMaxNc = 160LL * 1152;
inline size_t x_res_bytes(const Layout& L) {
    return L.Nc <= kXResMaxNc ? 256 + res_mem_bytes(L, kXResVals) : 0;
}

template <class Form, bool G1, bool G2>
static const void* x_resident_fn_mode(bool cluster) {
    return cluster ? (const void*)rb_resident_kernel<Form, G1, G2, RES_CLUSTER>
                   : (const void*)rb_resident_kernel<Form, G1, G2, RES_GRID>;
}
template <class Form>
static const void* x_resident_fn(bool g1, bool g2, bool cluster) {
    return g1 ? (g2 ? x_resident_fn_mode<Form, true, true>(cluster) : x_resident_fn_mode<Form, true, false>(cluster))
              : (g2 ? x_resident_fn_mode<Form, false, true>(cluster)
                    : x_resident_fn_mode<Form, false, false>(cluster));
}

// Run the whole solve resident, writing `out`: TSE_OK, TSE_ERR_LAUNCH, or 1
// when a streaming kernel should run.
template <class Form>
static int launch_rb_resident(const Form& F, SolveCtl& ctl, void* tail, size_t tail_bytes, double* out,
                              cudaStream_t stream) {
    if (ctl.L.Nc > kXResMaxNc || tail_bytes < x_res_bytes(ctl.L)) return 1;
    int dev = 0, sms = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    const bool g1 = F.res_g1(), g2 = F.res_g2();
    const int nst = g1 ? (g2 ? Form::template res_arrays<true, true>() : Form::template res_arrays<true, false>())
                       : (g2 ? Form::template res_arrays<false, true>() : Form::template res_arrays<false, false>());
    const int room = optin - 2048;
    auto smem = [nst](const ResPlan& P) { return x_res_smem(P, nst); };
    auto threads = [](const ResPlan&) { return kXResThreads; };
    ResPlan P;
    const void* fn = nullptr;
    bool cluster = false;
    // one block, one cluster, the whole GPU: the first that holds the grid
    for (int form = 0; form < 3 && !fn; ++form) {
        cluster = form == 1;
        const int maxb = form == 0 ? 1 : form == 1 ? kXResCluster : sms < kResMaxBlocks ? sms : kResMaxBlocks;
        if (!res_plan(ctl.L, kXResVals, maxb, form == 0 ? kXResSingle : 65535, room, smem, threads, false, P))
            continue;
        if (P.nb == 1) cluster = false;
        fn = x_resident_fn<Form>(g1, g2, cluster);
        if (!res_can_launch(fn, P, kXResThreads, room, cluster)) fn = nullptr;
    }
    if (!fn) return 1;
    char* base = (char*)(((uintptr_t)tail + 255) & ~(uintptr_t)255);
    XResCtl w;
    w.mem = res_mem(base, ctl.L, kXResVals);
    w.out = out;
    // tags count from 1
    if (!cluster && P.nb > 1 && cudaMemsetAsync(base, 0, res_mem_bytes(ctl.L, kXResVals), stream) != cudaSuccess)
        return TSE_ERR_LAUNCH;
    void* args[] = {(void*)&F, (void*)&ctl, (void*)&P, (void*)&w};
    return res_launch(fn, P, kXResThreads, cluster, args, stream) ? TSE_OK : TSE_ERR_LAUNCH;
}

}  // namespace tse
