// The mixed-precision solve of a grid whose FP32 state fits on the chip: one
// cooperative launch runs every correction cycle, with the records of a
// block's cells in its threads' registers and both colours' corrections in
// shared memory (see tse_resident.cuh for the tiling and the edge exchange).
//
// The iterations are dc_sweep_kernel's, cell update for cell update (relax()'s
// operations in relax()'s order), so the corrections are the same bits as the
// staged and the plain sweep's; a cycle's end (x += d, the FP64 residual, the
// dt halving) is done by the same kernel with the steps of tse_dc.cu, and its
// last one writes the natural-layout result and the status record.  Only the
// grouping of the check sums differs.
//
// Bound: an iteration is two exchanges (about 1,200 clocks each through L2,
// 500 in a cluster) and two passes over the tile (370 clocks for one group a
// thread, 1,200 for two); DRAM is idle.  Measured against the staged sweep, us
// per iteration with everything in the call (B200): 24^3 6.6 -> 1.6 (cluster),
// 33 x 29 x 31 6.9 -> 1.9, 64^3 7.1 -> 2.7, 96^3 9.8 -> 3.3, 100 x 90 x 81
// 9.3 -> 4.4.  Records in registers, 16-byte groups: with single cells a thread
// executed four times the instructions (96^3: 6.9 us).
#pragma once

#include "tse_dc.cuh"
#include "tse_resident.cuh"

namespace tse {

constexpr int kDcResVals = 4;   // floats a group

// shared memory of a plan: two colours of padded corrections, the edge
// groups' records and places
inline int dc_res_smem(const ResPlan& P) { return 2 * P.pad * 16 + ((P.halo * 6 + 15) & ~15); }

// Half-sweep of colour COL over a thread's NG groups (group g of a thread is
// the tile's group u = tid + g * NT, of both colours).
template <int NG, int COL, int MODE>
__device__ __forceinline__ void dc_res_sweep(const float (&k)[2][NG][4][6], const float (&r)[2][NG][4],
                                             const unsigned (&pf)[NG], float4* sw, const float4* sq,
                                             uint64_t* recs, int plane, int rrow, int rbase, unsigned tag,
                                             const ResPeers& peers, int dxp, int dyp, float sor, bool check,
                                             float& d2, float& dd) {
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        unsigned f = pf[g];
        // opaque to the compiler: addresses formed from it are not kept in
        // registers over the iterations in place of the records
        asm volatile("" : "+r"(f));
        if (f & RS_USED) {
            const int p = f & 0xffffu;
            const bool odd = (((f >> 16) & 1u) ^ COL) != 0;
            const float4 old4 = sw[p];
            const float4 xp = sq[p + dxp], xm = sq[p - dxp], yp = sq[p + dyp], ym = sq[p - dyp];
            const float4 o = sq[p];
            // odd cells have k + 1 a place further and k - 1 at their own,
            // even cells k + 1 at their own and k - 1 a place before
            const float e = reinterpret_cast<const float*>(sq + p)[odd ? 4 : -1];
            const float z[5] = {odd ? o.x : e, odd ? o.y : o.x, odd ? o.z : o.y, odd ? o.w : o.z,
                                odd ? e : o.w};
            const float vxp[4] = {xp.x, xp.y, xp.z, xp.w}, vxm[4] = {xm.x, xm.y, xm.z, xm.w};
            const float vyp[4] = {yp.x, yp.y, yp.z, yp.w}, vym[4] = {ym.x, ym.y, ym.z, ym.w};
            const float old[4] = {old4.x, old4.y, old4.z, old4.w};
            float na[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float* kk = k[COL][g][q];
                float acc = r[COL][g][q];
                acc = fmaf(kk[0], vxp[q], acc);
                acc = fmaf(kk[1], vxm[q], acc);
                acc = fmaf(kk[2], vyp[q], acc);
                acc = fmaf(kk[3], vym[q], acc);
                acc = fmaf(kk[4], z[q + 1], acc);
                acc = fmaf(kk[5], z[q], acc);
                na[q] = fmaf(sor, acc - old[q], old[q]);
            }
            sw[p] = make_float4(na[0], na[1], na[2], na[3]);
            if (f & RS_SHARED) {
                const unsigned a0 = __float_as_uint(na[0]), a1 = __float_as_uint(na[1]),
                               a2 = __float_as_uint(na[2]), a3 = __float_as_uint(na[3]);
                if (MODE == RES_CLUSTER)
                    peers.publish(f, sw + p, a0, a1, a2, a3);
                else
                    res_publish(recs, plane, p + (int)(f >> 24) * rrow + rbase, a0, a1, a2, a3, tag);
            }
            if (check) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float ch = na[q] - old[q];
                    d2 = fmaf(ch, ch, d2);
                    dd = fmaf(na[q], na[q], dd);
                }
            }
        }
    }
}

struct DcResCtl {
    ResMem mem;
    int nparts;   // x^2 partials the setup wrote
    double dt;
};

template <class Form, int NT, int NG, int MODE>
__global__ void __launch_bounds__(NT, 1)
    dc_resident_kernel(Form F, DcCtl c, ResPlan P, DcResCtl w, double* X_out, TseSolveStatus* status) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ ResSumShared sum;
    __shared__ int s_err;
    const unsigned nb = gridDim.x, b = blockIdx.x;
    const int tid = threadIdx.x;
    const int nx = c.L.nx, ny = c.L.ny, nz = c.L.nz, H = c.L.H;
    float4* s0 = reinterpret_cast<float4*>(res_smem);
    float4* s1 = s0 + P.pad;
    int* hrec = reinterpret_cast<int*>(s1 + P.pad);
    unsigned short* hp = reinterpret_cast<unsigned short*>(hrec + P.halo);
    volatile int* err = &s_err;
    ResTile T;
    T.init(c.L, P, (int)b);
    const int nh = MODE == RES_GRID && nb > 1 ? T.halo_groups(nx) : 0;
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
    unsigned pf[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) pf[g] = res_group_word(T, tid + g * NT, nx, nb > 1);
    // x^2 of the initial iterate from the setup's partials, the same bits in
    // every block
    double x2 = 0.0, unused = 0.0;
    for (int q = tid; q < w.nparts; q += NT) x2 = x2 + c.partials[q];
    __syncthreads();
    res_team_sum<NT, RES_GRID>(x2, unused, sum, nullptr, 1u, 0u, 0u, c.bar, err);   // this block alone
    __syncthreads();

    const float sor = c.sor;
    unsigned tag = 0, sums = 0, bars = 0;
    double t = 0.0, dt = w.dt, diff = 1e100;
    int num_it = 0, num_sub_it = 0, halvings = 0, nev = 0, cycles = 1, event = EV_ERROR;
    const bool leader = b == 0 && tid == 0;

    for (;;) {
        // ---- a correction cycle: the records and r' of the thread's cells
        float k[2][NG][4][6], r[2][NG][4];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            int ci = 0, cj = 0, gg = 0;
            const bool used = (pf[g] & RS_USED) != 0;
            if (used) T.decode(tid + g * NT, ci, cj, gg);
            const long long m0 = (long long)T.column(ci, cj) * H + 4 * gg;
#pragma unroll
            for (int col = 0; col < 2; ++col) {
                const float* Kc = col ? c.K[1] : c.K[0];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float2 a01 = make_float2(0.0f, 0.0f), a23 = a01, a45 = a01;
                    float rr = 0.0f;
                    if (used && 4 * gg + q < H) {
                        const float2* rec = k_rec(Kc, c.ks, m0 + q);
                        a01 = __ldcg(rec);
                        a23 = __ldcg(rec + 1);
                        a45 = __ldcg(rec + 2);
                        rr = __ldcg(k_rp(Kc, c.ks, m0 + q));
                    }
                    k[col][g][q][0] = a01.x;
                    k[col][g][q][1] = a01.y;
                    k[col][g][q][2] = a23.x;
                    k[col][g][q][3] = a23.y;
                    k[col][g][q][4] = a45.x;
                    k[col][g][q][5] = a45.y;
                    r[col][g][q] = rr;
                }
            }
        }
        for (int q = tid; q < 2 * P.pad; q += NT) s0[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        event = EV_CYCLE_END;
        bool halved = false, fresh = true, ok = true;
        const double rx2 = sqrt(x2 + 1e-200);
        for (int inner = 0; inner < c.cycle; ++inner) {
            num_it += 1;
            num_sub_it += 1;
            const bool check = c.pressure_schedule ? (num_it < 50 || num_it % 10 == 0) : true;
            float d2 = 0.0f, dd = 0.0f;
            // red: the other colour's edges are zero at a cycle's start
            if (MODE == RES_CLUSTER) {
                cluster_sync();
            } else {
                if (!fresh)
                    res_poll<NT>(w.mem.recs[1], w.mem.plane, tag, reinterpret_cast<uint4*>(s1), hrec, hp, nh, c.bar, err);
                fresh = false;
                __syncthreads();
            }
            dc_res_sweep<NG, 0, MODE>(k, r, pf, s0, s1, w.mem.recs[0], w.mem.plane, rrow, rbase, ++tag, peers, dxp, dyp, sor,
                                      check, d2, dd);
            if (MODE == RES_CLUSTER) {
                cluster_sync();
            } else {
                res_poll<NT>(w.mem.recs[0], w.mem.plane, tag, reinterpret_cast<uint4*>(s0), hrec, hp, nh, c.bar, err);
                __syncthreads();
            }
            dc_res_sweep<NG, 1, MODE>(k, r, pf, s1, s0, w.mem.recs[1], w.mem.plane, rrow, rbase, ++tag, peers, dxp, dyp, sor,
                                      check, d2, dd);
            diff = 1e100;
            bool refresh = false;
            if (check) {
                double a = (double)d2, e = (double)dd;
                // a poll of this block that ran out shows here
                ok = res_team_sum<NT, MODE>(a, e, sum, w.mem.slots, nb, b, sums++, c.bar, err);
                if (!ok) break;
                const double ra = sqrt(a), l2 = ra / rx2;
                diff = (l2 != l2) ? 1.0 : l2;
                refresh = ra < kRefresh * sqrt(e);
            }
            if (diff < c.conv || c.stop_on_first) {
                t += dt;
                if (num_sub_it < c.max_it / 2.0) dt = pymin(dt * c.inc_it, c.max_dt);
                event = EV_CONVERGED;
                break;
            }
            if (num_sub_it >= c.max_it) {
                if (leader && nev < 8) {
                    status->ev_it[nev] = num_it;
                    status->ev_dt[nev] = dt;
                    status->ev_diff[nev] = diff;
                }
                nev += 1;
                dt = dt / 2;
                num_sub_it = 0;
                halved = true;
                halvings += 1;
            }
            if (dt <= c.min_dt) { event = halved ? EV_STOP_HALVED : EV_STOP; break; }
            if (halved) { event = EV_HALVE; break; }
            if (refresh) { event = EV_REFRESH; break; }
        }
        // the block's corrections are in shared memory, and no block still
        // writes into another's rings
        if (MODE == RES_CLUSTER)
            cluster_sync();
        else
            __syncthreads();
        if (!ok || *err) { event = EV_ERROR; break; }
        // ---- the cycle's end, over the block's own cells
        const bool last = event == EV_CONVERGED || event == EV_STOP || event == EV_STOP_HALVED;
        const bool reset = event == EV_HALVE || event == EV_STOP_HALVED;
        for (int u = tid; u < 2 * T.groups; u += NT) {
            const int col = u >= T.groups;
            int ci, cj, g;
            T.decode(u - col * T.groups, ci, cj, g);
            const float* s = reinterpret_cast<const float*>((col ? s1 : s0) + T.p(ci, cj, g));
            double* X = col ? c.X[1] : c.X[0];
            const uint8_t* msk = col ? c.mask[1] : c.mask[0];
            const int i = T.i0 + ci, j = T.j0 + cj;
            for (int q = 0; q < 4 && 4 * g + q < H; ++q) {
                const long long m = (long long)T.column(ci, cj) * H + 4 * g + q;
                double x;
                if (reset) {
                    F.reassemble(col, m, dt);
                    scale_cell(F, c, col, m);
                    x = X[m];
                } else {
                    x = X[m];
                    if (msk[m] & F_ACTIVE) x = x + (double)s[q];
                    if (!last) X[m] = x;
                }
                const int z = 2 * (4 * g + q) + ((i + j + col) & 1);
                if (last && z < nz) X_out[((long long)i * ny + j) * nz + z] = x;
            }
        }
        if (last) break;
        // the residual reads neighbours' x
        if (MODE == RES_CLUSTER) {
            cluster_sync();
        } else if (nb > 1) {
            if (!count_sync(w.mem.counter, ++bars * nb, c.bar)) { event = EV_ERROR; break; }
        } else {
            __syncthreads();
        }
        double o2 = 0.0;
        for (int u = tid; u < 2 * T.groups; u += NT) {
            const int col = u >= T.groups;
            int ci, cj, g;
            T.decode(u - col * T.groups, ci, cj, g);
            for (int q = 0; q < 4 && 4 * g + q < H; ++q) {
                const long long m = (long long)T.column(ci, cj) * H + 4 * g + q;
                const uint8_t f = (col ? c.mask[1] : c.mask[0])[m];
                const double x = (col ? c.X[1] : c.X[0])[m];
                o2 = o2 + x * x;
                float rp = 0.0f;
                if (f & F_ACTIVE) {
                    const double den = F.den(col, m);
                    rp = (float)((F.sum(col, m, f, col ? c.X[0] : c.X[1]) - den * x) / den);
                }
                *k_rp(col ? c.K[1] : c.K[0], c.ks, m) = rp;
            }
        }
        x2 = o2;
        unused = 0.0;
        ok = res_team_sum<NT, MODE>(x2, unused, sum, w.mem.slots, nb, b, sums++, c.bar, err);
        if (!ok) { event = EV_ERROR; break; }
        cycles += 1;
        __syncthreads();
    }
    bool failed = event == EV_ERROR;
    if (res_last<MODE>(w.mem.leavers, nb, b, failed)) {
        TseSolveStatus* s = status;
        s->t = t;
        s->dt = dt;
        s->diff = diff;
        s->converged = event == EV_CONVERGED && !failed;
        s->num_it = num_it;
        s->num_sub_it = num_sub_it;
        s->halvings = halvings;
        s->error = failed ? TSE_STATUS_BARRIER_TIMEOUT : TSE_STATUS_OK;
        s->n_events = nev < 8 ? nev : 8;
        s->cycles = cycles;
    }
}

// The instances: a thread holds one group of either colour (57 registers)
// with 512 threads a block, or two with 384.
constexpr int kDcResCluster = 16;   // blocks of a cluster launch
constexpr int kDcResGroups1 = 512, kDcResGroups2 = 2 * 384;
// the largest grid (cells per colour) a workspace carries exchange memory
// for: what 160 blocks hold
constexpr long long kDcResMaxNc = 160LL * kDcResGroups2 * kDcResVals;

inline int dc_res_threads(const ResPlan& P) { return P.groups <= kDcResGroups1 ? 512 : 384; }

// workspace bytes after the DC arrays
inline size_t dc_res_bytes(const Layout& L) { return 256 + res_mem_bytes(L, kDcResVals); }

// Run the whole solve in one launch when the grid fits on the chip: TSE_OK,
// TSE_ERR_LAUNCH, or 1 when the streaming sweeps should run.
template <class Form>
static int run_dc_resident(SolveSetup<Form>& S, DcCtl& c, double dt, int cap, int nparts, double* X_out,
                           TseSolveStatus* d_status, TseDcOptions* timing, cudaStream_t stream) {
    const size_t before = dc_extra_bytes(S.L);
    if (nparts <= 0 || S.L.Nc > kDcResMaxNc || S.tail_bytes < before + dc_res_bytes(S.L)) return 1;
    // the streaming form synchronises the stream and so refuses a capture;
    // this form does not change that
    cudaStreamCaptureStatus cap_st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap_st) != cudaSuccess || cap_st != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return 1;
    }
    int dev = 0, sms = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    const int room = optin - 2048;
    ResPlan P;
    bool cluster = false;
    const void* fn = nullptr;
    int threads = 0;
    // one cluster where its blocks hold the grid (a half-sweep's exchange
    // through shared memory is shorter than through L2), else the whole GPU
    for (int form = 0; form < 2 && !fn; ++form) {
        cluster = form == 0;
        int maxb = cluster ? kDcResCluster : sms < kResMaxBlocks ? sms : kResMaxBlocks;
        if (cap > 0 && maxb > cap) maxb = cap;
        if (!res_plan(S.L, kDcResVals, maxb, kDcResGroups2, room, dc_res_smem, dc_res_threads, true, P))
            continue;
        if (P.nb == 1) cluster = false;
        threads = dc_res_threads(P);
        const bool one = threads == 512;
        fn = cluster ? (one ? (const void*)dc_resident_kernel<Form, 512, 1, RES_CLUSTER>
                            : (const void*)dc_resident_kernel<Form, 384, 2, RES_CLUSTER>)
                     : (one ? (const void*)dc_resident_kernel<Form, 512, 1, RES_GRID>
                            : (const void*)dc_resident_kernel<Form, 384, 2, RES_GRID>);
        if (!res_can_launch(fn, P, threads, room, cluster)) fn = nullptr;
    }
    if (!fn) return 1;
    char* base = (char*)(((uintptr_t)S.tail + before + 255) & ~(uintptr_t)255);
    DcResCtl w;
    w.mem = res_mem(base, S.L, kDcResVals);
    w.nparts = nparts;
    w.dt = dt;
    // tags count from 1
    if (!cluster && P.nb > 1 && cudaMemsetAsync(base, 0, res_mem_bytes(S.L, kDcResVals), stream) != cudaSuccess)
        return TSE_ERR_LAUNCH;
    void* args[] = {(void*)&S.F, (void*)&c, (void*)&P, (void*)&w, (void*)&X_out, (void*)&d_status};
    if (!timing) return res_launch(fn, P, threads, cluster, args, stream) ? TSE_OK : TSE_ERR_LAUNCH;
    // the one launch holds the cycles' residuals too
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int its = 0;
    float ms = 0.0f;
    const bool ok =
        cudaEventCreate(&ev0) == cudaSuccess && cudaEventCreate(&ev1) == cudaSuccess &&
        cudaEventRecord(ev0, stream) == cudaSuccess && res_launch(fn, P, threads, cluster, args, stream) &&
        cudaEventRecord(ev1, stream) == cudaSuccess &&
        cudaMemcpyAsync(&its, &d_status->num_it, sizeof(int), cudaMemcpyDeviceToHost, stream) == cudaSuccess &&
        cudaStreamSynchronize(stream) == cudaSuccess && cudaEventElapsedTime(&ms, ev0, ev1) == cudaSuccess;
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (!ok) return TSE_ERR_LAUNCH;
    timing->sweep_launches = 1;
    timing->sweep_iterations = its;
    timing->sweep_ms = ms;
    timing->loop_ms = 0.0;
    return TSE_OK;
}

}  // namespace tse
