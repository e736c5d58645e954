// Persistent red-black solver loop shared by the pressure and transport
// solves (tse.py:699-740 for compute_P, 877-914 for compute_C, 1045-1079 for
// compute_T).
//
// One cooperative launch runs the whole `while not converged` loop of the
// reference on the device: red half-sweep, grid barrier, black half-sweep,
// per-block partial sums of (new - old)^2 and old^2, grid barrier, the L2
// test, dt growth on convergence, or dt halving with a reset to the entry
// state after max_it sub-iterations.  Every block evaluates the L2 from the
// same partials in the same order, so all blocks take the same branch.
//
// Work mapping: block b, thread t owns compact cells m = b*blockDim + t +
// s*gridDim*blockDim of each colour for the whole solve, in the sweeps and in
// the reset alike, so a block only ever re-reads its own writes except for
// the other colour's values, which it loads through L2 (ld.cg).
#pragma once

#include "tse_common.cuh"

namespace tse {

struct SolveCtl {
    Layout L;
    long long Ncal;             // padded per-colour array length
    double dt, inc_it, max_dt, min_dt, conv;
    int max_it;
    int pressure_schedule;      // 1: L2 every it below 50, then every 10th
    int stop_on_first;          // 1: converged after one it (omega == 0)
    int plain_sweep;            // 1: plain-load kernel even where the staged one fits (plain_sweep())
    double* X[2];               // solution per colour
    const uint8_t* mask[2];
    double* partials;           // 2 doubles per block
    GridBarrier* bar;
    TseSolveStatus* status;
};

constexpr int kMaxBlocks = 16384;

// One block a SM (148 arrivals a barrier) of as many threads as registers last
// for, a cell a thread where that covers the grid.  Bound: latency, of the
// barrier and of the loads behind it; what a thread's first cell reads, but for
// the neighbours, is loaded before the barrier.  us an iteration on a B200
// (pressure, x and z buoyancy): 72^3 16.0 -> 12.9, 80^3 16.3 -> 14.8, 100^3 31.4 ->
// 27.6; 512 or 640 threads 12.5, 14.4 and from 96^3 on a tenth more, 1024 (which
// spills) 14.4 at 72^3.
constexpr int kPlainBlock = 768;
// From this many cells of a colour on the staged sweep (tse_rbsolve_tma.cuh) is
// the faster one, below this one (staged / plain: 72^3 19.3 / 12.9, 100^3 30.2 /
// 27.6, 110^3 35.8 / 33.4, 128 x 128 x 127 47.1 / 46.4, 192 x 160 x 101 65.1 / 74.4;
// 1300 x 1 x 1300 54.9 / 40.7).  A pressure solve of fewer than 50 iterations, which
// all check, is 2-5 % slower plain from 0.7 M cells on.
constexpr long long kStagedMinNc = 1000000;

// `sweep` as the entry points take it: 1 plain, 2 staged, else by size
inline int plain_sweep(int sweep, const Layout& L) { return sweep == 1 || (sweep != 2 && L.Nc < kStagedMinNc); }

// What the update of a cell reads that the other colour does not write.
template <class Form>
struct Ahead {
    double a[Form::kCoef], xold;
    uint8_t f;
    __device__ __forceinline__ void load(const Form& F, const SolveCtl& c, int col, long long m) {
        const double* b = (col ? F.arr[1] : F.arr[0]) + m;
        f = (col ? c.mask[1] : c.mask[0])[m];
        xold = (col ? c.X[1] : c.X[0])[m];
#pragma unroll
        for (int k = 0; k < Form::kCoef; ++k)
            if (F.reads(k)) a[k] = b[(long long)k * F.Ncal];
    }
};

template <class Form>
__global__ void __launch_bounds__(kPlainBlock, 1) rb_solve_kernel(Form F, SolveCtl c) {
    __shared__ double sh[kPlainBlock / 32];
    __shared__ double s_diff;
    const unsigned nb = gridDim.x;
    const long long tid0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)nb * blockDim.x;
    const long long Nc = c.L.Nc;
    const bool leader = (blockIdx.x == 0 && threadIdx.x == 0);

    double t = 0.0, dt = c.dt, diff = 1e100;
    int converged = 0, num_it = 0, num_sub_it = 0, halvings = 0, err = 0, nev = 0;

    Ahead<Form> own;
    if (tid0 < Nc) own.load(F, c, 0, tid0);
    while (!converged) {
        num_it += 1;
        num_sub_it += 1;
        double d2 = 0.0, o2 = 0.0;
        const bool check = c.pressure_schedule ? (num_it < 50 || num_it % 10 == 0) : true;
        for (int col = 0; col < 2; ++col) {
            double* Xw = col ? c.X[1] : c.X[0];
            const double* Xo = col ? c.X[0] : c.X[1];
            for (long long m = tid0; m < Nc; m += stride) {
                if (m != tid0) own.load(F, c, col, m);
                const uint8_t f = own.f;
                const double xold = own.xold;
                o2 = o2 + xold * xold;
                if (f & F_ACTIVE) {
                    const long long zo = f >> 7;
                    const double xn = F.update_with(
                        [&](int k) { return own.a[k]; },
                        [&](int q) { return __ldcg(Xo + m + nb_offset(q, F.SX, F.H, zo)); }, f, xold);
                    Xw[m] = xn;
                    const double d = xn - xold;
                    d2 = d2 + d * d;
                }
            }
            // the first cell's loads of the next half-sweep pass behind the
            // barrier: all of them were last written by this thread
            if (tid0 < Nc) own.load(F, c, col ^ 1, tid0);
            if (col == 1 && check) {
                // per-block partial sums, published by the barrier below
                double b1 = block_sum<kPlainBlock>(d2, sh);
                double b2 = block_sum<kPlainBlock>(o2, sh);
                if (threadIdx.x == 0) {
                    c.partials[2 * blockIdx.x] = b1;
                    c.partials[2 * blockIdx.x + 1] = b2;
                }
            }
            if (!grid_sync(c.bar, nb)) { err = 1; break; }
        }
        if (err) break;
        diff = 1e100;
        if (check) {
            double s1 = 0.0, s2 = 0.0;
            for (unsigned b = threadIdx.x; b < nb; b += blockDim.x) {
                s1 = s1 + __ldcg(c.partials + 2 * b);
                s2 = s2 + __ldcg(c.partials + 2 * b + 1);
            }
            s1 = block_sum<kPlainBlock>(s1, sh);
            s2 = block_sum<kPlainBlock>(s2, sh);
            if (threadIdx.x == 0) {
                double l2 = sqrt(s1) / sqrt(s2 + 1e-200);
                s_diff = (l2 != l2) ? 1.0 : l2;
            }
            __syncthreads();
            diff = s_diff;
            // the next iteration's partial writes come after the next
            // half-sweep barrier, which every block reaches only after this
            // read: one partials buffer is enough
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
                for (int col = 0; col < 2; ++col)
                    for (long long m = tid0; m < Nc; m += stride) F.reassemble(col, m, dt);
                if (tid0 < Nc) own.load(F, c, 0, tid0);
                if (!grid_sync(c.bar, nb)) { err = 1; break; }
            }
            if (dt <= c.min_dt) break;
        }
    }
    if (leader) {
        TseSolveStatus* s = c.status;
        s->t = t;
        s->dt = dt;
        s->diff = diff;
        s->converged = converged;
        s->num_it = num_it;
        s->num_sub_it = num_sub_it;
        s->halvings = halvings;
        s->error = err ? TSE_STATUS_BARRIER_TIMEOUT : TSE_STATUS_OK;
        s->n_events = nev < 8 ? nev : 8;
        s->cycles = 0;
        s->sweep = TSE_SWEEP_PLAIN;
    }
}

// Launch the persistent loop with as many co-resident blocks as useful.
template <class Form>
inline int launch_rb_solve(const Form& F, SolveCtl& ctl, cudaStream_t stream) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return TSE_ERR_LAUNCH;
    // a cell a thread, at most the co-resident blocks
    const long long want = (ctl.L.Nc + kPlainBlock - 1) / kPlainBlock;
    const long long nb = want < 1 ? 1 : want < sms ? want : sms;
    void* args[] = {(void*)&F, (void*)&ctl};
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)rb_solve_kernel<Form>, dim3((unsigned)nb),
                                                dim3(kPlainBlock), args, 0, stream);
    return e == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

}  // namespace tse
