// FP32 red-black SOR with FP64 defect correction: the mixed-precision form of
// the pressure, species and heat solves.
//
// The FP64 solves (tse_pressure.cu, tse_transport.cu) stream 11-15 double
// words per cell-update.  Here the same SOR iteration runs on a correction:
// with the FP64 iterate x, the residual of the reference's per-cell equation
//   r = sum(x) - Den * x            (sum / Den as in compute_P/C/T.solve)
// is formed in FP64, and red-black SOR sweeps
//   d = (1 - SOR) d + SOR (sum_q K'_q d_q + r')  with K'_q = k_q / Den, r' = r / Den
// run in FP32 from d = 0.  In exact arithmetic x + d follows the FP64 SOR
// iteration step for step, so the reference's convergence test (relative L2
// change of one iteration, checked on its schedule) and its dt control are
// applied to the change of d unchanged.  x += d in FP64 and the residual is
// formed again (a correction cycle ends) at convergence, every `cycle`
// iterations, and at a check whose change has fallen below kRefresh * |d|:
// FP32 resolves d to ~6e-8 |d|, so the measured change stays ~1e3 times above
// d's rounding and the iteration counts track the FP64 form's.
//
// Kernels: a grid that fits on the chip solves in one launch, cycles included
// (dc_resident_kernel, tse_dc_resident.cuh).  Else the FP32 sweeps run in one
// cooperative kernel that iterates until an event (converged, cycle end, dt halving, stop): dc_sweep_tma_kernel,
// which stages each chunk's data in shared memory with bulk asynchronous
// copies, or, where its stages do not fit, dc_sweep_kernel (48 registers,
// 5 blocks per SM, plain loads).  The FP64 residual, the x += d update and the dt
// halving (reset + new R terms) are separate, ordinary kernels, so their
// register appetite does not limit the sweeps' occupancy; the first cycle's
// records, residual and x^2 come from the assembly pass itself (setup_*_dc),
// and the last x += d is fused with the unpack.  The host reads one small
// state record per correction cycle.
//
// An inner cell-update streams the six FP32 coefficients (one 24-byte record),
// r' and the flag byte from DRAM -- 29 bytes; d and the neighbours' d stay in
// L2 -- against 89 bytes of coefficients and flags for the FP64 form.
//
// Compiled with FMA contraction (no bit-exactness is claimed for this form).
#include <cstddef>
#include <type_traits>

#include "tse_dc.cuh"
#include "tse_dc_resident.cuh"

namespace tse {

#ifndef TSE_SWEEP_MINB
#define TSE_SWEEP_MINB 5   // 48 registers, no spills (measured best of 4/5/6/8)
#endif
constexpr int kSweepMinBlocks = TSE_SWEEP_MINB;
#ifndef TSE_SWEEP_BLOCK
#define TSE_SWEEP_BLOCK 256
#endif
constexpr int kSweepBlock = TSE_SWEEP_BLOCK;

// Pipelines of the staged sweep: each has its own producer warp, its own ring
// of stages and its own consumer group, and takes every PIPES-th chunk of the
// block.  A producer warp issues its copies one after another, at a rate that
// bounds a pipeline's throughput: two pipelines per block, one block per SM,
// up to 4 stages a ring.  (Measured against one pipeline -- two consumer
// groups sharing a ring -- and two blocks per SM: faster at every grid from
// 96^3 to 256 x 256 x 128.)
constexpr int kDcPipes = 2;
constexpr int kDcMaxRing = 4;
//
// Consumers: 8 warps, or 16 (WIDE, two pipelines) where the solve's state stays
// in L2 and the chunks arrive faster than 8 warps relax them.  Measured, us per
// iteration with 8 and with 16: 128^3 14.8 and 13.5, 192 x 192 x 128 22.5 and
// 22.2, whole 256 x 256 x 128 solves at the power cap 460 and 467 ms.
template <int PIPES, bool WIDE = false>
struct DcLayout {
    static_assert(!WIDE || PIPES == 2, "one pipeline runs two blocks per SM");
    static constexpr int kConsumers = WIDE ? 2 * kTmaConsumers : kTmaConsumers;
    static constexpr int kThreads = kConsumers + 32 * PIPES + 64;   // consumers, producers, reporter, gatekeeper
    static constexpr int kMinBlocks = PIPES == 1 ? 2 : 1;
    static constexpr int kGroups = kConsumers / kTmaGroup;
    static constexpr int kGroupsPerPipe = kGroups / PIPES;
    static_assert(kGroups % PIPES == 0, "every pipeline has its own consumer groups");
};

// ------------------------------------------------------------ FP64 kernels
// a solve's state record at its start: all zero but dt and diff (written on
// the device, so starting a solve queues no host-memory copy)
__global__ void dc_init_state_kernel(DcState* st, double dt) {
    DcState s;
    memset(&s, 0, sizeof(s));
    s.dt = dt;
    s.diff = 1e100;
    *st = s;
}

// K'_q = k_q / Den for every cell (at the start and after dt halving)
template <class Form>
__global__ void dc_scale_kernel(Form F, DcCtl c) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * c.L.Nc) return;
    const int col = t >= c.L.Nc;
    scale_cell(F, c, col, t - col * c.L.Nc);
}

// dt halving: x = Xn, new R terms (tse.py:733-738), rescaled coefficients
template <class Form>
__global__ void dc_halve_kernel(Form F, DcCtl c) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * c.L.Nc) return;
    const int col = t >= c.L.Nc;
    const long long m = t - col * c.L.Nc;
    F.reassemble(col, m, c.st->dt);
    scale_cell(F, c, col, m);
}

// r' = (sum(x) - Den x) / Den in FP64, d = 0, per-block sums of x^2
template <class Form>
__global__ void __launch_bounds__(kBlock) dc_residual_kernel(Form F, DcCtl c) {
    __shared__ double sh[kBlock / 32];
    const double o2 = residual_block_cells(F, c, blockIdx.x, gridDim.x);
    const double b = block_sum<kBlock>(o2, sh);
    if (threadIdx.x == 0) c.partials[blockIdx.x] = b;
}

// x += d and the residual of the new iterate in one pass, the new iterate into
// another pair of arrays (Xn): neighbours' values are formed from their old
// ones and their corrections.  The corrections are zeroed after the launch.
// Bound: DRAM.  A thread takes two consecutive cells of a colour, and loads
// everything before it computes, neighbours the grid does not have included
// (inside the workspace and unused).  Cells of a colour: one thread each and
// loads under their flags took 222 us at 256 x 256 x 128.
template <class Form>
__global__ void __launch_bounds__(kBlock) dc_apply_residual_kernel(Form F, DcCtl c, double* Xn0, double* Xn1) {
    __shared__ double sh[kBlock / 32];
    const long long Nc = c.L.Nc, N = c.Ncal, sx = c.L.SX, pairs = (Nc + 1) / 2;
    const int h = c.L.H;
    double o2 = 0.0;
    for (long long t = (long long)blockIdx.x * kBlock + threadIdx.x; t < 2 * pairs;
         t += (long long)gridDim.x * kBlock) {
        const int col = t >= pairs;
        const long long m = 2 * (t - (col ? pairs : 0));
        const uint8_t* mk = (col ? c.mask[1] : c.mask[0]) + m;
        const double* b = (col ? F.arr[1] : F.arr[0]) + m;
        const double* Xo = (col ? c.X[0] : c.X[1]) + m;
        const float* Do = (col ? c.D[0] : c.D[1]) + m;
        // Ncal, the arrays' length, is a multiple of 32: a pair is inside
        const uint8_t f0 = mk[0], f1 = mk[1];
        double2 a[Form::kCoef];
#pragma unroll
        for (int k = 0; k < Form::kCoef; ++k)
            if (F.later(k)) a[k] = *reinterpret_cast<const double2*>(b + k * N);
        const double2 x = *reinterpret_cast<const double2*>((col ? c.X[1] : c.X[0]) + m);
        const float2 d = *reinterpret_cast<const float2*>((col ? c.D[1] : c.D[0]) + m);
        double xa[6], xb[6];
        float da[6], db[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const long long oa = nb_offset(q, sx, h, (long long)(f0 >> 7));
            const long long ob = 1 + nb_offset(q, sx, h, (long long)(f1 >> 7));
            xa[q] = Xo[oa];
            da[q] = Do[oa];
            xb[q] = Xo[ob];
            db[q] = Do[ob];
        }
        const double x0 = (f0 & F_ACTIVE) ? x.x + (double)d.x : x.x;
        const double x1 = (f1 & F_ACTIVE) ? x.y + (double)d.y : x.y;
        float r0 = 0.0f, r1 = 0.0f;
        if (f0 & F_ACTIVE) {
            const double s = F.sum_with([&](int k) { return a[k].x; }, [&](int q) { return xa[q] + (double)da[q]; }, f0);
            r0 = (float)((s - a[Form::kDen].x * x0) / a[Form::kDen].x);
        }
        if (f1 & F_ACTIVE) {
            const double s = F.sum_with([&](int k) { return a[k].y; }, [&](int q) { return xb[q] + (double)db[q]; }, f1);
            r1 = (float)((s - a[Form::kDen].y * x1) / a[Form::kDen].y);
        }
        *reinterpret_cast<double2*>((col ? Xn1 : Xn0) + m) = make_double2(x0, x1);
        *reinterpret_cast<float2*>(k_rp(col ? c.K[1] : c.K[0], c.ks, m)) = make_float2(r0, r1);
        o2 = o2 + x0 * x0;
        if (m + 1 < Nc) o2 = o2 + x1 * x1;
    }
    const double s2 = block_sum<kBlock>(o2, sh);
    if (threadIdx.x == 0) c.partials[blockIdx.x] = s2;
}

// x^2 total into the state; counts the cycle; zero_prog: the staged sweep's
// counters start at 0 (a memset of their own costs 4 us a cycle)
__global__ void dc_x2_kernel(DcCtl c, int nparts, int zero_prog = 0) {
    __shared__ double sh[kBlock / 32];
    if (zero_prog)
        for (int q = threadIdx.x; q < (int)(kProgBytes / sizeof(unsigned)); q += kBlock) c.prog[q] = 0;
    double s = 0.0;
    int b = threadIdx.x;
    // eight loads in flight, summed in the order of the plain loop
    for (; b + 7 * kBlock < nparts; b += 8 * kBlock) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = c.partials[b + u * kBlock];
#pragma unroll
        for (int u = 0; u < 8; ++u) s = s + v[u];
    }
    for (; b < nparts; b += kBlock) s = s + c.partials[b];
    s = block_sum<kBlock>(s, sh);
    if (threadIdx.x == 0) {
        c.st->x2 = s;
        c.st->cycles += 1;
    }
}

// x += d for active cells
__global__ void dc_apply_kernel(DcCtl c) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * c.L.Nc) return;
    const int col = t >= c.L.Nc;
    const long long m = t - col * c.L.Nc;
    if (c.mask[col][m] & F_ACTIVE) c.X[col][m] = c.X[col][m] + (double)c.D[col][m];
}

// x += d and the natural-layout result in one pass: the last cycle of a
// solve (dc_apply_kernel then unpack_kernel, without storing x)
__global__ void dc_apply_unpack_kernel(double* out, DcCtl c) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)c.L.nx * c.L.ny * c.L.nz;
    if (t >= total) return;
    int i, j, k;
    long long row;
    grid_coords(t, c.L.ny, c.L.nz, i, j, k, row);
    const long long m = (row * c.L.nzp + k) >> 1;
    const int col = (i + j + k) & 1;
    double x = c.X[col][m];
    if (c.mask[col][m] & F_ACTIVE) x = x + (double)c.D[col][m];
    out[t] = x;
}

// ------------------------------------------------------------ FP32 sweeps
__device__ __forceinline__ double reduce_slot(const double* parts, int slot, unsigned nb, double* sh,
                                              double* s_val) {
    double s = 0.0;
    for (unsigned b = threadIdx.x; b < nb; b += blockDim.x) s = s + __ldcg(parts + 4 * b + slot);
    s = block_sum<kSweepBlock>(s, sh);
    if (threadIdx.x == 0) *s_val = s;
    __syncthreads();
    const double r = *s_val;
    __syncthreads();
    return r;
}

// Inner iterations of one correction cycle.  Cells are interleaved over the
// grid (block b, thread t: m = b*256 + t + s*gridDim*256), which keeps all
// blocks streaming one narrow window of memory; colour phases are separated
// by the grid barrier.  Per-block partial sums alternate between two slot
// pairs by check parity, so a slot is rewritten only after a further barrier.
__global__ void __launch_bounds__(kSweepBlock, kSweepMinBlocks) dc_sweep_kernel(DcCtl c) {
    __shared__ double sh[kSweepBlock / 32];
    __shared__ double s_val;
    const unsigned nb = gridDim.x;
    const long long Nc = c.L.Nc, SX = c.L.SX;
    const int H = c.L.H;
    const int lane = threadIdx.x & 31;
    const long long end = Nc;
    const long long step = (long long)nb * blockDim.x;
    const long long w0 = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane;
    const bool leader = (blockIdx.x == 0 && threadIdx.x == 0);
    const float sor = c.sor;
    DcState* st = c.st;
    double t = st->t, dt = st->dt, diff = 1e100;
    const double x2 = st->x2;
    int num_it = st->num_it, num_sub_it = st->num_sub_it, checkno = st->checkno;
    int event = EV_CYCLE_END;
    bool halved = false;

    for (int inner = 0; inner < c.cycle; ++inner) {
        num_it += 1;
        num_sub_it += 1;
        const bool check = c.pressure_schedule ? (num_it < 50 || num_it % 10 == 0) : true;
        if (check) checkno += 1;
        float d2 = 0.0f, dd = 0.0f;
        bool ok = true;
        for (int col = 0; col < 2 && ok; ++col) {
            const float* __restrict__ Kc = c.K[col];
            float* dw = c.D[col];
            const float* dq = c.D[1 - col];
            const uint8_t* __restrict__ msk = c.mask[col];
            // all loads of a cell are independent: coefficients of absent
            // neighbours are 0 and dq's margins are 0; inactive cells have
            // all-zero coefficients and r' = 0 and stay at d = 0.  Trips are
            // counted per warp so every lane joins the shuffles; lanes past
            // the end load a valid cell and store nothing.
            for (long long w = w0; w < end; w += step) {
                const long long ma = w + lane;
                const bool va = ma < end;
                const long long la = va ? ma : end - 1;
                Cell a;
                load_cell(a, Kc, dw, dq, msk, la, c.ks, SX, H);
                const float na = relax(a, dq, la, end, sor);
                if (va) {
                    dw[ma] = na;
                    const float ch = na - a.old;
                    d2 = fmaf(ch, ch, d2);
                    dd = fmaf(na, na, dd);
                }
            }
            if (col == 1 && check) {
                const double b1 = block_sum<kSweepBlock>((double)d2, sh);
                const double b3 = block_sum<kSweepBlock>((double)dd, sh);
                if (threadIdx.x == 0) {
                    c.partials[4 * blockIdx.x + 2 * (checkno & 1)] = b1;
                    c.partials[4 * blockIdx.x + 2 * (checkno & 1) + 1] = b3;
                }
            }
            ok = grid_sync(c.bar, nb);
        }
        if (!ok) { event = EV_ERROR; break; }
        diff = 1e100;
        bool refresh = false;
        if (check) {
            const double s1 = reduce_slot(c.partials, 2 * (checkno & 1), nb, sh, &s_val);
            const double s3 = reduce_slot(c.partials, 2 * (checkno & 1) + 1, nb, sh, &s_val);
            const double l2 = sqrt(s1) / sqrt(x2 + 1e-200);
            diff = (l2 != l2) ? 1.0 : l2;
            refresh = sqrt(s1) < kRefresh * sqrt(s3);
        }
        if (diff < c.conv || c.stop_on_first) {
            t += dt;
            if (num_sub_it < c.max_it / 2.0) dt = pymin(dt * c.inc_it, c.max_dt);
            event = EV_CONVERGED;
            break;
        }
        if (num_sub_it >= c.max_it) {
            if (leader && st->nev < 8) {
                st->ev_it[st->nev] = num_it;
                st->ev_dt[st->nev] = dt;
                st->ev_diff[st->nev] = diff;
            }
            if (leader) st->nev += 1;
            dt = dt / 2;
            num_sub_it = 0;
            halved = true;
        }
        if (dt <= c.min_dt) { event = halved ? EV_STOP_HALVED : EV_STOP; break; }
        if (halved) { event = EV_HALVE; break; }
        if (refresh) { event = EV_REFRESH; break; }
    }
    if (leader) {
        st->t = t;
        st->dt = dt;
        st->diff = diff;
        st->num_it = num_it;
        st->num_sub_it = num_sub_it;
        st->checkno = checkno;
        st->event = event;
        if (halved) st->halvings += 1;
        if (event == EV_CONVERGED) st->converged = 1;
    }
}

// ------------------------------------------------ FP32 sweeps, bulk-copy staged
// (the staging pieces are in tse_dc.cuh)
//
// Colour phases are not separated by a device-wide barrier: a phase's first
// rounds begin while the phase before ends (sweep_head), so the copy pipelines
// run on from one phase into the next; only iterations that check the
// convergence end in a barrier.  A report costs the block no time of its own:
// the consumers arrive on a barrier of the block, a reporter warp waits there
// and makes their stores visible to the GPU, and a gatekeeper warp waits for
// the other blocks and opens the next rounds to the producers.  Every one of
// these steps on a consumer's or a producer's path made the sweep slower than
// the device-wide barrier did (consumers' fences 2.5 times, the producers'
// polls 1.5 times, the producers' proxy fences 1.2 times).  Bound: DRAM, 29
// bytes an update, and at the power cap's clocks the producers' issue rate (5
// copies a chunk) and the consumers'.  Barrier after every phase and now, us per iteration
// of the sweep alone (B200, both on one box, twice): 128^3 15.2 -> 14.6, 192 x
// 192 x 128 26.2 -> 23.3, 256 x 256 x 128 42.0-42.8 -> 39.7-42.3 (0.94 of the
// measured HBM rate at best), 320 x 320 x 160 88.3 -> 82.6-83.5; with the record
// blocks and 8 or 16 consumer warps 13.5, 22.2, 38.8-41.2 and 83.4-86.
template <int RING, int PIPES, int CHUNK, bool WIDE>
__global__ void __launch_bounds__(DcLayout<PIPES, WIDE>::kThreads, DcLayout<PIPES, WIDE>::kMinBlocks)
    dc_sweep_tma_kernel(DcCtl c, TmaStage T) {
    static_assert(CHUNK % kTmaGroup == 0 && CHUNK <= kDcMaxChunk, "whole cells per thread, in the margins");
    constexpr int kCellsPerThread = CHUNK / kTmaGroup;
    constexpr int kPipes = PIPES;
    constexpr int kThreads = DcLayout<PIPES, WIDE>::kThreads;
    constexpr int kConsumers = DcLayout<PIPES, WIDE>::kConsumers;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[RING * PIPES];
    __shared__ __align__(8) uint64_t empty[RING * PIPES];
    __shared__ double sh[kThreads / 32];
    __shared__ __align__(8) uint64_t seg_bar[kSegs], gate[kSegs];
    __shared__ int s_err;
    const unsigned nb = gridDim.x, b = blockIdx.x;
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const bool reporter = warp == kConsumers / 32 + kPipes;
    const bool gatekeeper = warp == kConsumers / 32 + kPipes + 1;
    const bool producer = !reporter && !gatekeeper && warp >= kConsumers / 32;
    const int group = tid / kTmaGroup;                  // consumers: 0, 1, ...
    const int gt = tid & (kTmaGroup - 1);               // thread within its group
    // this thread's pipeline (producer warp + its ring of stages +
    // its consumer groups), and a consumer group's rank within it
    const int pipe = producer ? warp - kConsumers / 32 : group % kPipes;
    const int grank = group / kPipes;
    constexpr int kGroupsPerPipe = DcLayout<PIPES, WIDE>::kGroupsPerPipe;
    constexpr unsigned ring = RING;                     // stages of a ring (T.stages / PIPES)
    const unsigned ring0 = (unsigned)pipe * ring;    // the pipeline's first stage
    const long long Nc = c.L.Nc, N = c.Ncal, SX = c.L.SX, C = CHUNK;
    const int H = c.L.H;
    const long long nch = (Nc + C - 1) / C;
    const long long mine = nch > (long long)b ? (nch - 1 - b) / nb + 1 : 0;   // chunks of this block
    // this pipeline's chunks of a phase: i = pipe, pipe + kPipes, ...
    const long long pmine = mine > pipe ? (mine - 1 - pipe) / kPipes + 1 : 0;
    unsigned* bar_count = c.prog;                // count_sync's counter, zeroed before the launch
    unsigned* seg_count = c.prog + kSegBase;     // the reports' likewise
    const int first = T.first;
    const int nseg = nch > (long long)first * nb ? 2 : 1;
    unsigned bars = 0;                           // device-wide barriers passed in this launch
    unsigned phases = 0;                         // colour phases before this one
    // blocks with chunks of report s, and the arrivals of this block's consumer
    // warps there (one a warp and chunk)
    auto seg_blocks = [&](int s) {
        const long long rest = nch - (s ? (long long)first * nb : 0);
        return rest < (long long)nb ? (unsigned)rest : nb;
    };
    auto seg_arrivals = [&](int s) {
        const long long n = s ? mine - first : mine < first ? mine : (long long)first;
        return (unsigned)(n * (kTmaGroup / 32));
    };
    const bool leader = (b == 0 && tid == 0);
    const float sor = c.sor;
    const uint64_t keep = l2_evict_last();
    DcState* st = c.st;
    double t = st->t, dt = st->dt, diff = 1e100;
    const double x2 = st->x2;
    int num_it = st->num_it, num_sub_it = st->num_sub_it, checkno = st->checkno;
    int event = EV_CYCLE_END;
    bool halved = false;
    volatile int* err = &s_err;

    if (tid == 0) {
        for (int s = 0; s < RING * kPipes; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kTmaGroup / 32);   // one arrival per warp of a group
        }
        for (int s = 0; s < nseg; ++s) {
            if (mine > (s ? first : 0)) mbar_init(&seg_bar[s], seg_arrivals(s));
            mbar_init(&gate[s], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_err = 0;
    }
    __syncthreads();
    unsigned uses = 0;      // this pipeline's chunks consumed, over all colour phases
    unsigned issued = 0;    // producer: this pipeline's chunks issued, over all phases
    // the corrections were written by the kernel before (generic stores)
    if (producer) fence_proxy_async();

    for (int inner = 0; inner < c.cycle; ++inner) {
        num_it += 1;
        num_sub_it += 1;
        const bool check = c.pressure_schedule ? (num_it < 50 || num_it % 10 == 0) : true;
        if (check) checkno += 1;
        float d2 = 0.0f, dd = 0.0f;
        for (int col = 0; col < 2; ++col, ++phases) {
            const float* Kc = c.K[col];
            float* dw = c.D[col];
            const float* dq = c.D[1 - col];
            if (producer) {
                if (lane == 0) {
                    for (long long j = 0; j < pmine; ++j, ++issued) {
                        const int i = pipe + (int)j * kPipes;
                        bool pok = true;
                        if (j == 0) pok = mbar_wait_flag(&gate[0], phases & 1u, err);
                        // the first of this pipeline's rounds past the head
                        if (nseg > 1 && i >= T.head && i - kPipes < T.head)
                            pok = pok && mbar_wait_flag(&gate[1], phases & 1u, err);
                        const unsigned s = ring0 + issued % ring;
                        if (!pok || (issued >= (unsigned)ring &&
                                     !mbar_wait_flag(&empty[s], (issued / ring - 1) & 1u, err)))
                            break;
                        const long long q = b + (long long)i * nb, m0 = q * C;
                        unsigned char* stg = smem + (size_t)s * T.bytes;
                        tma_issue_own(T, stg, &full[s], Kc + q * (29 * CHUNK / 4), dw + m0, (N - m0) < C ? (N - m0) : C);
                        tma_issue_windows(c, T, stg, &full[s], dq, m0);
                    }
                }
                __syncwarp();
            } else if (gatekeeper) {
                // the head opens when every block has made the first report of
                // the phase before, the rest when they have made the second
                if (lane == 0) {
                    bool gok = true;
                    for (int s = 0; gok && s < nseg; ++s) {
                        gok = seg_wait(seg_count + s * kSegWords, phases * seg_blocks(s), c.bar, err);
                        // the other colour was written by generic stores; the
                        // producers' copies read it through the async proxy
                        fence_proxy_async();
                        if (gok) mbar_arrive(&gate[s]);
                    }
                }
                __syncwarp();
            } else if (reporter) {
                if (lane == 0)
                    for (int s = 0; s < nseg && mine > (s ? first : 0); ++s) {
                        if (!mbar_wait_flag(&seg_bar[s], phases & 1u, err)) break;
                        red_release_add(seg_count + s * kSegWords, 1u);
                    }
                __syncwarp();
            } else {
                for (long long j = 0; j < pmine; ++j) {
                    const int i = pipe + (int)j * kPipes;
                    const unsigned u = uses + (unsigned)j;
                    // a stage belongs to one group for good: its parity waits
                    // then see every use.  (By chunk, a group could ask for a
                    // stage's next use while the other group's was still
                    // arriving, and the parity would pass.)
                    if ((int)((u % ring) % kGroupsPerPipe) != grank) continue;
                    const unsigned s = ring0 + u % ring;
                    const long long m0 = (b + (long long)i * nb) * C;
                    const int nval = (int)((Nc - m0) < C ? (Nc - m0) : C);
                    float* out = dw + m0;
                    // warp-uniform: lane 0 waits, the warp follows its outcome,
                    // then every lane observes the completed phase (acquire)
                    int okw = 1;
                    if (lane == 0) okw = mbar_wait_flag(&full[s], (u / ring) & 1u, err);
                    if (!__shfl_sync(0xffffffffu, okw, 0)) break;
                    mbar_try_wait(&full[s], (u / ring) & 1u);
                    const unsigned char* stg = smem + (size_t)s * T.bytes;
                    // window offsets of cell l of the chunk (32-bit from here on)
                    const int oz = (int)(m0 - ((m0 - H - 1) & ~3LL));
                    const int oxp = (int)(m0 + SX - ((m0 + SX) & ~3LL));
                    const int oxm = (int)(m0 - SX - ((m0 - SX) & ~3LL));
                    const float2* rec = reinterpret_cast<const float2*>(stg + T.rec);
                    const float* rp = reinterpret_cast<const float*>(stg + T.rp);
                    const uint8_t* fl = stg + T.msk;
                    const float* dwo = reinterpret_cast<const float*>(stg + T.dw);
                    const float* wz = reinterpret_cast<const float*>(stg + T.wz);
                    const float* wxp = reinterpret_cast<const float*>(stg + T.wxp);
                    const float* wxm = reinterpret_cast<const float*>(stg + T.wxm);
#pragma unroll
                    for (int r = 0; r < kCellsPerThread; ++r) {
                        const int l = gt + r * kTmaGroup;
                        if (l < nval) {
                            const float2 k01 = rec[3 * l], k23 = rec[3 * l + 1], k45 = rec[3 * l + 2];
                            const bool odd = (fl[l] & F_KODD) != 0;
                            const float old = dwo[l];
                            const int iz = l + oz;
                            const float z0 = wz[iz - 1], z1 = wz[iz], z2 = wz[iz + 1];
                            float acc = rp[l];
                            acc = fmaf(k01.x, wxp[l + oxp], acc);
                            acc = fmaf(k01.y, wxm[l + oxm], acc);
                            acc = fmaf(k23.x, wz[iz + H], acc);
                            acc = fmaf(k23.y, wz[iz - H], acc);
                            acc = fmaf(k45.x, odd ? z2 : z1, acc);
                            acc = fmaf(k45.y, odd ? z1 : z0, acc);
                            const float na = fmaf(sor, acc - old, old);
                            st_hint(out + l, na, keep);
                            const float ch = na - old;
                            d2 = fmaf(ch, ch, d2);
                            dd = fmaf(na, na, dd);
                        }
                    }
                    // the warp's reads of the stage are done: release it
                    // and its stores belong to the phase's report
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&empty[s]);
                        mbar_arrive(&seg_bar[i >= first]);
                    }
                }
            }
            uses += (unsigned)pmine;
        }
        diff = 1e100;
        bool refresh = false;
        if (check) {
            __syncthreads();
            if (*err) { event = EV_ERROR; break; }   // block-uniform after the barrier
            const double b1 = block_sum<kThreads>((double)d2, sh);
            const double b3 = block_sum<kThreads>((double)dd, sh);
            if (tid == 0) {
                c.partials[4 * b + 2 * (checkno & 1)] = b1;
                c.partials[4 * b + 2 * (checkno & 1) + 1] = b3;
            }
            if (!count_sync(bar_count, ++bars * nb, c.bar)) { event = EV_ERROR; break; }
            double s1 = 0.0, s3 = 0.0;
            for (unsigned q = tid; q < nb; q += blockDim.x) {
                s1 = s1 + __ldcg(c.partials + 4 * q + 2 * (checkno & 1));
                s3 = s3 + __ldcg(c.partials + 4 * q + 2 * (checkno & 1) + 1);
            }
            s1 = block_sum<kThreads>(s1, sh);
            s3 = block_sum<kThreads>(s3, sh);
            if (tid == 0) {
                sh[0] = s1;
                sh[1] = s3;
            }
            __syncthreads();
            s1 = sh[0];
            s3 = sh[1];
            __syncthreads();
            const double l2 = sqrt(s1) / sqrt(x2 + 1e-200);
            diff = (l2 != l2) ? 1.0 : l2;
            refresh = sqrt(s1) < kRefresh * sqrt(s3);
        }
        if (diff < c.conv || c.stop_on_first) {
            t += dt;
            if (num_sub_it < c.max_it / 2.0) dt = pymin(dt * c.inc_it, c.max_dt);
            event = EV_CONVERGED;
            break;
        }
        if (num_sub_it >= c.max_it) {
            if (leader && st->nev < 8) {
                st->ev_it[st->nev] = num_it;
                st->ev_dt[st->nev] = dt;
                st->ev_diff[st->nev] = diff;
            }
            if (leader) st->nev += 1;
            dt = dt / 2;
            num_sub_it = 0;
            halved = true;
        }
        if (dt <= c.min_dt) { event = halved ? EV_STOP_HALVED : EV_STOP; break; }
        if (halved) { event = EV_HALVE; break; }
        if (refresh) { event = EV_REFRESH; break; }
    }
    __syncthreads();
    if (*err) event = EV_ERROR;
    if (event == EV_ERROR && producer && lane == 0) {
        // every copy this block issued lands before its shared memory is
        // released (bounded waits, flag ignored): the last issued use of each
        // stage
        atomicExch(&c.bar->error, 1);
        const unsigned first = issued > (unsigned)ring ? issued - ring : 0u;
        for (unsigned v = first; v < issued; ++v) mbar_wait_bounded(&full[ring0 + v % ring], (v / ring) & 1u);
    }
    // no block waits for another's last two phases, so the event is the last
    // block's to write.  (Another barrier at launches that end unchecked: 0.5 %
    // slower at 256 x 256 x 128, by the registers' allocation.)
    if (tid == 0) {
        bool failed = event == EV_ERROR;
        if (last_out(c.prog + kSegBase + kSegs * kSegWords, nb, failed)) st->event = failed ? EV_ERROR : event;
    }
    if (leader) {
        st->t = t;
        st->dt = dt;
        st->diff = diff;
        st->num_it = num_it;
        st->num_sub_it = num_sub_it;
        st->checkno = checkno;
        if (halved) st->halvings += 1;
        if (event == EV_CONVERGED) st->converged = 1;
    }
}

// copy the final state into the caller's status record
__global__ void dc_status_kernel(const DcState* st, TseSolveStatus* s) {
    s->t = st->t;
    s->dt = st->dt;
    s->diff = st->diff;
    s->converged = st->converged;
    s->num_it = st->num_it;
    s->num_sub_it = st->num_sub_it;
    s->halvings = st->halvings;
    s->error = st->event == EV_ERROR ? TSE_STATUS_BARRIER_TIMEOUT : TSE_STATUS_OK;
    s->n_events = st->nev < 8 ? st->nev : 8;
    for (int q = 0; q < 8; ++q) {
        s->ev_it[q] = st->ev_it[q];
        s->ev_dt[q] = st->ev_dt[q];
        s->ev_diff[q] = st->ev_diff[q];
    }
    s->cycles = st->cycles;
}

// ------------------------------------------------------------------ host
size_t dc_extra_bytes(const Layout& L) {
    const long long Ncal = (L.Nc + 31) & ~31LL;
    return 2 * ((size_t)k_floats(L) + (size_t)dc_delta_len(L, Ncal)) * sizeof(float) +
           align256(sizeof(DcState)) + 256 + align256(kProgBytes);
}

size_t dc_resident_bytes(const Layout& L) {
    return L.Nc <= kDcResMaxNc ? dc_res_bytes(L) : 0;
}

static int sweep_blocks(long long Nc, int cap) {
    static int cached_dev = -1, cached_per_sm = 0, cached_sms = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != cached_dev) {
        cudaDeviceGetAttribute(&cached_sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cached_per_sm, dc_sweep_kernel, kSweepBlock, 0);
        cached_dev = dev;
    }
    long long maxb = (long long)cached_sms * (cached_per_sm > 0 ? cached_per_sm : 1);
    long long want = (Nc + (long long)kSweepBlock * 4 - 1) / ((long long)kSweepBlock * 4);
    if (want < 1) want = 1;
    long long nb = want < maxb ? want : maxb;
    // the setup's partials region holds 2 * kMaxBlocks doubles
    if (nb > kMaxBlocks / 2) nb = kMaxBlocks / 2;
    if (cap > 0 && nb > cap) nb = cap;
    return (int)nb;
}

#ifndef TSE_SWEEP_TMA
#define TSE_SWEEP_TMA 1   // 1: bulk-copy staged sweeps where the stages fit in shared memory
#endif
// dynamic shared memory ceiling of the staged sweep: the device's per-block
// opt-in limit less the kernel's static arrays and a margin
static size_t tma_max_smem() {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return optin > 2048 ? (size_t)optin - 2048 : 0;
}

// blocks of the staged sweep: as many as fit (dynamic shared memory
// included), at most one per chunk of a colour; 0 when the stages for this
// grid's windows do not fit (the plain sweep kernel runs instead)
// the instantiation for rings of `ring` stages (2 .. 4), `pipes` pipelines
// per block (1: two blocks per SM) and chunks of `chunk` cells
template <int PIPES, int CHUNK, bool WIDE>
static const void* tma_kernel_r(int ring) {
    return ring <= 2 ? (const void*)dc_sweep_tma_kernel<2, PIPES, CHUNK, WIDE>
         : ring == 3 ? (const void*)dc_sweep_tma_kernel<3, PIPES, CHUNK, WIDE>
                     : (const void*)dc_sweep_tma_kernel<4, PIPES, CHUNK, WIDE>;
}
template <int PIPES, bool WIDE>
static const void* tma_kernel_c(int ring, int chunk) {
    return chunk == 256 ? tma_kernel_r<PIPES, 256, WIDE>(ring)
         : chunk == 1024 ? tma_kernel_r<PIPES, 1024, WIDE>(ring)
                         : tma_kernel_r<PIPES, 512, WIDE>(ring);
}
static const void* tma_kernel(int ring, int pipes, int chunk, bool wide) {
    return pipes == 1 ? tma_kernel_c<1, false>(ring, chunk)
         : wide ? tma_kernel_c<2, true>(ring, chunk)
                : tma_kernel_c<2, false>(ring, chunk);
}
// 16 consumer warps where a solve's records and corrections (33 bytes a cell)
// fit in L2
static bool tma_wide(long long Nc, int pipes) {
    int dev = 0, l2 = 0;
    if (pipes != 2 || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return 2 * Nc * 33 <= (long long)l2;
}

static int tma_blocks(long long Nc, int cap, size_t smem, const void* kernel, int threads, int chunk) {
    const size_t ceil_smem = tma_max_smem();
    if (!TSE_SWEEP_TMA || smem == 0 || smem > ceil_smem) return 0;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // the same ceiling for every grid, so concurrent callers never lower it
    // below another's launch
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ceil_smem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) !=
            cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        return 0;
    }
    long long nb = (long long)sms * per_sm;
    const long long nch = (Nc + chunk - 1) / chunk;
    if (nb > nch) nb = nch;
    if (nb > kMaxBlocks / 2) nb = kMaxBlocks / 2;
    if (cap > 0 && nb > cap) nb = cap;
    return nb < 1 ? 1 : (int)nb;
}

// the record blocks' cells: the chunk the call's options name (512 otherwise)
static int dc_block_log2(const TseDcOptions* opts) {
    return opts && opts->chunk == 256 ? 8 : opts && opts->chunk == 1024 ? 10 : 9;
}

// A lean setup's dt halving assembles again: again(dt, nparts).
struct NeverAgain {
    int operator()(double, int*) const { return TSE_ERR_LAUNCH; }
};
template <class Form, class Again = NeverAgain>
static int run_dc(SolveSetup<Form>& S, double dt, double inc_it, double max_dt, double min_dt,
                  double conv, int max_it, int pressure_schedule, int stop_on_first,
                  TseDcOptions* opts, double sor, int x_index, double* X_out,
                  TseSolveStatus* d_status, cudaStream_t stream, int first_parts,
                  Again again = Again()) {
    const int cycle = opts ? opts->cycle : 0;
    const int cap = opts ? opts->max_blocks : 0;
    if (S.tail_bytes < dc_extra_bytes(S.L)) return TSE_ERR_WORKSPACE;
    DcCtl c;
    dc_carve(S, c, x_index);
    c.inc_it = inc_it;
    c.max_dt = max_dt;
    c.min_dt = min_dt;
    c.conv = conv;
    c.max_it = max_it;
    c.pressure_schedule = pressure_schedule;
    c.stop_on_first = stop_on_first;
    c.cycle = cycle > 0 ? cycle : 256;
    c.sor = (float)sor;
    const bool timing = opts && opts->timing;
    // a grid that fits on the chip, and no staged variant asked for
    if (!S.lean && (!opts || (opts->chunk == 0 && opts->ring == 0 && opts->pipes == 0))) {
        const int rc = run_dc_resident(S, c, dt, cap, first_parts, X_out, d_status, timing ? opts : nullptr,
                                       stream);
        if (rc != 1) return rc;
    }
    const long long dlen = dc_delta_len(S.L, S.Ncal);
    float* dbase = c.D[0] - dc_margin(S.L);
    // the margins must read as 0 (kernels rewrite the interior only)
    if (cudaMemsetAsync(dbase, 0, (size_t)2 * dlen * sizeof(float), stream) != cudaSuccess)
        return TSE_ERR_LAUNCH;
    dc_init_state_kernel<<<1, 1, 0, stream>>>(c.st, dt);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    const long long cells2 = 2 * S.L.Nc;
    const unsigned gcells = (unsigned)((cells2 + kBlock - 1) / kBlock);
    // the staged sweep's variant: chunk size, pipelines per block and ring
    // length from the call's options (0: 512 cells, 2 pipelines, as many
    // stages as fit up to 4 a ring)
    const int chunk = 1 << S.ks;
    const int pipes = (opts && opts->pipes == 1) ? 1 : kDcPipes;
    const int want_ring = (opts && opts->ring >= 2 && opts->ring <= kDcMaxRing) ? opts->ring : kDcMaxRing;
    TmaStage T = tma_stage(S.L.H, chunk);
    {
        // one pipeline per block runs two blocks per SM: each gets half
        const size_t room = tma_max_smem() / (pipes == 1 ? 2 : 1);
        int st = (int)std::min<size_t>((size_t)(want_ring * pipes), room / (size_t)T.bytes);
        st -= st % pipes;
        T.stages = st >= 2 * pipes ? st : 0;
    }
    const size_t tma_smem = (size_t)T.stages * T.bytes;
    const bool wide = tma_wide(S.L.Nc, pipes);
    const int tma_threads = pipes == 1 ? DcLayout<1>::kThreads
                            : wide     ? DcLayout<2, true>::kThreads
                                       : DcLayout<2>::kThreads;
    const void* tma_k = T.stages > 0 ? tma_kernel(T.stages / pipes, pipes, chunk, wide) : nullptr;
    const int nb_tma = tma_k ? tma_blocks(S.L.Nc, cap, tma_smem, tma_k, tma_threads, chunk) : 0;
    if (opts) {
        // the variant that ran (0 when the plain-load sweep did)
        opts->chunk = nb_tma > 0 ? chunk : 0;
        opts->pipes = nb_tma > 0 ? pipes : 0;
        opts->ring = nb_tma > 0 ? T.stages / pipes : 0;
    }
    const int nb = nb_tma > 0 ? nb_tma : sweep_blocks(S.L.Nc, cap);
    if (nb_tma > 0) sweep_head(S.L, nb_tma, T);
    // the setup has written the records, r' and first_parts x^2 partials (the
    // first cycle's scale and residual).  A lean setup's two iterates take
    // turns, the later one in the arrays it leaves free.
    constexpr int kAlt = std::is_same<Form, TransportForm>::value ? (int)TA_XN : 0;
    double* alt[2] = {S.F.arr[0] + (size_t)kAlt * S.Ncal, S.F.arr[1] + (size_t)kAlt * S.Ncal};
    double* const x0[2] = {c.X[0], c.X[1]};
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    if (timing) {
        opts->sweep_launches = 0;
        opts->sweep_iterations = 0;
        opts->sweep_ms = 0.0;
        opts->loop_ms = 0.0;
        if (cudaEventCreate(&ev0) != cudaSuccess || cudaEventCreate(&ev1) != cudaSuccess)
            return TSE_ERR_LAUNCH;
    }
    int prev_it = 0;
    int rc = TSE_OK;
    bool final_apply = false;
    for (;;) {
        if (first_parts > 0) {
            dc_x2_kernel<<<1, kBlock, 0, stream>>>(c, first_parts, nb_tma > 0);
            first_parts = 0;
        } else {
            const unsigned rb = (unsigned)res_blocks(S.L.Nc);
            dc_residual_kernel<<<rb, kBlock, 0, stream>>>(S.F, c);
            dc_x2_kernel<<<1, kBlock, 0, stream>>>(c, (int)rb, nb_tma > 0);
        }
        void* args[] = {(void*)&c};
        void* targs[] = {(void*)&c, (void*)&T};
        if (timing) cudaEventRecord(ev0, stream);
        if (cudaGetLastError() != cudaSuccess) {
            rc = TSE_ERR_LAUNCH;
            break;
        }
        const cudaError_t le =
            nb_tma > 0 ? cudaLaunchCooperativeKernel(tma_k, dim3(nb),
                                                     dim3(tma_threads), targs, tma_smem, stream)
                       : cudaLaunchCooperativeKernel((const void*)dc_sweep_kernel, dim3(nb),
                                                     dim3(kSweepBlock), args, 0, stream);
        if (le != cudaSuccess) {
            rc = TSE_ERR_LAUNCH;
            break;
        }
        if (timing) cudaEventRecord(ev1, stream);
        // one read of the scalars (a pageable copy waits for the stream anyway)
        struct {
            double t, dt, diff, x2;
            int num_it, num_sub_it, halvings, converged, event;
        } head;
        static_assert(offsetof(DcState, event) == offsetof(decltype(head), event) &&
                          offsetof(DcState, num_it) == offsetof(decltype(head), num_it) &&
                          offsetof(DcState, dt) == offsetof(decltype(head), dt),
                      "DcState begins like this");
        if (cudaMemcpyAsync(&head, c.st, offsetof(DcState, event) + sizeof(int), cudaMemcpyDeviceToHost, stream) !=
                cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess) {
            rc = TSE_ERR_LAUNCH;
            break;
        }
        const int event = head.event;
        if (timing) {
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, ev0, ev1);
            opts->sweep_launches += 1;
            opts->sweep_iterations += head.num_it - prev_it;
            opts->sweep_ms += ms;
        }
        prev_it = head.num_it;
        if (S.lean && event == EV_STOP_HALVED) {
            // the caller's field still holds the entry state
            dc_status_kernel<<<1, 1, 0, stream>>>(c.st, d_status);
            if (timing) {
                cudaEventDestroy(ev0);
                cudaEventDestroy(ev1);
            }
            return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
        }
        if (S.lean && event == EV_HALVE) {
            if (cudaMemsetAsync(dbase, 0, (size_t)2 * dlen * sizeof(float), stream) != cudaSuccess ||
                again(head.dt, &first_parts) != TSE_OK) {
                rc = TSE_ERR_LAUNCH;
                break;
            }
            if (c.X[0] != x0[0]) {
                std::swap(c.X[0], alt[0]);
                std::swap(c.X[1], alt[1]);
            }
            continue;
        }
        if (event == EV_HALVE || event == EV_STOP_HALVED) {
            dc_halve_kernel<<<gcells, kBlock, 0, stream>>>(S.F, c);
            if (cudaGetLastError() != cudaSuccess) { rc = TSE_ERR_LAUNCH; break; }
            if (event == EV_STOP_HALVED) break;
            continue;
        }
        if (event == EV_ERROR) break;
        if (event == EV_CONVERGED || event == EV_STOP) {
            final_apply = true;   // x += d fused with the unpack below
            break;
        }
        if (S.lean) {
            const int rb = res_blocks(S.L.Nc);
            if constexpr (std::is_same<Form, TransportForm>::value)
                dc_apply_residual_kernel<<<(unsigned)rb, kBlock, 0, stream>>>(S.F, c, alt[0], alt[1]);
            std::swap(c.X[0], alt[0]);
            std::swap(c.X[1], alt[1]);
            first_parts = rb;
            if (cudaMemsetAsync(dbase, 0, (size_t)2 * dlen * sizeof(float), stream) != cudaSuccess ||
                cudaGetLastError() != cudaSuccess) {
                rc = TSE_ERR_LAUNCH;
                break;
            }
            continue;
        }
        dc_apply_kernel<<<gcells, kBlock, 0, stream>>>(c);
        if (cudaGetLastError() != cudaSuccess) { rc = TSE_ERR_LAUNCH; break; }
    }
    if (timing) {
        cudaEventDestroy(ev0);
        cudaEventDestroy(ev1);
    }
    if (rc != TSE_OK) return rc;
    dc_status_kernel<<<1, 1, 0, stream>>>(c.st, d_status);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    if (final_apply) {
        const long long nat = (long long)S.L.nx * S.L.ny * S.L.nz;
        dc_apply_unpack_kernel<<<(unsigned)((nat + kBlock - 1) / kBlock), kBlock, 0, stream>>>(X_out, c);
        return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
    }
    return launch_unpack(X_out, c.X[0], c.X[1], S.L, stream);
}

// ------------------------------------------- per-model steps, for batches
// The steps run_dc takes for one model, for drivers that interleave many
// models (tse_batch.cu): start (state record, zero margins, scaled records),
// residual (r', d = 0, x^2), halving (reset + new R terms + rescale), x += d,
// and finish (status record + natural-layout result).
template <class Form>
int dc_begin(const Form& F, const DcCtl& c, double dt, cudaStream_t stream) {
    float* dbase = c.D[0] - dc_margin(c.L);
    const long long dlen = dc_delta_len(c.L, c.Ncal);
    if (cudaMemsetAsync(dbase, 0, (size_t)2 * dlen * sizeof(float), stream) != cudaSuccess)
        return TSE_ERR_LAUNCH;
    dc_init_state_kernel<<<1, 1, 0, stream>>>(c.st, dt);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    const unsigned g = (unsigned)((2 * c.L.Nc + kBlock - 1) / kBlock);
    dc_scale_kernel<<<g, kBlock, 0, stream>>>(F, c);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

template <class Form>
int dc_residual(const Form& F, const DcCtl& c, cudaStream_t stream) {
    const unsigned rb = (unsigned)res_blocks(c.L.Nc);
    dc_residual_kernel<<<rb, kBlock, 0, stream>>>(F, c);
    dc_x2_kernel<<<1, kBlock, 0, stream>>>(c, (int)rb);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

template <class Form>
int dc_halve(const Form& F, const DcCtl& c, cudaStream_t stream) {
    const unsigned g = (unsigned)((2 * c.L.Nc + kBlock - 1) / kBlock);
    dc_halve_kernel<<<g, kBlock, 0, stream>>>(F, c);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

int dc_apply(const DcCtl& c, cudaStream_t stream) {
    const unsigned g = (unsigned)((2 * c.L.Nc + kBlock - 1) / kBlock);
    dc_apply_kernel<<<g, kBlock, 0, stream>>>(c);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

int dc_begin_fused(const DcCtl& c, double dt, int nparts, cudaStream_t stream) {
    float* dbase = c.D[0] - dc_margin(c.L);
    const long long dlen = dc_delta_len(c.L, c.Ncal);
    if (cudaMemsetAsync(dbase, 0, (size_t)2 * dlen * sizeof(float), stream) != cudaSuccess)
        return TSE_ERR_LAUNCH;
    dc_init_state_kernel<<<1, 1, 0, stream>>>(c.st, dt);
    dc_x2_kernel<<<1, kBlock, 0, stream>>>(c, nparts);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

int dc_finish(const DcCtl& c, TseSolveStatus* d_status, double* X_out, cudaStream_t stream) {
    dc_status_kernel<<<1, 1, 0, stream>>>(c.st, d_status);
    if (cudaGetLastError() != cudaSuccess) return TSE_ERR_LAUNCH;
    return launch_unpack(X_out, c.X[0], c.X[1], c.L, stream);
}

template int dc_begin<PressureForm>(const PressureForm&, const DcCtl&, double, cudaStream_t);
template int dc_begin<TransportForm>(const TransportForm&, const DcCtl&, double, cudaStream_t);
template int dc_residual<PressureForm>(const PressureForm&, const DcCtl&, cudaStream_t);
template int dc_residual<TransportForm>(const TransportForm&, const DcCtl&, cudaStream_t);
template int dc_halve<PressureForm>(const PressureForm&, const DcCtl&, cudaStream_t);
template int dc_halve<TransportForm>(const TransportForm&, const DcCtl&, cudaStream_t);

}  // namespace tse

using namespace tse;

// transport solves too large to be resident keep the later cycles' words only
static bool lean_grid(const TseGrid* grid) {
    return make_layout(grid->nx, grid->ny, grid->nz).Nc > kDcResMaxNc;
}

extern "C" int32_t tse_compute_P_dc(const TseGrid* grid, const TsePressureArgs* args,
                                    TseDcOptions* opts,
                                    TseSolveStatus* d_status, void* d_ws, size_t ws_bytes,
                                    void* stream_) {
    if (!grid || !args || !d_status || !d_ws) return TSE_ERR_ARG;
    if (grid->nx < 1 || grid->ny < 1 || grid->nz < 1 || args->max_it < 1) return TSE_ERR_ARG;
    if (!args->P || !args->Pn || !args->c_f || !args->nue || !args->rho_f || !args->phi ||
        !args->Kx || !args->Ky || !args->Kz || !args->c_r || !args->BP || !args->WP)
        return TSE_ERR_ARG;
    cudaStream_t stream = (cudaStream_t)stream_;
    PressureSetup S;
    S.ks = dc_block_log2(opts);
    int nparts = 0;
    int rc = setup_pressure_dc(grid, args, d_ws, ws_bytes, stream, S, &nparts);
    if (rc != TSE_OK) return rc;
    return run_dc(S, args->dt_P, args->inc_it, args->max_dt, args->min_dt, args->P_conv,
                  args->max_it, 1, 0, opts, args->SOR, PA_P, args->P, d_status, stream, nparts);
}

extern "C" int32_t tse_compute_C_dc(const TseGrid* grid, const TseSpeciesArgs* a,
                                    TseDcOptions* opts,
                                    TseSolveStatus* d_status, void* d_ws, size_t ws_bytes,
                                    void* stream_) {
    if (!grid || !a || !d_status || !d_ws) return TSE_ERR_ARG;
    if (grid->nx < 1 || grid->ny < 1 || grid->nz < 1 || a->max_it < 1) return TSE_ERR_ARG;
    if (!a->C || !a->D_fx || !a->D_fy || !a->D_fz || !a->phi || !a->rho_f || !a->qx || !a->qy ||
        !a->qz || !a->BC || !a->WC || !a->RC || !a->e || !a->l_l || !a->l_t)
        return TSE_ERR_ARG;
    cudaStream_t stream = (cudaStream_t)stream_;
    TransportSetup S;
    S.ks = dc_block_log2(opts);
    S.lean = lean_grid(grid);
    int nparts = 0;
    int rc = setup_species_dc(grid, a, d_ws, ws_bytes, stream, S, &nparts);
    if (rc != TSE_OK) return rc;
    auto again = [&](double dt, int* np) {
        TseSpeciesArgs half = *a;
        half.dt = dt;
        return again_species_dc(grid, &half, stream, S, np);
    };
    return run_dc(S, a->dt, a->inc_it, a->max_dt, a->min_dt, a->conv, a->max_it, 0,
                  a->omega == 0.0, opts, a->SOR, TA_X, a->C, d_status, stream, nparts, again);
}

extern "C" int32_t tse_compute_T_dc(const TseGrid* grid, const TseHeatArgs* a,
                                    TseDcOptions* opts,
                                    TseSolveStatus* d_status, void* d_ws, size_t ws_bytes,
                                    void* stream_) {
    if (!grid || !a || !d_status || !d_ws) return TSE_ERR_ARG;
    if (grid->nx < 1 || grid->ny < 1 || grid->nz < 1 || a->max_it < 1) return TSE_ERR_ARG;
    if (!a->T || !a->l_f || !a->cp_f || !a->rho_f || !a->phi || !a->qx || !a->qy || !a->qz ||
        !a->BT || !a->WT || !a->e || !a->l_r || !a->rho_r || !a->cp_r || !a->l_l || !a->l_t)
        return TSE_ERR_ARG;
    cudaStream_t stream = (cudaStream_t)stream_;
    TransportSetup S;
    S.ks = dc_block_log2(opts);
    S.lean = lean_grid(grid);
    int nparts = 0;
    int rc = setup_heat_dc(grid, a, d_ws, ws_bytes, stream, S, &nparts);
    if (rc != TSE_OK) return rc;
    auto again = [&](double dt, int* np) {
        TseHeatArgs half = *a;
        half.dt = dt;
        return again_heat_dc(grid, &half, stream, S, np);
    };
    return run_dc(S, a->dt, a->inc_it, a->max_dt, a->min_dt, a->conv, a->max_it, 0,
                  a->omega == 0.0, opts, a->SOR, TA_X, a->T, d_status, stream, nparts, again);
}
