"""The resident mixed-precision solve (csrc/tse_dc_resident.cuh) against the staged sweeps.

The resident kernel makes the staged sweep's cell updates operation for operation, so a
solve's fields, iteration counts and dt are the same bits whichever runs: on one block, one
cluster and the whole GPU, at the sizes where the tiling changes (largest tile of either
instance, columns that do not fill their last group, single rows and columns), through
cycle ends, refreshes, dt halvings and stops, and with the blocks capped."""
import numpy
import pytest

from tests.helpers import NumpyKernels, model_for

pytestmark = pytest.mark.gpu

STAGED = (512, 4, 2)
# (shape, whether it is small enough to be resident): one block of 512 and of 768 groups,
# the smallest and the largest cluster, the first whole-GPU tilings, its largest, too large
SHAPES = [((16, 16, 16), True), ((16, 16, 24), True), ((17, 16, 24), True), ((44, 44, 46), True),
          ((45, 47, 46), True), ((33, 17, 21), True), ((96, 96, 64), True), ((96, 96, 96), True),
          ((100, 100, 100), False), ((1, 1, 1), True), ((1, 1, 4000), True), ((1, 90, 70), True),
          ((200, 1, 3), True), ((5, 7, 2), True)]


def _case(shape, seed):
    from transportse_b200 import workloads
    rng = numpy.random.default_rng(seed)
    cfg = workloads.base_config("res", *shape, rng.uniform(0.5, 2, shape[0]), rng.uniform(0.5, 2, shape[1]),
                                rng.uniform(0.5, 2, shape[2]))
    cfg.beta = 3.0
    cfg.c_r[:] = 1e-10
    K = 1e-12 * numpy.exp(rng.standard_normal(shape))
    args = (4.5e-10 * numpy.ones(shape), rng.uniform(8e-4, 1.2e-3, shape), rng.uniform(995, 1150, shape),
            rng.uniform(0.05, 0.3, shape), K, 0.7 * K, 0.3 * K)
    P = workloads.hydrostatic(cfg) + rng.uniform(-300, 300, shape)
    BP = (rng.uniform(size=shape) < 0.02).astype(float)
    BP.reshape(-1)[0] = 1.0
    WP = numpy.where(rng.uniform(size=shape) < 0.2, rng.uniform(-1e-4, 1e-4, shape), 0.0)
    return cfg, rng, args, P, BP, WP


def _both(cfg, device, call, max_blocks=0, cycle=None):
    out = []
    for variant in ((0, 0, 0), STAGED):
        m = model_for(cfg, device, "fp32dc")
        m.sweep_variant = variant
        m.max_blocks = max_blocks
        if cycle:
            m.dc_cycle = cycle
        out.append((call(NumpyKernels(m)), m.last_variant, m.last_status))
    return out


def _same(a, b):
    for x, y in zip(a, b):
        if isinstance(x, numpy.ndarray):
            assert numpy.array_equal(x, y, equal_nan=True)
        else:
            assert x == y


@pytest.mark.parametrize("shape,resident", SHAPES)
def test_pressure_solve_equals_the_staged_form(shape, resident, cuda_device):
    cfg, rng, args, P, BP, WP = _case(shape, sum(shape))
    z = numpy.zeros(shape)

    def call(nk):
        return nk.compute_P(P.copy(), *args, z, z, z, 3600.0, BP, WP, SOR=1.7, max_it=20000, inc_it=1.25,
                            max_dt=1e5, min_dt=1e-8, P_conv=1e-10)

    (r, ran, st), (s, _, ss) = _both(cfg, cuda_device, call)
    assert (ran == (0, 0, 0)) == resident
    _same(r, s)
    assert (st.cycles, st.num_sub_it, st.halvings) == (ss.cycles, ss.num_sub_it, ss.halvings)
    assert r[4] and (r[5] > 50 or min(shape) == 1)


@pytest.mark.parametrize("shape", [(16, 16, 24), (33, 17, 21), (60, 50, 41)])
@pytest.mark.parametrize("max_blocks", [0, 5])
def test_cycles_halvings_and_stops_equal_the_staged_form(shape, max_blocks, cuda_device):
    """Cycles of 30 iterations; a solve that halves dt until it converges or
    falls below min_dt; a NaN in the pressure."""
    cfg, rng, args, P, BP, WP = _case(shape, 3)
    z = numpy.zeros(shape)
    bad = P.copy()
    bad[shape[0] // 2, 3, 4] = numpy.nan

    def call(p0, max_it, min_dt):
        return lambda nk: nk.compute_P(p0.copy(), *args, z, z, z, 3600.0, BP, WP, SOR=1.7, max_it=max_it,
                                       inc_it=1.25, max_dt=1e5, min_dt=min_dt, P_conv=1e-10)

    for p0, max_it, min_dt in ((P, 20000, 1e-8), (P, 75, 1.0), (P, 7, 400.0), (bad, 12, 1000.0)):
        (r, _, st), (s, _, ss) = _both(cfg, cuda_device, call(p0, max_it, min_dt), max_blocks, 30)
        _same(r, s)
        assert (st.cycles, st.num_sub_it, st.halvings, st.n_events) == (ss.cycles, ss.num_sub_it, ss.halvings,
                                                                        ss.n_events)
        assert list(st.ev_it[:st.n_events]) == list(ss.ev_it[:ss.n_events])


@pytest.mark.parametrize("shape", [(16, 16, 24), (31, 20, 27), (64, 64, 50)])
@pytest.mark.parametrize("omega", [1.0, 0.5, 0.0])
def test_transport_solves_equal_the_staged_form(shape, omega, cuda_device):
    cfg, rng, args, P, BP, WP = _case(shape, 8)
    cfg.lf_l[:] = rng.uniform(0, 1, shape)
    cfg.lf_t[:] = rng.uniform(0, 0.3, shape)
    cfg.l_r[:] = rng.uniform(1.5, 3.5, shape)
    cfg.rho_r[:], cfg.cp_r[:] = 2650.0, 900.0
    cfg.C_IMBLFLO = cfg.T_IMBLFLO = True
    C, T = rng.uniform(0, 1, shape), rng.uniform(15, 80, shape)
    D = 1e-6 * rng.uniform(0.5, 1.5, shape)
    B = (rng.uniform(size=shape) < 0.1).astype(float)
    W = numpy.where(rng.uniform(size=shape) < 0.2, 1e-5, 0.0)
    e = rng.uniform(-1e-6, 1e-6, shape)
    q = [rng.uniform(-1e-4, 1e-4, shape) for _ in range(3)]
    one = numpy.ones(shape)
    kw = dict(omega=omega, SOR=1.1, max_it=100, inc_it=1.05, max_dt=1e5, min_dt=1e-8)

    def species(nk):
        return nk.compute_C(C.copy(), D, D, D, args[3], args[2], *q, 600.0, B, W, one, e, C_conv=1e-11, **kw)

    def heat(nk):
        m = nk.m
        r = m.compute_T(T.copy(), 0.6 * one, 4180.0 * one, args[2], args[3], *q, 600.0, B, W, e, T_conv=1e-11,
                        **kw)
        return (r[0], r[1], r[2].cpu().numpy(), r[3], r[4])

    for call in (species, heat):
        (r, ran, _), (s, _, _) = _both(cfg, cuda_device, call)
        assert ran == (0, 0, 0)
        _same(r, s)


# FP64: one block (at most 480 groups of two cells), clusters, the whole GPU, too large
EXACT = [((12, 10, 16), True), ((11, 11, 16), True), ((24, 24, 24), True), ((33, 17, 21), True),
         ((48, 48, 48), True), ((60, 52, 60), True), ((80, 80, 80), False), ((1, 1, 1), True),
         ((1, 1, 900), True), ((1, 60, 30), True), ((200, 1, 3), True), ((5, 7, 2), True)]


@pytest.mark.parametrize("shape,resident", EXACT)
def test_exact_solves_equal_the_streaming_kernels(shape, resident, cuda_device):
    """FP64 pressure and species solves (x and z buoyancy, omega < 1, the
    IMBLFLO term), resident, staged and with plain loads: the same bits; and
    dt halvings, a stop at min_dt and a NaN."""
    import ctypes as ct
    from transportse_b200 import _native as N
    cfg, rng, args, P, BP, WP = _case(shape, 21)
    cfg.lf_l[:] = rng.uniform(0, 1, shape)
    cfg.lf_t[:] = rng.uniform(0, 0.3, shape)
    cfg.C_IMBLFLO = True
    C = rng.uniform(0, 1, shape)
    D = 1e-6 * rng.uniform(0.5, 1.5, shape)
    B = (rng.uniform(size=shape) < 0.1).astype(float)
    W = numpy.where(rng.uniform(size=shape) < 0.2, 1e-5, 0.0)
    e = rng.uniform(-1e-6, 1e-6, shape)
    q = [rng.uniform(-1e-4, 1e-4, shape) for _ in range(3)]
    one, z = numpy.ones(shape), numpy.zeros(shape)
    bad = P.copy()
    bad.reshape(-1)[-1] = numpy.nan
    m = model_for(cfg, cuda_device)
    # the workspace carries the exchange records just where the form may run
    plain = N.lib().tse_workspace_bytes(ct.byref(m.grid), N.TSE_WS_PRESSURE)
    assert m.ws_bytes >= plain
    nk = NumpyKernels(m)
    out = []
    for mode in (0, 2, 1):
        m.sweep = mode
        got = []
        for p0, max_it, min_dt in ((P, 20000, 1e-8), (P, 40, 1.0), (P, 7, 400.0), (bad, 12, 1000.0)):
            r = nk.compute_P(p0.copy(), *args, z, z, z, 3600.0, BP, WP, SOR=1.7, max_it=max_it, inc_it=1.25,
                             max_dt=1e5, min_dt=min_dt, P_conv=1e-10)
            s = m.last_status
            got += [*r, s.num_sub_it, s.halvings, s.n_events]
        for omega in (1.0, 0.5, 0.0):
            got += [*nk.compute_C(C.copy(), D, D, D, args[3], args[2], *q, 600.0, B, W, one, e, omega=omega,
                                  SOR=1.1, max_it=100, inc_it=1.05, max_dt=1e5, min_dt=1e-8, C_conv=1e-11)]
        out.append(got)
    _same(out[0], out[1])
    _same(out[0], out[2])


# cells of a colour: one block's threads and one more pair, every SM's threads and more
@pytest.mark.parametrize("shape", [(16, 16, 6), (16, 16, 8), (37, 96, 64), (111, 64, 32), (111, 64, 34), (5, 211, 431)])
def test_plain_loads_ahead_of_the_barrier_equal_the_staged_kernel(shape, cuda_device):
    """The plain-load FP64 kernel, whose threads load their first cell of the
    next half-sweep before the barrier, against the staged one: convergence,
    dt halvings, stops, omega < 1; and whichever of them the size selects."""
    cfg, rng, args, P, BP, WP = _case(shape, 5)
    C, D, one, z = rng.uniform(0, 1, shape), 1e-6 * rng.uniform(0.5, 1.5, shape), numpy.ones(shape), numpy.zeros(shape)
    q = [rng.uniform(-1e-4, 1e-4, shape) for _ in range(3)]
    m = model_for(cfg, cuda_device)
    nk, out = NumpyKernels(m), []
    for mode in (0, 1, 2):
        m.sweep, got = mode, []
        for max_it, min_dt in ((20000, 1e-8), (40, 1.0), (7, 400.0)):
            got += [*nk.compute_P(P.copy(), *args, z, z, z, 3600.0, BP, WP, SOR=1.7, max_it=max_it, inc_it=1.25,
                                  max_dt=1e5, min_dt=min_dt, P_conv=1e-10), m.last_status.halvings]
        for omega in (1.0, 0.5, 0.0):
            got += [*nk.compute_C(C.copy(), D, D, D, args[3], args[2], *q, 600.0, BP, WP, one, z, omega=omega, SOR=1.1,
                                  max_it=100, inc_it=1.05, max_dt=1e5, min_dt=1e-8, C_conv=1e-11)]
        out.append(got)
    _same(out[0], out[1])
    _same(out[0], out[2])
