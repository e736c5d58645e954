"""Transport solves whose divisors are at the ends of the exponent range: a steady state
(an infinite dt), a spacing whose square overflows.  One iteration each (a tolerance no
change fails), mixed precision against FP64: resident, streamed and lean assemblies."""
import numpy
import pytest

from tests.helpers import NumpyKernels, model_for

pytestmark = pytest.mark.gpu


def _solve(cfg, device, precision, heat, dt, omega, f):
    nk = NumpyKernels(model_for(cfg, device, precision))
    kw = dict(omega=omega, SOR=1.1, max_it=100, inc_it=1.05, max_dt=1e5, min_dt=1e-8)
    with numpy.errstate(all="ignore"):
        if heat:
            return nk.compute_T(f["T"].copy(), 0.6 * f["one"], 4180.0 * f["one"], f["rho"], f["phi"], *f["q"], dt,
                                f["B"], f["W"], f["e"], T_conv=2.0, **kw)
        return nk.compute_C(f["C"].copy(), f["D"], f["D"], f["D"], f["phi"], f["rho"], *f["q"], dt, f["B"], f["W"],
                            f["one"], f["e"], C_conv=2.0, **kw)


@pytest.mark.parametrize("heat", [False, True])
@pytest.mark.parametrize("shape", [(24, 20, 17), (100, 100, 93), (130, 127, 64)])
@pytest.mark.parametrize("dt,wide", [(numpy.inf, 1.0), (1.7e308, 1.0), (600.0, 1e200), (numpy.inf, 1e200)])
def test_divisors_at_the_ends_of_the_range(shape, heat, dt, wide, cuda_device):
    from transportse_b200 import workloads
    rng = numpy.random.default_rng(sum(shape))
    cfg = workloads.base_config("steady", *shape, *(rng.uniform(0.5, 2, n) for n in shape))
    cfg.dx = numpy.where(numpy.arange(shape[0]) == 3, cfg.dx * wide, cfg.dx)
    cfg.lf_l[:], cfg.lf_t[:] = 0.5, 0.1
    cfg.l_r[:], cfg.rho_r[:], cfg.cp_r[:] = rng.uniform(1.5, 3.5, shape), 2650.0, 900.0
    f = dict(C=rng.uniform(0, 1, shape), T=rng.uniform(15, 80, shape), D=1e-6 * rng.uniform(0.5, 1.5, shape),
             B=(rng.uniform(size=shape) < 0.1).astype(float), W=numpy.zeros(shape),
             e=rng.uniform(-1e-9, 1e-9, shape), q=[rng.uniform(-1e-7, 1e-7, shape) for _ in range(3)],
             one=numpy.ones(shape), phi=rng.uniform(0.05, 0.3, shape), rho=rng.uniform(995, 1150, shape))
    for omega in (1.0, 0.5):
        a = _solve(cfg, cuda_device, "fp32dc", heat, dt, omega, f)
        b = _solve(cfg, cuda_device, "fp64", heat, dt, omega, f)
        assert (a[0], a[1], a[3], a[4]) == (b[0], b[1], b[3], b[4]) and a[4] == 1
        assert numpy.isfinite(b[2]).all()
        # a correction is formed in FP32: seven roundings of values up to the change
        change = numpy.abs(b[2] - (f["T"] if heat else f["C"])).max()
        assert numpy.abs(a[2] - b[2]).max() <= 1e-6 * change + 1e-12 * numpy.abs(b[2]).max()
