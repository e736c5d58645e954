"""The flow error's walks of grids from two million cells on (four blocks a SM) against the
oracle, bit for bit, operands at the ends of the range included."""
import numpy
import pytest

from oracle.oracle import OracleModel
from tests.helpers import NumpyKernels, model_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extremes", [False, True])
@pytest.mark.parametrize("shape", [(130, 127, 124), (3, 850, 803), (33000, 2, 31)])
def test_flow_error_of_large_grids(shape, extremes, cuda_device):
    from transportse_b200 import workloads
    rng = numpy.random.default_rng(sum(shape))
    cfg = workloads.base_config("flow", *shape, *(rng.uniform(0.5, 2, n) for n in shape))
    cfg.c_r[:] = 1e-10

    def spread(x):
        if extremes:
            for v in (0.0, -0.0, 1e-310, 3e-200, 7e250, numpy.inf, numpy.nan, 1.0):
                x[rng.uniform(size=shape) < 0.004] = v
        return x

    rho, phi = spread(rng.uniform(995, 1150, shape)), spread(rng.uniform(0.05, 0.3, shape))
    c_f, P = spread(4.5e-10 * rng.uniform(0.5, 1.5, shape)), spread(1e5 + 300 * rng.standard_normal(shape))
    Pn = P + rng.standard_normal(shape)
    WP = numpy.where(rng.uniform(size=shape) < 0.2, rng.uniform(-1e-4, 1e-4, shape), 0.0)
    q = [spread(rng.uniform(-1e-5, 1e-5, shape) * 10.0 ** rng.integers(-12, 6, shape)) for _ in range(3)]
    args = (P, Pn, *q, WP, phi, c_f, cfg.c_r, rho, 3600.0)
    with numpy.errstate(all="ignore"):
        want = OracleModel(cfg).flow_error(*args)
    got = NumpyKernels(model_for(cfg, cuda_device)).flow_error(*args)
    real = ~numpy.isnan(want)
    assert numpy.array_equal(got, want, equal_nan=True)
    assert numpy.array_equal(numpy.signbit(got)[real], numpy.signbit(want)[real])
