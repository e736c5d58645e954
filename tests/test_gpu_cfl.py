"""The CFL limit where porosities or spacings are not the usual positive numbers; the largest
shape gives a warp several cells, so that a maximum meets further candidates."""
import numpy
import pytest

from oracle.oracle import OracleModel
from tests.helpers import model_for

pytestmark = pytest.mark.gpu


def _case(shape, seed):
    from transportse_b200 import workloads
    rng = numpy.random.default_rng(seed)
    cfg = workloads.base_config("cfl", *shape, *(rng.uniform(0.5, 2, n) for n in shape))
    q = [rng.uniform(-1e-5, 1e-5, shape) * 10.0 ** rng.integers(-4, 4, shape) for _ in range(3)]
    return cfg, rng, q, rng.uniform(0.05, 0.3, shape)


@pytest.mark.parametrize("shape", [(5, 1, 3), (33, 17, 21), (120, 101, 91), (170, 160, 150)])
@pytest.mark.parametrize("kind", ["all negative", "some negative", "spacings", "tiny", "huge", "underflow"])
def test_cfl_of_unusual_operands_equals_the_oracle(kind, shape, cuda_device):
    """Every quotient's sign and rounding counts: a maximum of negative
    quotients, one that only a rounded-up subnormal reaches, products beyond
    either end of the range."""
    cfg, rng, q, phi = _case(shape, sum(shape))
    if kind == "all negative":
        phi = -phi
    elif kind == "some negative":
        phi = numpy.where(rng.uniform(size=shape) < 0.5, -phi, phi)
    elif kind == "spacings":
        cfg.dx, cfg.dz = -cfg.dx, cfg.dz * 1e-200
    elif kind == "tiny":
        phi = phi * 10.0 ** rng.integers(-170, -100, shape)
        cfg.dy = cfg.dy * 1e-160
    elif kind == "huge":
        phi = phi * 10.0 ** rng.integers(100, 300, shape)
        q = [x * 1e290 for x in q]
    else:
        q = [x * 1e-315 for x in q]
        cfg.dx, cfg.dy, cfg.dz = cfg.dx * 1e-306, cfg.dy * 1e-306, cfg.dz * 1e-306
    with numpy.errstate(all="ignore"):
        want = OracleModel(cfg).dt_cfl(*q, phi)
    assert numpy.array_equal(model_for(cfg, cuda_device).dt_cfl(*q, phi), want, equal_nan=True)
