"""Which FP64 kernel a solve runs on, and that the three agree bit for bit: plain loads, bulk-copy
staged (rings of two stages and stages that do not fit included), resident."""
import numpy
import pytest

from tests.helpers import NumpyKernels, model_for
from transportse_b200._native import TSE_SWEEP_PLAIN as PLAIN
from transportse_b200._native import TSE_SWEEP_RESIDENT as RESIDENT
from transportse_b200._native import TSE_SWEEP_STAGED as STAGED

pytestmark = pytest.mark.gpu

# shape; the kernels of a pressure solve with sweep 0 and 2 (1 is plain) and of a species
# solve.  (3, 2, 1000): rings of two stages; (1, 2, 3000): a column too long for a
# block's shared memory, and the pressure solve's stages fit no ring; grids whose state does
# not fit the SMs' shared memory; either side of a million cells of a colour
CASES = [((64, 48, 40), (RESIDENT, STAGED), (RESIDENT, STAGED)),
         ((37, 23, 51), (RESIDENT, STAGED), (RESIDENT, STAGED)),
         ((3, 2, 1000), (RESIDENT, STAGED), (RESIDENT, STAGED)),
         ((1, 2, 3000), (PLAIN, PLAIN), (PLAIN, STAGED)),
         ((1, 1, 1), (RESIDENT, STAGED), (RESIDENT, STAGED)),
         ((72, 72, 71), (PLAIN, STAGED), (PLAIN, STAGED)),
         ((96, 96, 64), (PLAIN, STAGED), (PLAIN, STAGED)),
         ((125, 128, 124), (PLAIN, STAGED), (PLAIN, STAGED)),
         ((125, 128, 126), (STAGED, STAGED), (STAGED, STAGED))]


@pytest.mark.parametrize("shape,pressure,species", CASES)
def test_the_chosen_kernel_runs_and_all_agree(shape, pressure, species, cuda_device):
    from transportse_b200 import workloads
    rng = numpy.random.default_rng(sum(shape))
    cfg = workloads.base_config("fp64", *shape, *(rng.uniform(0.5, 2, n) for n in shape))
    cfg.beta = 3.0
    cfg.c_r[:] = 1e-10
    cfg.lf_l[:], cfg.lf_t[:] = rng.uniform(0, 1, shape), rng.uniform(0, 0.3, shape)
    cfg.C_IMBLFLO = True
    K = 1e-12 * numpy.exp(rng.standard_normal(shape))
    phi, rho = rng.uniform(0.05, 0.3, shape), rng.uniform(995, 1150, shape)
    args = (4.5e-10 * numpy.ones(shape), rng.uniform(8e-4, 1.2e-3, shape), rho, phi, K, 0.7 * K, 0.3 * K)
    P = workloads.hydrostatic(cfg) + rng.uniform(-300, 300, shape)
    BP = (rng.uniform(size=shape) < 0.05).astype(float)
    BP.reshape(-1)[0] = 1.0
    WP = numpy.where(rng.uniform(size=shape) < 0.2, rng.uniform(-1e-4, 1e-4, shape), 0.0)
    C, D = rng.uniform(0, 1, shape), 1e-6 * rng.uniform(0.5, 1.5, shape)
    e, one, z = rng.uniform(-1e-6, 1e-6, shape), numpy.ones(shape), numpy.zeros(shape)
    q = [rng.uniform(-1e-4, 1e-4, shape) for _ in range(3)]
    m = model_for(cfg, cuda_device)
    nk, out = NumpyKernels(m), []
    for mode in (0, 1, 2):
        m.sweep = mode
        p = nk.compute_P(P.copy(), *args, z, z, z, 3600.0, BP, WP, SOR=1.7, max_it=20000, inc_it=1.25, max_dt=1e5,
                         min_dt=1e-8, P_conv=1e-7)
        ran = [m.last_status.sweep]
        c = [nk.compute_C(C.copy(), D, D, D, phi, rho, *q, 3600.0, BP, WP, one, e, omega=om, SOR=1.1, max_it=100,
                          inc_it=1.05, max_dt=1e5, min_dt=1e-8, C_conv=1e-12) for om in (1, 0.5)]
        ran.append(m.last_status.sweep)
        assert ran == [PLAIN, PLAIN] if mode == 1 else ran == [pressure[mode // 2], species[mode // 2]]
        out.append([p, *c])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            for x, y in zip(a, b):
                assert numpy.array_equal(x, y, equal_nan=True)
