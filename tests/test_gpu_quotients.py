"""The flux kernels' quotients and reciprocals (csrc/tse_quotient.cuh) against NumPy's divisions,
bit for bit, over the operands the kernels let through and what they derive from them."""
import ctypes as ct

import numpy
import pytest

from transportse_b200 import _native as N

pytestmark = pytest.mark.gpu


def _values(rng, n, e):
    """Magnitudes 2^-e .. 2^e: random significands, and those beside 1, 2 and their middle."""
    m = rng.uniform(1.0, 2.0, n)
    for v in (1.0, 1.5, numpy.nextafter(1.0, 2), numpy.nextafter(2.0, 1), numpy.nextafter(1.5, 1),
              numpy.nextafter(numpy.nextafter(2.0, 1), 1)):
        m[rng.uniform(size=n) < 0.05] = v
    x = numpy.ldexp(m, rng.integers(-e, e + 1, n))
    x[:8] = [2.0 ** -e, 2.0 ** e, numpy.nextafter(2.0 ** -e, 1), numpy.nextafter(2.0 ** e, 0), 1.0, 2.0,
             numpy.nextafter(2.0, 1), numpy.nextafter(1.0, 0)]
    return x


# operands as they come in; sums of quotients of such; harmonic means and their products
@pytest.mark.parametrize("eb,ea", [(80, 80), (80, 300), (161, 161), (241, 780)])
def test_quotients_are_the_divided_ones(eb, ea, cuda_device):
    import torch
    rng = numpy.random.default_rng(eb + ea)
    n = 1 << 21
    b = _values(rng, n, eb)
    a = _values(rng, n, ea) * rng.choice((-1.0, 1.0), n)
    a[rng.uniform(size=n) < 0.01] = 0.0
    a[rng.uniform(size=n) < 0.01] = -0.0
    # exact and nearly exact quotients
    k = rng.uniform(size=n) < 0.1
    a[k] = b[k] * rng.integers(1, 1000, k.sum())
    da, db = (torch.as_tensor(x, device=cuda_device) for x in (a, b))
    q, y = torch.empty_like(da), torch.empty_like(da)
    p = lambda t: ct.c_void_p(t.data_ptr())
    rc = N.lib().tse_selftest_quotients(p(da), p(db), p(q), p(y), n,
                                        ct.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream))
    assert rc == 0
    bits = lambda x: numpy.ascontiguousarray(x).view(numpy.int64)
    assert numpy.array_equal(bits(y.cpu().numpy()), bits(1.0 / b))
    assert numpy.array_equal(bits(q.cpu().numpy()), bits(a / b))
