"""The FP64 pair loop's reciprocal, square root and exponential against 80-bit
arithmetic, over the ranges their arguments have (through the bounds-checking build,
which exports them)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(x, z):
    import torch

    from geauxdock_b200 import build

    lib = C.CDLL(str(build.CHECK_LIB))
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, z)]
    out = torch.zeros((len(x), 5), dtype=torch.float64, device="cuda")
    rc = lib.gd_check_math64(len(x), *(C.c_void_p(t.data_ptr()) for t in (*d, out)))
    assert rc == 0
    return out.cpu().numpy()


def _rel(got, want):
    return float(np.max(np.abs((got.astype(np.longdouble) - want) / want)))


def test_errors(lib):
    """Half an ulp of the last operation (1.11e-16) and, for each, what the operations before it leave: the third
    power of the approximation's 1e-6 (rcp), half the rounding of the product before (d, its reciprocal); of the
    exponential the rounding of exp(r) - 1 (2e-19) and the series' remainder (1e-17), and without the table's second
    part half an ulp more."""
    rng = np.random.default_rng(1)
    n = 1 << 20
    x = (1 + 3 * rng.random(n)) * np.array([1e-2, 1.0, 64.0, 4096.0, 1e9, 1e30, 1e70, 1e-300])[np.arange(n) % 8]
    z = np.where(np.arange(n) % 2, rng.uniform(-60, 10, n), rng.uniform(-700, 700, n))
    z[:512] = np.log(2) / 512 * (np.arange(512) - 256 + 0.5)  # the ends of the table's intervals
    o = _call(x, z)
    xl, el = x.astype(np.longdouble), np.exp(z.astype(np.longdouble))
    assert _rel(o[:, 0], 1 / xl) <= 1.12e-16
    assert _rel(o[:, 1], np.sqrt(xl)) <= 1.7e-16
    assert _rel(o[:, 2], 0.5 / np.sqrt(xl)) <= 1.7e-16
    assert _rel(o[:, 3], el) <= 1.3e-16
    assert _rel(o[:, 4], el) <= 2.4e-16


def test_ends_of_range(lib):
    z = np.array([0.0, -0.0, 701.0, np.inf, -701.0, -np.inf, np.nan, -1e300])
    o = _call(np.ones(8), z)
    for e in (o[:, 3], o[:, 4]):
        assert e[:2].tolist() == [1.0, 1.0]
        assert e[2:4].tolist() == [2.0**1000] * 2  # whose reciprocal is as good as 0
        assert e[4:6].tolist() == [0.0] * 2 and np.isnan(e[6]) and e[7] == 0
