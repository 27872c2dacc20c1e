"""The FP64 pair loop's own reciprocals, square root and exponential at the ends
of their ranges: atoms on, next to and far from points (to 1e5 A), pairs whose
pmf exponent under- and overflows double, against the FP64 oracle."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_PREC_FP64
from oracle import tolerance as TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [0.0, 1e2, 1e5])
@pytest.mark.parametrize("pmf0", [None, 60.0, -200.0])
def test_fp64_ends_of_range(lib, enepara, oracle_lib, far, pmf0):
    rng = np.random.default_rng(8)
    pk = synth.make_pocket(rng, 200, 1)
    job = synth.make_job(rng, pk, 13, 1, 60, 3, [1.0], seed=2)
    ep = enepara.copy()
    if pmf0 is not None:  # (6 - d/2)(d - pmf0) beyond +-745 within the pocket's distances
        ep["pmf0"][:] = np.float32(pmf0)
    cx = synth.to_complex(job, pk, ep)
    mm = synth.config4_poses(3, 24, radius=5.0)
    mm[12:, 0] += np.float32(far)
    # an atom 1e-3 A from a point
    mm[0, :3] = pk.xyz[0, 5] - job.lig_xyz[0, 2] - job.lig_center[0] + np.float32(1e-3)
    mm[0, 3:] = 0
    conf = np.zeros((24, 2), np.int32)
    _, _, out64 = dock.eval_poses(cx, conf, mm, GD_PREC_FP64, want64=True)
    ref = np.array([oracle_lib.energy(cx, 0, 0, m)[0] for m in mm])
    assert np.isfinite(ref).all() and np.isfinite(out64).all()
    # the FP64 kernel's tolerance; terms 4 and 6 carry the reference's float constants (and the total with them)
    err = np.abs(out64 - ref) / np.maximum(np.abs(ref), TOL.TAU)
    assert np.delete(err, [4, 6, 9], axis=1).max() <= 1e-9
    assert err.max() <= 2e-7


def test_fp64_coincident_atom_and_point(lib, enepara):
    """Exactly on a point: every term is the limit at d -> 0, finite."""
    rng = np.random.default_rng(9)
    pk = synth.make_pocket(rng, 100, 1)
    job = synth.make_job(rng, pk, 1, 1, 10, 1, [1.0], seed=2)
    job.lig_xyz[:] = 0
    job.lig_center[:] = 0
    pk.xyz[0, 7] = (1.0, 2.0, 3.0)
    cx = synth.to_complex(job, pk, enepara)
    mm = np.array([[1.0, 2.0, 3.0, 0, 0, 0], [1.0, 2.0, np.nextafter(np.float32(3.0), np.float32(4.0)), 0, 0, 0]],
                  np.float32)
    _, _, out64 = dock.eval_poses(cx, np.zeros((2, 2), np.int32), mm, GD_PREC_FP64, want64=True)
    assert np.isfinite(out64).all()
    np.testing.assert_allclose(out64[0, :4], out64[1, :4], rtol=1e-4, atol=1e-4)
