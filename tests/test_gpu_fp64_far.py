"""FP64 energies of poses so far away (1e12 A and more) that powers of the distance
leave the range of double, against pockets with and without padding points: finite,
and those of the FP64 oracle."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_PREC_FP64
from oracle import tolerance as TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e11, 1e13, 1e20, 1e30, 1e37])
@pytest.mark.parametrize("points", [200, 256])
def test_fp64_far_poses(lib, enepara, oracle_lib, points, far):
    rng = np.random.default_rng(8)
    pk = synth.make_pocket(rng, points, 1)
    job = synth.make_job(rng, pk, 13, 1, 60, 3, [1.0], seed=2)
    cx = synth.to_complex(job, pk, enepara)
    mm = synth.config4_poses(3, 12, radius=5.0)
    mm[::2, 0] += np.float32(far)
    _, _, out64 = dock.eval_poses(cx, np.zeros((12, 2), np.int32), mm, GD_PREC_FP64, want64=True)
    ref = np.array([oracle_lib.energy(cx, 0, 0, m)[0] for m in mm])
    assert np.isfinite(ref).all() and np.isfinite(out64).all()
    # the FP64 kernel's tolerance; terms 4 and 6 carry the reference's float constants (and the total with them)
    err = np.abs(out64 - ref) / np.maximum(np.abs(ref), TOL.TAU)
    assert np.delete(err, [4, 6, 9], axis=1).max() <= 1e-9
    assert err.max() <= 2e-7
