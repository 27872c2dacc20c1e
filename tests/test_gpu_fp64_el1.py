"""The near field of the electrostatic term in FP64 is where el1 d < 1, for any el1."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_PREC_FP64
from oracle import tolerance as TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("el1", [0.5, 0.07, 3.0, -0.5])
def test_fp64_near_field(lib, enepara, oracle_lib, el1):
    rng = np.random.default_rng(8)
    pk = synth.make_pocket(rng, 200, 1)
    job = synth.make_job(rng, pk, 13, 1, 60, 3, [1.0], seed=2)
    ep = enepara.copy()
    ep["el1"] = np.float32(el1)
    cx = synth.to_complex(job, pk, ep)
    mm = synth.config4_poses(3, 12, radius=5.0)
    _, _, out64 = dock.eval_poses(cx, np.zeros((12, 2), np.int32), mm, GD_PREC_FP64, want64=True)
    ref = np.array([oracle_lib.energy(cx, 0, 0, m)[0] for m in mm])
    err = np.abs(out64 - ref) / np.maximum(np.abs(ref), TOL.TAU)
    assert err[:, 1].max() <= 1e-9  # the FP64 kernel's tolerance
