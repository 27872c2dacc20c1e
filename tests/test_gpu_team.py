"""Teams of warps: where one wave of the GPU holds the replicas (or poses) of a
launch, each gets 2 to 16 warps.  The sums are combined in the one-warp kernel's
order, so the results are the same bits on any number of warps; option "warps"
set fixes one warp per replica."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64, check

pytestmark = pytest.mark.gpu

# atoms, points, KDE points, templates, ligand / protein conformations, temperatures: one replica (16 warps); an odd
# atom count, one row, no KDE point and more replicas than SMs (8 warps or 4); two runs of templates and more walk
# chunks than a team keeps (24 of 32 slots and cells); 1056 replicas (2 warps)
SHAPES = [(24, 600, 200, 8, 1, 1, 1), (1, 1, 0, 1, 2, 1, 3), (33, 129, 0, 16, 10, 4, 4), (61, 700, 1500, 40, 3, 2, 2),
          (15, 260, 90, 17, 11, 6, 16)]


def _case(shape, seed=3):
    L, P, K, M, nlig, nprt, ntmp = shape
    rng = np.random.default_rng(seed)
    pk = synth.make_pocket(rng, P, nprt)
    job = synth.make_job(rng, pk, L, nlig, K, M, synth.ladder(ntmp, 0.3, 3.0) if ntmp > 1 else [0.3], seed=seed)
    if K > 1000:  # a cell for every (class-2 point, type)
        job.psp = np.where(job.psp == 0, np.float32(-0.25), job.psp).astype(np.float32)
    return pk, job


@pytest.mark.parametrize("prec", [GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64])
@pytest.mark.parametrize("shape", SHAPES)
def test_team_matches_one_warp(lib, enepara, shape, prec):
    pk, job = _case(shape)
    cx = synth.to_complex(job, pk, enepara)
    out = []
    try:
        check(lib.gd_set_option(b"precision", prec))
        for warps in (0, 4):  # the library's choice; 4 replicas of one warp per CTA
            check(lib.gd_set_option(b"warps", warps))
            with dock.Ensemble.from_complexes([cx], [9]) as e:
                e.init()
                e.run(20, 6 if shape[6] > 1 else 0)  # 20 steps: past the 16 whose draws a team makes at once
                e.sync()
                out.append((e.replicas(0), e.stats(0)))
    finally:
        check(lib.gd_set_option(b"warps", 0))
        check(lib.gd_set_option(b"precision", GD_PREC_FP32_KAHAN))
    for f in out[0][0].dtype.names:
        assert out[0][0][f].tobytes() == out[1][0][f].tobytes(), f
    assert out[0][1].tobytes() == out[1][1].tobytes()


@pytest.mark.parametrize("prec", [GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64])
@pytest.mark.parametrize("shape", SHAPES[:4])
def test_team_poses_match_one_warp(lib, enepara, shape, prec):
    """A few poses (teams) and the same among thousands (one warp each)."""
    pk, job = _case(shape)
    n = 9
    rng = np.random.default_rng(2)
    conf = np.stack([rng.integers(0, shape[4], n), rng.integers(0, shape[5], n)], axis=1).astype(np.int32)
    mm = synth.config4_poses(4, n, radius=5.0)
    with dock.Ensemble.from_jobs([pk], [job], enepara) as e:
        few = e.eval_poses(0, conf, mm, prec, want64=True, want_raw=True)
        many = e.eval_poses(0, np.tile(conf, (450, 1)), np.tile(mm, (450, 1)), prec, want64=True, want_raw=True)
    for a, b in zip(few, many):
        assert a.tobytes() == b[-n:].tobytes()
