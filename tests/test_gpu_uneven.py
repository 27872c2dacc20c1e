"""Launch shapes of several jobs: teams in several waves where the ligands are
uneven, one warp per replica with more registers where 16 or fewer share an SM.
The results are the same bits as with 8 replicas of one warp per CTA (option
"warps")."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64, check

pytestmark = pytest.mark.gpu


# 1600 replicas of uneven ligands (teams of 4), of even ones (one wave of 11 warps per SM), 2000 (more than 16 per
# SM on some), and few replicas of very uneven ligands
@pytest.mark.parametrize("prec", [GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64])
@pytest.mark.parametrize("atoms,nlig,nprt,ntmp", [((8, 14, 25, 70), 10, 5, 8), ((31, 31, 30, 31), 10, 5, 8),
                                                  ((80, 9, 9, 9, 9), 10, 5, 8), ((77, 5), 7, 3, 3)])
def test_shapes_of_several_jobs(lib, enepara, prec, atoms, nlig, nprt, ntmp):
    rng = np.random.default_rng(8)
    pk = synth.make_pocket(rng, 270, nprt)
    temps = synth.ladder(ntmp, 0.3, 3.0)
    jobs = [synth.make_job(rng, pk, L, nlig, 60, 5, temps, seed=L + 100 * i) for i, L in enumerate(atoms)]
    out = []
    try:
        check(lib.gd_set_option(b"precision", prec))
        for warps in (0, 8):
            check(lib.gd_set_option(b"warps", warps))
            with dock.Ensemble.from_jobs([pk], jobs, enepara) as e:
                e.init()
                e.run(7, 3)
                e.sync()
                out.append([(e.replicas(j), e.stats(j)) for j in range(len(jobs))])
    finally:
        check(lib.gd_set_option(b"warps", 0))
        check(lib.gd_set_option(b"precision", GD_PREC_FP32_KAHAN))
    for (ra, sa), (rb, sb) in zip(*out):
        for f in ra.dtype.names:
            assert ra[f].tobytes() == rb[f].tobytes(), f
        assert sa.tobytes() == sb.tobytes()
