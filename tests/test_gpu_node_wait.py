"""The wait of a cluster's CTAs for each other's energies is bounded by option
wait_limit (at least 10 ms): with bytes announced that nobody sends (stall_test 2: one
CTA gives up, the others miss it a round later) the host gets GD_E_TIMEOUT, and the next
ensemble runs as ever.  That the hook is reached shows that the chunk ran on clusters."""

import time

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_E_TIMEOUT, GD_PREC_FP32_KAHAN, GD_PREC_FP64, GdockError, check

pytestmark = pytest.mark.gpu


# one replica, 11 and 36 of them; a chunk of many rounds, and of one round (no CTA has another to miss)
@pytest.mark.parametrize("prec", [GD_PREC_FP32_KAHAN, GD_PREC_FP64])
@pytest.mark.parametrize("nlig,ntmp,steps", [(1, 1, 60), (11, 1, 40), (9, 4, 50), (1, 1, 2)])
def test_wait_for_nodes_is_bounded(lib, enepara, prec, nlig, ntmp, steps):
    rng = np.random.default_rng(5)
    pk = synth.make_pocket(rng, 300, 1)
    temps = synth.ladder(ntmp, 0.3, 3.0) if ntmp > 1 else [0.3]
    cx = synth.to_complex(synth.make_job(rng, pk, 19, nlig, 70, 5, temps, seed=5), pk, enepara)

    def run():
        with dock.Ensemble.from_complexes([cx], [4]) as e:
            e.init()
            e.sync()
            e.run(steps)
            t0 = time.perf_counter()
            try:
                e.sync()
            finally:
                took.append(time.perf_counter() - t0)
            r, s = e.replicas(0), e.stats(0)
            return [r[f].tobytes() for f in r.dtype.names] + [s.tobytes()]

    took = []
    check(lib.gd_set_option(b"precision", prec))
    try:
        want = run()
        check(lib.gd_set_option(b"wait_limit", 1000))
        assert run() == want
        check(lib.gd_set_option(b"stall_test", 2))
        for _ in range(2):
            with pytest.raises(GdockError) as ei:
                run()
            assert ei.value.code == GD_E_TIMEOUT
            assert took[-1] < 0.5  # not the second that the option's default allows
        check(lib.gd_set_option(b"stall_test", 0))
        assert run() == want
    finally:
        check(lib.gd_set_option(b"stall_test", 0))
        check(lib.gd_set_option(b"wait_limit", 0))
        check(lib.gd_set_option(b"precision", GD_PREC_FP32_KAHAN))
