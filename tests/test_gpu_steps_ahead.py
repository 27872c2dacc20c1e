"""Chunks on thread-block clusters: where the GPU has SMs that no replica's team
needs, the steps that may follow are evaluated at the same time.  Decisions,
states, statistics and Records are those of one step after the other, bit for
bit; option "warps" set keeps a replica on one CTA."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64, check

pytestmark = pytest.mark.gpu


def _complex(enepara, nlig, ntmp, steps, temps, exchange=0, seed=5):
    rng = np.random.default_rng(seed)
    pk = synth.make_pocket(rng, 300, 1)
    job = synth.make_job(rng, pk, 19, nlig, 70, 5, temps if temps else synth.ladder(ntmp, 0.3, 3.0), seed=seed)
    return synth.to_complex(job, pk, enepara, steps, min(steps, 200), exchange)


def _both(lib, options, run):
    out = []
    try:
        for k, v in options.items():
            check(lib.gd_set_option(k, v))
        for warps in (0, 8):  # the library's choice; one CTA per replica or for several
            check(lib.gd_set_option(b"warps", warps))
            out.append(run())
    finally:
        check(lib.gd_set_option(b"warps", 0))
        check(lib.gd_set_option(b"replica_warps", 1))
        check(lib.gd_set_option(b"precision", GD_PREC_FP32_KAHAN))
    for a, b in zip(*out):
        assert a.tobytes() == b.tobytes()


# conformations and temperatures: clusters of 16, 13 (or what 11 of them fit), 4 and 2; steps: fewer than a round's
# nodes, past the 64 whose random numbers a CTA keeps, several chunks with exchange; all but no and nearly all moves
# accepted
@pytest.mark.parametrize("prec,V", [(GD_PREC_FP32, 1), (GD_PREC_FP32_KAHAN, 1), (GD_PREC_FP32_KAHAN, 8),
                                    (GD_PREC_FP64, 1)])
@pytest.mark.parametrize("nlig,ntmp,steps,exchange,temps", [(1, 1, 150, 0, [0.3]), (1, 1, 2, 0, [0.3]),
                                                            (1, 1, 90, 0, [1e-4]), (1, 1, 90, 0, [1e5]),
                                                            (11, 1, 40, 0, [0.5]), (9, 4, 30, 7, None),
                                                            (15, 4, 33, 10, None)])
def test_cluster_chunk_matches_one_step_at_a_time(lib, enepara, prec, V, nlig, ntmp, steps, exchange, temps):
    cx = _complex(enepara, nlig, ntmp, steps, temps)

    def run():
        with dock.Ensemble.from_complexes([cx], [4]) as e:
            e.init()
            e.run(steps, exchange)
            e.run(3, exchange)  # goes on from the statistics of the first
            e.sync()
            return e.replicas(0), e.stats(0)

    _both(lib, {b"precision": prec, b"replica_warps": V}, run)


@pytest.mark.parametrize("nlig,steps", [(1, 120), (20, 17)])
def test_cluster_records(lib, enepara, nlig, steps):
    cx = _complex(enepara, nlig, 1, steps, [0.4])

    def run():
        c = cx.copy()
        with dock.DockSession(1, seed=6) as s:
            rec = s.dock(c)
        n = rec["next_entry"]
        return (n, c[0]["replica"][:nlig], np.concatenate([r["replica"][:k] for r, k in zip(rec, n)]))

    _both(lib, {}, run)
