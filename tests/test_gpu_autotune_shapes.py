"""gd_ensemble_autotune times the shape an ensemble has before its candidates, and
gives these the kernel with 128 registers where 16 or fewer warps share an SM: tuning
does not lose a shape that only the library's own choice has."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth

pytestmark = pytest.mark.gpu


def _tuned(enepara, atoms, points, nlig, nprt, ntmp, steps):
    rng = np.random.default_rng(2)
    pk = synth.make_pocket(rng, points, nprt)
    jobs = [synth.make_job(rng, pk, L, nlig, 60, 5, synth.ladder(ntmp, 0.3, 3.0), seed=i) for i, L in enumerate(atoms)]
    with dock.Ensemble.from_jobs([pk], jobs, enepara) as e:
        e.init()
        e.sync()
        lines = e.autotune(steps).strip().splitlines()
        again = e.autotune(steps).strip().splitlines()
    return lines, again


def _of(line):
    return {k: int(v) for k, v in (w.split("=") for w in line.replace(":", " ").split() if "=" in w)}


def _ms(line):
    return float(line.split()[-2])


def test_present_shape_is_a_candidate(lib, enepara):
    # 1200 replicas in teams of two
    lines, again = _tuned(enepara, (60, 60, 60), 700, 10, 5, 8, 6)
    chosen = _of(lines[-1])
    # whatever was chosen was the fastest timed, the first among them, and is the first of the next tuning
    least = min(map(_ms, lines[:-1]))
    assert any(all(_of(x)[k] == chosen[k] for k in chosen) for x in lines[:-1] if _ms(x) == least)
    assert all(_of(again[0])[k] == chosen[k] for k in chosen)


def test_wide_kernel_stays_where_it_is_faster(lib, enepara):
    # 80 atoms against 2200 points: 402 us a step with 80 registers, 353 with 128 (8 warps per SM)
    lines, _ = _tuned(enepara, (80, 80, 80), 2200, 10, 5, 8, 10)
    first = _of(lines[0])
    assert first["wide"] == 1 and first["kpl"] == 4 and first["ab"] == 8
    assert any(_of(x)["wide"] == 1 for x in lines[1:-1])
    assert _of(lines[-1])["wide"] == 1
