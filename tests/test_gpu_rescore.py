"""gd_eval_poses packs its Complex on the GPU: the same bits as the poses of a
resident ensemble, whose Complex the host packs, and the host packer's errors."""

import threading

import numpy as np
import pytest

from geauxdock_b200 import dock, layout, synth
from geauxdock_b200._lib import GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64, check

pytestmark = pytest.mark.gpu


def _complex(enepara, L, P, K, M, nlig, nprt, dense=False, seed=2):
    rng = np.random.default_rng(seed)
    pk = synth.make_pocket(rng, P, nprt)
    job = synth.make_job(rng, pk, L, nlig, K, M, [0.3], seed=seed)
    if dense:  # a cell for every (class-2 point, type)
        job.psp = np.where(job.psp == 0, np.float32(-0.25), job.psp).astype(np.float32)
    return synth.to_complex(job, pk, enepara)


def _poses(n, nlig, nprt, seed=7):
    rng = np.random.default_rng(seed)
    conf = np.stack([rng.integers(0, nlig, n), rng.integers(0, nprt, n)], axis=1).astype(np.int32)
    return conf, synth.config4_poses(seed, n, radius=5.0)


# one atom and one point; the capacity of a Complex; an odd atom count; conformations of unequal point counts; one pose,
# a team of 2 to 16 warps per pose, one warp each
@pytest.mark.parametrize("L,P,K,M,nlig,nprt,dense", [(1, 1, 0, 1, 1, 1, False), (64, 2048, 900, 512, 3, 20, True),
                                                     (33, 129, 1, 17, 64, 2, False), (40, 700, 400, 16, 5, 7, False)])
@pytest.mark.parametrize("n", [1, 50, 700, 6000])
@pytest.mark.parametrize("prec", [GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64])
def test_equals_resident_ensemble(lib, enepara, L, P, K, M, nlig, nprt, dense, n, prec):
    cx = _complex(enepara, L, P, K, M, nlig, nprt, dense)
    if P == 700:
        cx[0]["prt"]["prt_npoint"][1:nprt] = [699, 1, 640, 641, 128, 300]
    conf, mm = _poses(n, nlig, nprt)
    got = dock.eval_poses(cx, conf, mm, prec, want64=True)
    with dock.Ensemble.from_complexes([cx], [1]) as e:
        want = e.eval_poses(0, conf, mm, prec, want64=True, want_raw=True)
    for a, b in zip(got, want):
        assert a.tobytes() == b.tobytes()


def _set(path, value):
    def change(cx):
        at = cx[0]
        for k in path[:-1]:
            at = at[k]
        at[path[-1]] = value
    return change


@pytest.mark.parametrize("change,message", [
    (_set(("lig", 0, "t2", 3), 24), "ligand atom"),
    (_set(("prt", 1, "t", 5), 30), "protein conformation 1 point 5"),
    (_set(("prt", 1, "prt_npoint"), 0), "prt_npoint = 0"),
    (_set(("lig", 1, "lig_natom"), 5), "conformation 1 has 5 atoms"),
    (_set(("enepara", "p1a", 2, 3), 0.0), "p1a"),
    (_set(("size", "n_tmp"), 0), "n_tmp = 0"),
    (_set(("size", "n_rep"), 0), "n_rep = 0"),
    (_set(("size", "mcs_nrow"), 0), "mcs_nrow = 0"),
    (_set(("replica", 0, "idx_tmp"), 9), "replica 0"),
    (_set(("mcs", 2, "x", slice(None)), layout.MCS_INVALID_COORD), "MCS row 2"),
])
def test_errors_are_the_host_packers(lib, enepara, change, message):
    cx = _complex(enepara, 20, 200, 30, 4, 2, 2)
    change(cx)
    conf, mm = _poses(3, 2, 2)
    with pytest.raises(Exception, match=message):
        dock.eval_poses(cx, conf, mm)


def test_threads_and_kept_blocks(lib, enepara):
    """Calls of several threads at once, of sizes that grow and shrink, with and without blocks kept."""
    shapes = [(12, 200, 40, 3, 2, 2), (40, 900, 400, 16, 5, 3), (64, 2048, 100, 40, 2, 6)]
    cases = []
    for s, (L, P, K, M, nlig, nprt) in enumerate(shapes):
        cx = _complex(enepara, L, P, K, M, nlig, nprt, seed=s)
        for n in (3, 400):
            conf, mm = _poses(n, nlig, nprt, seed=s + n)
            with dock.Ensemble.from_complexes([cx], [1]) as e:
                cases.append((cx, conf, mm, e.eval_poses(0, conf, mm, GD_PREC_FP32)[0].tobytes()))
    bad = []

    def work(k):
        for r in range(4):
            for j in range(len(cases)):
                cx, conf, mm, want = cases[(j * (k + 1) + r) % len(cases)]
                if dock.eval_poses(cx, conf, mm, GD_PREC_FP32)[0].tobytes() != want:
                    bad.append((k, r, j))

    try:
        for keep in (1, 0, 1):
            check(lib.gd_set_option(b"eval_cache", keep))
            ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
            assert not bad
    finally:
        check(lib.gd_set_option(b"eval_cache", 1))
