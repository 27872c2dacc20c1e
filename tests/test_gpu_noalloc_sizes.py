"""gd_eval_poses_noalloc at the sizes where its launch or its packing changes:
one pose and a few (teams of warps), more than one wave of CTAs, a potential that
is non-zero everywhere, no KDE point, an odd atom count and one row of points.
In FP64 its sums are combined as gd_eval_poses combines them, in FP32 as the
tile (2, 8) does with compensated sums (one warp per pose) or as a replica split
over two warps (teams): the same bits."""

import ctypes as C

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_E_INVALID, GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64, check

pytestmark = pytest.mark.gpu


def _call(lib, cx, conf, mm, prec):
    import torch

    n = len(conf)
    d_cx = torch.from_numpy(cx.view(np.uint8).reshape(-1).copy()).cuda()
    d_conf, d_mm = torch.from_numpy(conf).cuda(), torch.from_numpy(mm).cuda()
    out, raw = torch.zeros((n, 10), device="cuda"), torch.zeros((n, 9), device="cuda")
    rc = lib.gd_eval_poses_noalloc(C.c_void_p(d_cx.data_ptr()), n, C.c_void_p(d_conf.data_ptr()),
                                   C.c_void_p(d_mm.data_ptr()), prec, C.c_void_p(out.data_ptr()),
                                   C.c_void_p(raw.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return rc, out.cpu().numpy(), raw.cpu().numpy()


def _case(L, P, K, M, nlig, nprt, dense, n):
    rng = np.random.default_rng(L + n)
    pk = synth.make_pocket(rng, P, nprt)
    job = synth.make_job(rng, pk, L, nlig, K, M, [1.0], seed=1)
    if dense:
        job.psp = np.where(job.psp == 0, np.float32(-0.25), job.psp).astype(np.float32)
    conf = np.stack([rng.integers(0, nlig, n), rng.integers(0, nprt, n)], axis=1).astype(np.int32)
    return pk, job, conf, synth.config4_poses(n, n, radius=5.0)


SIZES = [(24, 600, 200, 8, 1, 1, False, 1), (33, 129, 0, 17, 3, 2, False, 150), (64, 2048, 1000, 40, 2, 3, True, 600),
         (17, 300, 60, 1, 4, 4, True, 5000)]


@pytest.mark.parametrize("L,P,K,M,nlig,nprt,dense,n", SIZES)
def test_noalloc_fp64_equals_eval_poses(lib, enepara, L, P, K, M, nlig, nprt, dense, n):
    pk, job, conf, mm = _case(L, P, K, M, nlig, nprt, dense, n)
    cx = synth.to_complex(job, pk, enepara)
    want, want_raw, _ = dock.eval_poses(cx, conf, mm, GD_PREC_FP64)
    rc, out, raw = _call(lib, cx, conf, mm, GD_PREC_FP64)
    assert rc == 0
    assert out.tobytes() == want.tobytes() and raw.tobytes() == want_raw.tobytes()


@pytest.mark.parametrize("prec", [GD_PREC_FP32, GD_PREC_FP32_KAHAN])
@pytest.mark.parametrize("L,P,K,M,nlig,nprt,dense,n", SIZES)
def test_noalloc_fp32_sums(lib, enepara, L, P, K, M, nlig, nprt, dense, n, prec):
    pk, job, conf, mm = _case(L, P, K, M, nlig, nprt, dense, n)
    try:
        if n > 1776:
            cx = synth.to_complex(job, pk, enepara)
            check(lib.gd_set_option(b"kpl", 2))
            want = dock.eval_poses(cx, conf, mm, GD_PREC_FP32_KAHAN)[0]
        else:
            # the poses as the initial states of replicas split over two warps
            ntmp = n // (nlig * nprt)
            job.temps = np.linspace(0.3, 3.0, ntmp).astype(np.float32)
            cx = synth.to_complex(job, pk, enepara)
            reps = cx[0]["replica"][:n]
            reps["movematrix"] = mm
            conf = np.stack([reps["idx_lig"], reps["idx_prt"]], axis=1).astype(np.int32)
            check(lib.gd_set_option(b"replica_warps", 2))
            with dock.Ensemble.from_complexes([cx], [1]) as e:
                e.init()
                e.sync()
                want = np.ascontiguousarray(e.replicas(0)["energy"])
    finally:
        check(lib.gd_set_option(b"kpl", 0))
        check(lib.gd_set_option(b"replica_warps", 1))
    rc, out, _ = _call(lib, cx, conf, mm, prec)
    assert rc == 0
    assert out.tobytes() == want.tobytes()


@pytest.mark.parametrize("n", [40, 4000])
def test_noalloc_refuses_bad_conformation(lib, enepara, n):
    """A pose whose conformation is out of range fails the call; the others are evaluated."""
    pk, job, conf, mm = _case(20, 200, 50, 4, 2, 2, False, n)
    cx = synth.to_complex(job, pk, enepara)
    good = _call(lib, cx, conf, mm, GD_PREC_FP32)[1]
    conf[7] = (0, 2)
    rc, out, _ = _call(lib, cx, conf, mm, GD_PREC_FP32)
    assert rc == GD_E_INVALID and np.isnan(out[7]).all()
    keep = np.arange(n) != 7
    assert out[keep].tobytes() == good[keep].tobytes()
