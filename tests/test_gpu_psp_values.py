"""The pocket-specific term adds the value of a cell where an atom is within its
distance, and there alone: with infinite values and NaN in the potential, poses out
of reach of every cell have the energy they have with any other values."""

import ctypes as C

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64, check

pytestmark = pytest.mark.gpu


def _noalloc(lib, cx, conf, mm, prec):
    import torch

    d = [torch.from_numpy(x).cuda() for x in (cx.view(np.uint8).reshape(-1).copy(), conf, mm)]
    out = torch.zeros((len(conf), 10), device="cuda")
    check(lib.gd_eval_poses_noalloc(C.c_void_p(d[0].data_ptr()), len(conf), C.c_void_p(d[1].data_ptr()),
                                    C.c_void_p(d[2].data_ptr()), prec, C.c_void_p(out.data_ptr()), None,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return out.cpu().numpy()


def _resident(lib, cx, conf, mm, prec):
    with dock.Ensemble.from_complexes([cx], [1]) as e:
        return e.eval_poses(0, conf, mm, prec)[0]


# (the resident FP32 loop multiplies the value by the hits, as it always has)
@pytest.mark.parametrize("call,prec", [(_noalloc, GD_PREC_FP32), (_noalloc, GD_PREC_FP32_KAHAN), (_noalloc, GD_PREC_FP64),
                                       (_resident, GD_PREC_FP64)])
@pytest.mark.parametrize("n", [5, 700, 5000])
def test_cells_out_of_reach_add_nothing(lib, enepara, call, prec, n):
    rng = np.random.default_rng(3)
    pk = synth.make_pocket(rng, 300, 1)
    job = synth.make_job(rng, pk, 14, 1, 40, 3, [0.3], seed=3)
    conf, mm = np.zeros((n, 2), np.int32), synth.config4_poses(n, n, radius=5.0)
    mm[:, 0] += np.float32(200.0)
    out = []
    for value in (-1.0, np.inf, np.nan):
        job.psp = np.where(job.psp == 0, np.float32(0), np.float32(value)).astype(np.float32)
        out.append(call(lib, synth.to_complex(job, pk, enepara), conf, mm, prec))
    assert np.isfinite(out[0]).all()
    assert out[0].tobytes() == out[1].tobytes() == out[2].tobytes()
