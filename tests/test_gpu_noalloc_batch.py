"""A pose's energy from gd_eval_poses_noalloc beside different numbers of other poses:
the same bits in FP64; in FP32 the same bits among calls of few poses and among calls
of many, and between the two within twice the parity tolerance."""

import ctypes as C

import numpy as np
import pytest

from geauxdock_b200 import synth
from geauxdock_b200._lib import GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64, check
from oracle import tolerance as TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [GD_PREC_FP32, GD_PREC_FP32_KAHAN, GD_PREC_FP64])
@pytest.mark.parametrize("L,P", [(24, 600), (33, 129)])
def test_pose_beside_others(lib, enepara, L, P, prec):
    import torch

    rng = np.random.default_rng(L)
    pk = synth.make_pocket(rng, P, 2)
    cx = synth.to_complex(synth.make_job(rng, pk, L, 2, 80, 9, [1.0], seed=1), pk, enepara)
    d_cx = torch.from_numpy(cx.view(np.uint8).reshape(-1).copy()).cuda()
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    # few: a team of warps per pose in one wave; many: more than 24 warps per SM
    few, many = [1, 7, nsm, 8 * nsm], [25 * nsm, 40 * nsm + 3]
    n = max(many)
    conf = torch.from_numpy(np.stack([np.arange(n) % 2, np.arange(n) // 2 % 2], axis=1).astype(np.int32)).cuda()
    mm = torch.from_numpy(synth.config4_poses(3, n, radius=5.0)).cuda()

    def call(k):
        out = torch.zeros((k, 10), device="cuda")
        check(lib.gd_eval_poses_noalloc(C.c_void_p(d_cx.data_ptr()), k, C.c_void_p(conf.data_ptr()),
                                        C.c_void_p(mm.data_ptr()), prec, C.c_void_p(out.data_ptr()), None,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return out.cpu().numpy()

    a, b = call(few[-1]), call(many[-1])
    for k in few:
        assert call(k).tobytes() == a[:k].tobytes(), k
    for k in many:
        assert call(k).tobytes() == b[:k].tobytes(), k
    if prec == GD_PREC_FP64:
        assert a.tobytes() == b[:len(a)].tobytes()
    else:
        assert TOL.scaled_error(a, b[:len(a)]).max() <= 2.0
