"""gd_eval_poses_noalloc with so many poses that 6 x their number is past 32 bits:
every pose is read from, and its result written to, its own place."""

import ctypes as C

import numpy as np
import pytest

from geauxdock_b200 import synth
from geauxdock_b200._lib import GD_PREC_FP32, check

pytestmark = pytest.mark.gpu


def test_noalloc_more_poses_than_32_bit_offsets(lib, enepara):
    import torch

    n, m = (2**31 // 6 + 1) // 1000 * 1000 + 2000, 1000  # the last 1058 start past 2^31 values
    if torch.cuda.mem_get_info()[0] < 40 * 10**9:
        pytest.skip("needs 26 GB of device memory")
    rng = np.random.default_rng(5)
    pk = synth.make_pocket(rng, 20, 1)
    job = synth.make_job(rng, pk, 1, 1, 0, 1, [1.0], seed=1)
    cx = synth.to_complex(job, pk, enepara)
    d_cx = torch.from_numpy(cx.view(np.uint8).reshape(-1).copy()).cuda()
    few = torch.from_numpy(synth.config4_poses(3, m, radius=5.0)).cuda()
    mm = torch.empty((n // m, m, 6), device="cuda")
    mm[:] = few
    conf = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    out = torch.zeros((n // m, m, 10), device="cuda")
    check(lib.gd_eval_poses_noalloc(C.c_void_p(d_cx.data_ptr()), n, C.c_void_p(conf.data_ptr()),
                                    C.c_void_p(mm.data_ptr()), GD_PREC_FP32, C.c_void_p(out.data_ptr()), None,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.isfinite(out[0]).all() and len(torch.unique(out[0, :, 9])) > m // 2
    for i in range(0, n // m, 4096):
        assert (out[i:i + 4096] == out[0]).all()
    del mm, conf, out
    torch.cuda.empty_cache()
