"""Pose energies in more than one CUDA context of a process (run by
test_gpu_contexts.py): `second` alternates between the primary context and another
one, `reset` resets the primary context between calls.  Prints one JSON line: whether
each call gave the first call's bytes, and the device memory lost meanwhile."""

import ctypes as C
import json
import sys
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

from geauxdock_b200 import dock, params, synth  # noqa: E402
from geauxdock_b200._lib import GD_PREC_FP32, load  # noqa: E402


def main(what: str) -> None:
    load()
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc

    def free():
        a, b = C.c_size_t(), C.c_size_t()
        ok(cu.cuMemGetInfo_v2(C.byref(a), C.byref(b)))
        return a.value

    rng = np.random.default_rng(1)
    pk = synth.make_pocket(rng, 900, 2)
    cx = synth.to_complex(synth.make_job(rng, pk, 40, 2, 50, 6, [1.0], seed=1), pk,
                          params.optimize_enepara(params.default_enepara0()))

    def run():
        out = b""
        for n in (40, 6000):  # 16 warps a pose, and one
            conf = np.stack([np.arange(n) % 2, np.arange(n) // 2 % 2], axis=1).astype(np.int32)
            out += dock.eval_poses(cx, conf, synth.config4_poses(n, n, radius=5.0), GD_PREC_FP32)[0].tobytes()
        return out

    want, same = run(), []
    ok(cu.cuInit(0))
    if what == "second":
        ctx, primary = C.c_void_p(), C.c_void_p()
        ok(cu.cuCtxGetCurrent(C.byref(primary)))
        ok(cu.cuCtxCreate_v2(C.byref(ctx), 0, 0))
        before = None
        for k in range(6):
            ok(cu.cuCtxSetCurrent(ctx if k % 2 == 0 else primary))
            same.append(run() == want)
            if k == 1:
                before = free()
        lost = before - free()
    else:
        lost = 0
        for _ in range(3):
            ok(cu.cuDevicePrimaryCtxReset_v2(0))
            same.append(run() == want)
    print(json.dumps({"same": same, "free_lost": lost}))


if __name__ == "__main__":
    main(sys.argv[1])
