"""The padding bytes of a Complex's replicas have no part in what a Dock call
returns: states and Records are the same bytes whatever they hold."""

import numpy as np
import pytest

from geauxdock_b200 import dock, synth
from geauxdock_b200._lib import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_pack", [0, 1])
def test_dock_ignores_replica_padding(lib, enepara, device_pack):
    rng = np.random.default_rng(4)
    pk = synth.make_pocket(rng, 150, 1)
    cx = synth.to_complex(synth.make_job(rng, pk, 11, 3, 20, 2, [0.4], seed=4), pk, enepara, 12, 12)
    size = cx.dtype["replica"].base.itemsize
    used = max(off + t.itemsize for t, off, *_ in cx.dtype["replica"].base.fields.values())
    assert used < size
    raw = cx.view(np.uint8).reshape(-1)
    at = cx.dtype.fields["replica"][1]
    out = []
    check(lib.gd_set_option(b"dock_device_pack", device_pack))
    try:
        for fill in (0, 0xAB):
            with dock.DockSession(1, seed=6) as s:
                for _ in range(2):  # the second call refills the first's state
                    c = np.frombuffer(bytearray(raw.tobytes()), dtype=cx.dtype)
                    for r in range(3):
                        c.view(np.uint8)[at + r * size + used:at + (r + 1) * size] = fill
                    rec = s.dock(c)
                    out.append((c[0]["replica"][:3].tobytes(),
                                [r["replica"][:int(r["next_entry"])].tobytes() for r in rec[:3]]))
    finally:
        check(lib.gd_set_option(b"dock_device_pack", 1))
    assert out[0] == out[2] and out[1] == out[3]
