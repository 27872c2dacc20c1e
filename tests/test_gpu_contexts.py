"""Two CUDA contexts on one GPU in one process, and a primary context that is reset
between calls: nothing of one (a kernel's shared-memory limit, a kept block or
stream) is taken for the other's.  In a child process (tests/contexts_worker.py)."""

import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("what", ["second", "reset"])
def test_contexts(lib, what):
    r = subprocess.run([sys.executable, str(ROOT / "tests" / "contexts_worker.py"), what], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    d = json.loads([ln for ln in r.stdout.splitlines() if ln.startswith("{")][-1])
    assert d["same"] == [True] * len(d["same"]) and d["free_lost"] < 8 << 20
