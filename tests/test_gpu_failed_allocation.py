"""Device allocations that do not fit: the call that needs one fails with a CUDA error, and
only that call."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import bitz_b200 as bz
from bitz_b200 import _lib
from oracle import ffi as of

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# a claim of 2^40 bits wants terabytes of scratch before it reads any input
_NEXT_CALL = """
import ctypes
import numpy as np
import torch
import bitz_b200 as bz
from bitz_b200 import _lib
from oracle import ffi as of
lib, u64p = _lib.load(), ctypes.POINTER(ctypes.c_uint64)
word = torch.zeros((1, 2), dtype=torch.int64, device="cuda")
buf = np.zeros((64, 2), dtype=np.uint64)
out = buf.ctypes.data_as(u64p)
ts = bz.build_prover(b"s", b"i")
rc = lib.bitz_post_gkr_prove_dev(word.data_ptr(), 32, word.data_ptr(), 8, out, word.data_ptr(), 100, ts.handle, out, out)
assert rc != 0 and b"out of memory" in lib.bitz_last_error(), lib.bitz_last_error()
rng = np.random.default_rng(5)
images, cols = (rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64) for n in (128, 64))
assert np.array_equal(bz.gkr_outputs(images, cols), of.gkr_outputs(images, cols))
"""


def test_a_failed_allocation_does_not_fail_the_next_call():
    r = subprocess.run([sys.executable, "-c", _NEXT_CALL], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_calls_after_a_failed_growth_use_no_freed_tables():
    """A growth frees a lane's tables before it takes larger ones. When those do not fit, the
    next smaller call must allocate again, not run on what was freed."""
    import torch
    rng = np.random.default_rng(6)
    draw = lambda n: rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64)  # noqa: E731
    lib, u64p = _lib.load(), ctypes.POINTER(ctypes.c_uint64)
    word = torch.zeros((1, 2), dtype=torch.int64, device="cuda")
    out = np.zeros((64, 2), dtype=np.uint64).ctypes.data_as(u64p)
    images, cols, rows, few, packed = draw(128), draw(64), draw(1 << 9), draw(2), draw(1 << 3)
    target = of.weighted_sum(rows, few, packed)

    def small_calls():
        ts = bz.build_prover(b"s", b"i")
        point, value = bz.post_gkr_prove(rows, few, target, packed, 100, ts)
        return bz.gkr_outputs(images, cols).tobytes(), point.tobytes(), value.tobytes(), ts.narg()

    want = small_calls()
    ts = bz.build_prover(b"s", b"i")
    # 279 GB of layers, and 8.8 TB a table: refused before any input is read
    assert lib.bitz_gkr_prove_dev(word.data_ptr(), word.data_ptr(), 28, out, 100, ts.handle, out, out) != 0
    assert b"out of memory" in lib.bitz_last_error()
    assert lib.bitz_post_gkr_prove_dev(word.data_ptr(), 32, word.data_ptr(), 8, out, word.data_ptr(),
                                       100, ts.handle, out, out) != 0
    assert b"out of memory" in lib.bitz_last_error()
    assert small_calls() == want
