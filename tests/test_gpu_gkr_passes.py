"""The GKR's multi-round passes, its column counts for the two lowest layers and
the host's last rounds against the CPU oracle, at the sizes where their
schedule changes: no device rounds, one pass, several, chunks of 128 columns
partly filled, and sparse or full columns."""
import numpy as np
import pytest

import bitz_b200 as bz
from oracle import ffi as of

pytestmark = pytest.mark.gpu


def rand_f128(rng, n):
    return rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64)


@pytest.fixture(autouse=True)
def fast_oracle():
    of.lib().o_set_clmul_mode(1)
    yield
    of.lib().o_set_clmul_mode(0)


@pytest.mark.parametrize("s,fill", [
    (1, "random"), (2, "random"), (3, "sparse"), (5, "full"), (6, "random"), (7, "random"),
    (8, "sparse"), (9, "random"), (10, "zero"), (12, "random"), (13, "sparse"), (14, "random"),
])
def test_gkr_schedules_match_oracle(s, fill):
    rng = np.random.default_rng(4000 + s)
    images = rand_f128(rng, 128)
    cols = rand_f128(rng, 1 << s)
    if fill == "sparse":
        cols &= rand_f128(rng, 1 << s) & rand_f128(rng, 1 << s)
        cols[(1 << s) * 3 // 4:] = 0
    elif fill != "random":
        cols[:] = 0 if fill == "zero" else np.uint64(2**64 - 1)
    zeta = rand_f128(rng, s)
    ot = of.Transcript(b"gkr-passes", b"prove")
    opoint, oclaim = of.gkr_prove(images, cols, zeta, 0, ot)
    gt = bz.build_prover(b"gkr-passes", b"prove")
    gpoint, gclaim = bz.gkr_prove(images, cols, zeta, 100, gt)
    assert gt.narg() == ot.narg()
    assert np.array_equal(gpoint, opoint) and np.array_equal(gclaim, oclaim)


@pytest.mark.parametrize("s,at", [(11, 10), (11, 9), (11, 0), (12, 4)])
def test_zero_and_one_coordinates(s, at):
    """A zero coordinate in a round the device sums sends sum(1)."""
    rng = np.random.default_rng(77 + at)
    images = rand_f128(rng, 128)
    cols = rand_f128(rng, 1 << s)
    zeta = rand_f128(rng, s)
    zeta[at] = 0
    zeta[(at + 1) % s] = (1, 0)
    ot = of.Transcript(b"z", b"z")
    _, oclaim = of.gkr_prove(images, cols, zeta, 0, ot)
    gt = bz.build_prover(b"z", b"z")
    _, gclaim = bz.gkr_prove(images, cols, zeta, 100, gt)
    assert gt.narg() == ot.narg() and np.array_equal(gclaim, oclaim)


@pytest.mark.parametrize("s,fill,zero", [
    (15, "random", 14), (16, "full", 0), (16, "random", 15), (17, "sparse", 3), (20, "random", 19),
])
def test_large_schedules_match_oracle(s, fill, zero):
    """Column counts with 16 sums a thread (2^16 columns on), weights of three factors above
    the lowest 14 coordinates (2^20), a zero coordinate in a round that a pass sums, and a
    one above it."""
    rng = np.random.default_rng(5000 + s)
    images, cols, zeta = rand_f128(rng, 128), rand_f128(rng, 1 << s), rand_f128(rng, s)
    if fill == "sparse":
        cols &= rand_f128(rng, 1 << s) & rand_f128(rng, 1 << s)
        cols[(1 << s) * 3 // 4:] = 0
    elif fill == "full":
        cols[:] = np.uint64(2**64 - 1)
    zeta[zero] = 0
    zeta[(zero + 1) % s] = (1, 0)
    ot = of.Transcript(b"gkr-passes", b"large")
    opoint, oclaim = of.gkr_prove(images, cols, zeta, 0, ot)
    gt = bz.build_prover(b"gkr-passes", b"large")
    gpoint, gclaim = bz.gkr_prove(images, cols, zeta, 100, gt)
    assert gt.narg() == ot.narg()
    assert np.array_equal(gpoint, opoint) and np.array_equal(gclaim, oclaim)


def test_scalar_host_rounds_give_the_same_transcript():
    """BITZ_HOST_SIMD=0 runs the host's last rounds with one product at a time."""
    import hashlib
    import os
    import subprocess
    import sys
    code = """
import hashlib
import numpy as np
import bitz_b200 as bz
from oracle import ffi as of
rng = np.random.default_rng(12)
draw = lambda n: rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64)
h = hashlib.sha256()
for s in (1, 2, 9, 11):
    t = bz.build_prover(b"simd", b"gkr")
    bz.gkr_prove(draw(128), draw(1 << s), draw(s), 100, t)
    h.update(t.narg())
of.lib().o_set_clmul_mode(1)
for lr, lc in ((8, 0), (13, 0), (7, 1), (7, 9)):
    rows, cols, packed = draw(1 << lr), draw(1 << lc), draw(1 << (lr + lc - 7))
    t = bz.build_prover(b"simd", b"post")
    bz.post_gkr_prove(rows, cols, of.weighted_sum(rows, cols, packed), packed, 100, t)
    h.update(t.narg())
print(h.hexdigest())
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    got = [subprocess.run([sys.executable, "-c", code], cwd=root, check=True, capture_output=True,
                          text=True, env=dict(os.environ, BITZ_HOST_SIMD=flag)).stdout.strip()
           for flag in ("0", "1")]
    assert got[0] == got[1] and len(got[0]) == 2 * hashlib.sha256().digest_size
