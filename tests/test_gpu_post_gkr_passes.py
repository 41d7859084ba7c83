"""The post-GKR sumcheck's paths against the CPU oracle: one column (rounds from
the bits), few columns, columns in chunks of 128 with one or more words each,
and table sizes around each change of schedule."""
import numpy as np
import pytest

import bitz_b200 as bz
from oracle import ffi as of

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fast_oracle():
    of.lib().o_set_clmul_mode(1)
    yield
    of.lib().o_set_clmul_mode(0)


@pytest.mark.parametrize("log_rows,log_cols,fill", [
    (8, 0, "random"), (9, 0, "sparse"), (11, 0, "random"), (12, 0, "random"), (13, 0, "sparse"),
    (17, 0, "random"), (20, 0, "sparse"), (7, 2, "random"), (9, 6, "random"), (14, 1, "random"),
    (17, 2, "sparse"), (7, 7, "random"), (7, 11, "random"), (8, 9, "random"), (12, 7, "sparse"),
    (13, 7, "random"), (10, 10, "random"),
])
def test_post_gkr_paths_match_oracle(log_rows, log_cols, fill):
    rng = np.random.default_rng(900 + 40 * log_rows + log_cols)
    draw = lambda n: rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64)  # noqa: E731
    rows, cols = draw(1 << log_rows), draw(1 << log_cols)
    packed = draw((1 << (log_rows - 7)) << log_cols)
    if fill == "sparse":
        packed &= draw(len(packed)) & draw(len(packed))
        packed[len(packed) * 5 // 8:] = 0
    target = of.weighted_sum(rows, cols, packed)
    ot = of.Transcript(b"post-gkr-passes", b"reduce")
    rc, opoint, ovalue = of.post_gkr_prove(rows, cols, target, packed, 0, ot)
    assert rc == 0
    gt = bz.build_prover(b"post-gkr-passes", b"reduce")
    gpoint, gvalue = bz.post_gkr_prove(rows, cols, target, packed, 100, gt)
    assert gt.narg() == ot.narg()
    assert np.array_equal(gpoint, opoint) and np.array_equal(gvalue, ovalue)


@pytest.mark.parametrize("log_rows,log_cols", [(8, 0), (13, 0), (7, 1), (7, 8), (12, 3)])
def test_false_claims_are_rejected_on_every_path(log_rows, log_cols):
    rng = np.random.default_rng(31 + log_rows)
    draw = lambda n: rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64)  # noqa: E731
    rows, cols = draw(1 << log_rows), draw(1 << log_cols)
    packed = draw((1 << (log_rows - 7)) << log_cols)
    target = of.weighted_sum(rows, cols, packed)
    target[1] ^= np.uint64(4)
    t = bz.build_prover(b"s", b"i")
    with pytest.raises(bz.BitzError) as e:
        bz.post_gkr_prove(rows, cols, target, packed, 100, t)
    assert e.value.code == "ClaimDoesNotHold" and t.narg() == b""
