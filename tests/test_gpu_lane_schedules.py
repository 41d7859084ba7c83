"""The default lane splits a sumcheck pass into a tile per SM, a pooled lane into 32: the
same proofs, equal to the oracle's. The statements are where the Spartan passes of either
lane change (tile sizes from 4 to 32 positions, sums posted by every block or added up by
the last one, all blocks of the largest grid in use): the block counts on the two sides of
such a change, for 440 + 696 k rows and 20,713 + 20,968 k columns at k blocks."""
import pytest

import bitz_b200 as bz
from bitz_b200 import statements as ci
from oracle import ffi as of

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fast_oracle():
    of.lib().o_set_clmul_mode(1)
    yield
    of.lib().o_set_clmul_mode(0)


@pytest.mark.parametrize("blocks", [6, 11, 12, 21, 24, 27, 54, 94, 108])
def test_default_and_pooled_lanes_match_oracle(blocks):
    kind = "sha256-block-aligned"
    inp, out, _ = ci.instance(kind, blocks, 60 + blocks)
    rc, want, _ = of.prove(ci.KINDS[kind], inp, out, 100)
    assert rc == 0
    ps = bz.CircuitProofSystem(kind, inp, out, 100)
    stats = ps.stats()
    assert stats["constraints"] == 440 + 696 * blocks
    assert stats["assignment_bits"] == 20713 + 20968 * blocks
    assert ps.prove()[0] == want
    assert bz.batch_prove([ps], 1)[0] == [want]
