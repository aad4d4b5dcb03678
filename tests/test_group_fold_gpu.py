"""Where a chain's groups of chunks get their starting states: folded by the group's own CTA for up to 16
groups, by a kernel of its own beyond -- both sides of the line, against the oracle."""
import pytest

import wkv_testlib as TL
import test_chunked_gpu as CG
import test_time_groups_gpu as TG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,T", [(16, 16 * 64), (17, 17 * 64), (2, 65), (18, 18 * 64 - 1), (33, 33 * 64)])
def test_group_starts_on_both_sides_of_the_line(groups, T):
    W, wkv56 = CG._pkg()
    q = TL.case56("v6", 1, T, 2, TG.BF, seed=groups)
    got = TG.run("v6", q, W.WKV_STATE_VK, groups, True, W, wkv56)
    want = CG.floored_oracle("v6", q)
    for n in TG.NAMES:
        TL.assert_close(f"v6.{n} G={groups}", got[n], want[n], 2e-2)
