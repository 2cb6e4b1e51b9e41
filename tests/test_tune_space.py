"""The tuner's default candidates are different launches (CPU): the learned
criterion's walk holds 16 warps per SM, so two and more units of 8 are one."""
import dataclasses

import pytest

from tree_b200.tune import default_space


@pytest.mark.parametrize("learned", [False, True])
def test_no_candidate_is_measured_twice(learned):
    space = default_space(learned)
    launches = {dataclasses.replace(c, blocks_per_sm=min(c.blocks_per_sm, 2)) if c.eta > 0 else c
                for c in space}
    assert len(launches) == len(space)
    assert {c.eta for c in space} == ({0.0, 1e-5, 3e-5, 1e-4} if learned else {0.0})
    assert {c.blocks_per_sm for c in space if c.eta == 0.0} == {2, 3}
