"""Groups handed to the tree's direct sum: chunks of 256 sources and more, one
group and several, whose rows are exact (FP64 sums of the same terms: 1e-11)."""
import numpy as np
import pytest

from starsmasher_b200 import Context, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12289, 20011, 70001, 300000])
@pytest.mark.parametrize("nkernel", [0, 2])
def test_core_row_is_exact(n, nkernel):
    s = inputs.red_giant(n, seed=n)
    a = (s.x, s.y, s.z, s.m, s.range2)
    with Context(0) as ctx:
        ctx.set_theta(0.5)
        got = ctx.forces(*a, nkernel, "tree")
        groups, heavy = ctx.tree_stats()
        ref = ctx.forces(*a, nkernel, "fp64")
    amag = np.sqrt(ref[0] ** 2 + ref[1] ** 2 + ref[2] ** 2)
    d = np.sqrt(sum((g - r) ** 2 for g, r in zip(got[:3], ref[:3])))
    assert heavy >= 1
    assert d[0] <= 1e-11 * np.median(amag)
    assert abs(got[3][0] - ref[3][0]) <= 1e-11 * abs(ref[3][0])
    assert np.sqrt(np.mean((d / amag)[amag > 1e-3 * np.median(amag)] ** 2)) <= 2e-3
