"""Split-FP32 shapes whose rows share threads, many items per CTA one after another:
the first thread of a row reads the sums of the others at the end of an item, and
they zero those sums for the next.  Every call must give the same bits, and W the
potentials' sum."""
import numpy as np
import pytest

from starsmasher_b200 import Context, inputs
from starsmasher_b200.api import variant_names

from conftest import err_report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["f32split_w12_k1_q2_tj256_ns7", "f32split_w15_k1_q2_tj256",
                                  "f32split_w8_k1_q4_tj256", "f32split_w12_k1_q4_tj256_ns7"])
def test_short_items(name):
    sizes = np.random.default_rng(3).integers(200, 700, 600)  # items of one to three j-tiles
    base = inputs.single_polytrope(700, 1.5, seed=11)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    x, y, z, m, r2 = (np.concatenate([getattr(base, f)[:k] for k in sizes])
                      for f in ("x", "y", "z", "m", "range2"))
    with Context(0) as ctx:
        ctx.force_variant("f32split", variant_names("f32split").index(name))
        got = ctx.batch_forces(offs, x, y, z, m, r2, 0, "f32split")
        for _ in range(4):
            again = ctx.batch_forces(offs, x, y, z, m, r2, 0, "f32split")
            assert all(np.array_equal(a, b) for a, b in zip(got, again))
        ref = ctx.batch_forces(offs, x, y, z, m, r2, 0, "fp64")
    e = err_report(*got[:4], *ref[:4])
    assert e["acc_max"] <= 1e-6 and e["pot_max"] <= 1e-6, e
