"""What one call leaves for the next: bounding boxes, queue heads and the W
block counter are reset on the device, whatever calls alternate; W of few and
of many sets (where a kernel of its own adds the tiles)."""
import numpy as np
import pytest

from starsmasher_b200 import Context, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsets", [1, 3, 255, 256, 400])
@pytest.mark.parametrize("precision", ["fp64", "f32split", "tree"])
def test_w_of_many_sets(nsets, precision):
    base = inputs.single_polytrope(90, 1.5, seed=2)
    rng = np.random.default_rng(nsets)
    sizes = rng.integers(1, 90, nsets)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    x, y, z, m, r2 = (np.concatenate([getattr(base, f)[:k] for k in sizes])
                      for f in ("x", "y", "z", "m", "range2"))
    with Context(0) as ctx:
        for _ in range(2):
            out = ctx.batch_forces(offs, x, y, z, m, r2, 0, precision)
            w = [0.5 * np.sum(m[a:b] * out[3][a:b]) for a, b in zip(offs[:-1], offs[1:])]
            assert np.allclose(out[4], w, rtol=1e-13, atol=0)


def test_alternating_calls_repeat_bit_for_bit():
    small = inputs.single_polytrope(700, 1.5, seed=4)
    large = inputs.config2(seed=6, n_each=2500)
    calls = [(s, p) for s in (small, large) for p in ("f32split", "fp64", "tree")]

    def arrays(s):
        return s.x, s.y, s.z, s.m, s.range2

    want = []
    for s, p in calls:
        with Context(0) as ctx:
            want.append(ctx.forces(*arrays(s), 0, p))
    with Context(0) as ctx:
        for k in (0, 3, 1, 4, 2, 5, 0, 5, 3):
            got = ctx.forces(*arrays(calls[k][0]), 0, calls[k][1])
            assert all(np.array_equal(a, b) for a, b in zip(got, want[k])), k


@pytest.mark.parametrize("precision", ["fp64", "f32split", "tree"])
def test_w_of_empty_sets(precision):
    s = inputs.single_polytrope(300, 1.5, seed=3)
    none = [np.zeros(0)] * 5
    with Context(0) as ctx:
        full = ctx.batch_forces([0, 100, 200, 300], s.x, s.y, s.z, s.m, s.range2, 0, precision)
        assert (full[4] < 0.0).all()
        empty = ctx.batch_forces([0, 0, 0, 0], *none, 0, precision)
        assert not empty[4].any()


@pytest.mark.parametrize("precision", ["fp64", "f32split", "tree"])
def test_more_sets_than_a_grid_dimension(precision):
    """Batches may hold 2^20 sets; a grid's second dimension ends at 65,535."""
    pairs = 66001
    rng = np.random.default_rng(1)
    d, m = rng.uniform(0.5, 2.0, pairs), rng.uniform(0.1, 1.0, 2 * pairs)
    x = np.zeros(2 * pairs)
    x[1::2] = d  # two point masses in each set, farther apart than their H
    zero, r2 = np.zeros(2 * pairs), np.full(2 * pairs, -0.01)
    offs = np.concatenate([[0, 0], 2 * np.arange(1, pairs + 1)])  # the first set is empty
    with Context(0) as ctx:
        ax, ay, az, pot, w = ctx.batch_forces(offs, x, zero, zero, m, r2, 0, precision)
    want = np.empty_like(x)
    want[0::2], want[1::2] = m[1::2] / d ** 2, -m[0::2] / d ** 2
    assert np.allclose(ax, want, rtol=1e-6) and not ay.any() and not az.any()
    assert np.allclose(pot, -np.abs(want) * np.repeat(d, 2), rtol=1e-6)
    assert w[0] == 0.0 and np.allclose(w[1:], -m[0::2] * m[1::2] / d, rtol=1e-6)
