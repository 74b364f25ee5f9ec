"""The curve sort in tiles at the edges of its tiles and of its range (65,536
particles), with coincident particles (equal keys), one set and a batch whose
sets end inside tiles.  The tree needs the keys sorted and the particles
complete, so its error against the FP64 direct sum shows both; its bits depend
on the order of equal keys, so they show whether that is the device-wide sort's."""
import numpy as np
import pytest

from starsmasher_b200 import Context, inputs

from conftest import err_report

pytestmark = pytest.mark.gpu


def _model(n, seed):
    s = inputs.single_polytrope(n, 1.5, seed=seed)
    a = [getattr(s, f).copy() for f in ("x", "y", "z", "m", "range2")]
    for v in a[:3]:
        v[n // 2:n // 2 + 7] = v[n // 2]
    return a


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4097, 16385, 65535, 65536, 65537])
def test_tile_edges(n):
    a = _model(n, n)
    with Context(0) as ctx:
        ctx.set_theta(0.3)
        e = err_report(*ctx.forces(*a, 0, "tree"), *ctx.forces(*a, 0, "fp64"))
    assert e["acc_rms"] <= 2e-4 and e["pot_max"] <= 2e-4, e


def test_batch_across_tiles():
    sizes = [0, 1500, 700, 1, 0, 3000, 2049, 90, 0]
    parts = [_model(max(n, 70), 7 + k) for k, n in enumerate(sizes)]
    x, y, z, m, r2 = (np.concatenate([p[q][:n] for p, n in zip(parts, sizes)]) for q in range(5))
    offs = np.concatenate([[0], np.cumsum(sizes)])
    with Context(0) as ctx:
        ctx.set_theta(0.3)
        tree = ctx.batch_forces(offs, x, y, z, m, r2, 0, "tree")
        ref = ctx.batch_forces(offs, x, y, z, m, r2, 0, "fp64")
    for a, b in zip(offs[:-1], offs[1:]):
        if b - a > 1:
            e = err_report(*(v[a:b] for v in tree[:4]), *(v[a:b] for v in ref[:4]))
            assert e["acc_rms"] <= 5e-4 and e["pot_max"] <= 5e-4, (a, b, e)
    assert np.allclose(tree[4], ref[4], rtol=1e-4)


def _runs(n, seed):
    """A model with a third of its particles in runs of 2 to 16 coincident ones of
    different masses, in the caller's order all over the tiles."""
    s = inputs.single_polytrope(n, 1.5, seed=seed)
    x, y, z, m, r2 = (getattr(s, f).copy() for f in ("x", "y", "z", "m", "range2"))
    rng = np.random.default_rng(seed)
    m *= rng.uniform(0.5, 2.0, n)
    pick, runs, k = rng.permutation(n)[: n // 3], [], 0
    while k + 16 <= len(pick):
        runs.append(np.sort(pick[k : k + rng.integers(2, 17)]))
        k += 16
    for run in runs:
        for v in (x, y, z):
            v[run] = v[run[0]]
    return (x, y, z, m, r2), runs


# a set alone and beside another: sorted in tiles and device-wide, or the other way round
@pytest.mark.parametrize("n1, n2", [(40000, 30000), (65536, 300), (6001, 60000), (3000, 4000), (4096, 2049)])
def test_equal_keys_keep_the_caller_order(n1, n2):
    a, runs = _runs(n1, 3)
    b, _ = _runs(n2, 4)
    both = [np.concatenate(v) for v in zip(a, b)]
    swapped = [v.copy() for v in a]
    for run in runs:  # the run's masses and H in the opposite order
        for v in swapped[3:]:
            v[run] = v[run[::-1]]
    back = np.arange(n1)
    for run in runs:
        back[run] = run[::-1]
    with Context(0) as ctx:
        ctx.set_theta(0.5)
        alone = ctx.forces(*a, 0, "tree")
        batch = ctx.batch_forces([0, n1, n1 + n2], *both, 0, "tree")
        other = ctx.forces(*swapped, 0, "tree")
    assert all(np.array_equal(v, w[:n1]) for v, w in zip(alone, batch))
    # the same particles with equal keys in another order: the bits do depend on it
    assert not np.array_equal(alone[0], other[0][back])
