"""The FP64 refine's plan, row-chunk pass and merge at the edges of its units:
a threshold far below every row's G / |a| lists all requested rows, so the
split-FP32 call must return the FP64 kernel's answer on all of them."""
import numpy as np
import pytest

from starsmasher_b200 import Context, inputs

from conftest import rel_err_vec

pytestmark = pytest.mark.gpu

# FP64 sums in another order: the rows' plain FP64 rounding, 8u sum|t_j| / |a|
# with sum|t_j| / |a| up to ~1e3 on the rows kept below (|a| >= 1e-3 median)
TOL = 8 * 2.0 ** -53 * 1e3


def _check(a, b):
    amag = np.sqrt(b[0] ** 2 + b[1] ** 2 + b[2] ** 2)
    good = amag >= 1e-3 * np.median(amag)
    assert rel_err_vec(*a[:3], *b[:3])[good].max() <= TOL
    assert (np.abs(a[3] - b[3]) / np.abs(b[3])).max() <= TOL


@pytest.mark.parametrize("ni", [1, 31, 32, 33, 127, 128, 129, 3001])
def test_refine_of_every_listed_row(ni):
    s = inputs.config2(seed=9, n_each=3000)
    i0 = 1500  # spans both stars for the larger slices
    with Context(0) as ctx:
        ctx.set_refine(1e-9)
        a = ctx.forces(s.x, s.y, s.z, s.m, s.range2, 0, "f32split", i0, ni)
        assert ctx.last_refine_rows() == ni
        b = ctx.forces(s.x, s.y, s.z, s.m, s.range2, 0, "fp64", i0, ni)
    sl = slice(i0, i0 + ni)
    _check([v[sl] for v in a], [v[sl] for v in b])
    for v in a:  # no other row is written
        assert not v[:i0].any() and not v[i0 + ni:].any()


def test_refine_of_a_batch_with_both_routes():
    sizes = [20, 0, 700, 33, 32, 1025, 1]  # <= 32 listed rows: row-chunk items; more: tiles
    parts = [inputs.single_polytrope(max(n, 70), 1.5, seed=20 + k) for k, n in enumerate(sizes)]
    x, y, z, m, r2 = (np.concatenate([getattr(p, f)[:n] for p, n in zip(parts, sizes)])
                      for f in ("x", "y", "z", "m", "range2"))
    r2 = 0.01 * r2  # every row then has far pairs, so an error scale
    offs = np.concatenate([[0], np.cumsum(sizes)])
    with Context(0) as ctx:
        ctx.set_refine(1e-9)
        a = ctx.batch_forces(offs, x, y, z, m, r2, 1, "f32split")
        # the lone particle has no acceleration and no error scale: not listed
        assert ctx.last_refine_rows() == sum(sizes) - 1
        b = ctx.batch_forces(offs, x, y, z, m, r2, 1, "fp64")
    keep = np.arange(offs[-1]) != offs[-1] - 1
    _check([v[keep] for v in a[:4]], [v[keep] for v in b[:4]])
    assert np.allclose(a[3], b[3], rtol=1e-6) and np.allclose(a[4], b[4], rtol=1e-6)


@pytest.mark.parametrize("nsets", [2048, 2049, 2100])
def test_more_light_rows_than_row_chunk_items(nsets):
    """Sets of 32 rows, all listed: 65,536 row-chunk items hold 2,048 of them."""
    base = inputs.single_polytrope(96, 1.5, seed=5)
    x, y, z, m, r2 = (np.tile(getattr(base, f)[:32], nsets) for f in ("x", "y", "z", "m", "range2"))
    x = x * (1.0 + 1e-3 * np.repeat(np.arange(nsets) % 7, 32))  # not one set over and over
    r2 = 0.01 * r2
    offs = 32 * np.arange(nsets + 1)
    with Context(0) as ctx:
        ctx.set_refine(1e-9)
        a = ctx.batch_forces(offs, x, y, z, m, r2, 0, "f32split")
        assert ctx.last_refine_rows() == 32 * nsets
        b = ctx.batch_forces(offs, x, y, z, m, r2, 0, "fp64")
    _check(a[:4], b[:4])
    assert np.allclose(a[4], b[4], rtol=1e-12)


@pytest.mark.parametrize("n", [3001, 20011, 60000])
@pytest.mark.parametrize("refine", [1.0, 0.0])
def test_point_mass_core(n, refine):
    """A core whose softening sphere holds most of the star: with the refine on
    the split kernel leaves its near pairs to it, without it evaluates them."""
    s = inputs.red_giant(n, seed=n)
    a = (s.x, s.y, s.z, s.m, s.range2)
    with Context(0) as ctx:
        ctx.set_refine(refine)
        got = ctx.forces(*a, 0, "f32split")
        rows = ctx.last_refine_rows()
        ref = ctx.forces(*a, 0, "fp64")
    assert (rows >= 1) == (refine > 0.0)
    amag = np.sqrt(ref[0] ** 2 + ref[1] ** 2 + ref[2] ** 2)
    good = amag >= 1e-3 * np.median(amag)
    e = rel_err_vec(*got[:3], *ref[:3])
    assert e[good].max() <= (1e-6 if refine else 3e-6)
    core = np.sqrt(sum((g[0] - r[0]) ** 2 for g, r in zip(got[:3], ref[:3])))
    assert core <= (1e-9 if refine else 1e-6) * np.median(amag)
    assert abs(got[3][0] - ref[3][0]) <= 1e-6 * abs(ref[3][0])


@pytest.mark.parametrize("n", [20011, 60000])
def test_error_scale_of_a_core(n):
    """The error scale is that of the FP32 tile sums, whether the row's near pairs
    are in the sums or left to the refine, which then takes the row at any threshold."""
    s = inputs.red_giant(n, seed=n)
    a = (s.x, s.y, s.z, s.m, s.range2)
    G = {}
    with Context(0) as ctx:
        ctx.keep_error_scale(True)
        for refine in (0.0, 1.0, 1e6):
            ctx.set_refine(refine)
            got = ctx.forces(*a, 0, "f32split")
            G[refine] = ctx.error_scale(n)
        rows = ctx.last_refine_rows()
        ref = ctx.forces(*a, 0, "fp64")
    assert np.isfinite(G[0.0][0]) and all(np.array_equal(G[0.0], g) for g in G.values())
    assert rows >= 1
    amag = np.sqrt(ref[0] ** 2 + ref[1] ** 2 + ref[2] ** 2)
    assert np.sqrt(sum((g[0] - r[0]) ** 2 for g, r in zip(got[:3], ref[:3]))) <= 1e-9 * np.median(amag)
