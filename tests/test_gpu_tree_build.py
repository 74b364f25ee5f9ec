"""The tree's one-pass build and the split walk: sizes around a leaf, a group,
the padding and the particle counts where the walk's parts change; theta = 0
opens every node, so the result must be the direct sum (far pairs in FP32)."""
import numpy as np
import pytest

from starsmasher_b200 import Context, inputs

from conftest import err_report

pytestmark = pytest.mark.gpu


def _direct_and_tree(ctx, a, theta, nkernel=0):
    ref = ctx.forces(*a, nkernel, "fp64")
    ctx.set_theta(theta)
    return ref, ctx.forces(*a, nkernel, "tree")


@pytest.mark.parametrize("n", [2, 16, 17, 32, 33, 255, 256, 257, 1029])
def test_small_sets(n):
    s = inputs.single_polytrope(max(n, 70), 1.5, seed=n)
    a = [getattr(s, f)[:n].copy() for f in ("x", "y", "z", "m", "range2")]
    a[4] *= 0.05
    if n > 40:  # coincident particles: a leaf that cannot split
        for v in a[:3]:
            v[5:45] = v[5]
    with Context(0) as ctx:
        ref, got = _direct_and_tree(ctx, a, 0.0)
    e = err_report(*got, *ref)
    assert e["acc_max"] <= 2e-6 and e["pot_max"] <= 1e-6, e


# eight parts up to 23,000 particles, then 4, 2 and one walk per group
@pytest.mark.parametrize("n", [22999, 30011, 60013, 120011, 190007])
def test_parts_of_a_walk(n):
    s = inputs.red_giant(n, seed=n % 97)
    a = (s.x, s.y, s.z, s.m, s.range2)
    with Context(0) as ctx:
        ref, got = _direct_and_tree(ctx, a, 0.5)
        assert ctx.tree_stats()[1] >= 1  # the core's group is handed over
        again = ctx.forces(*a, 0, "tree")
        half = ctx.forces(*a, 0, "tree", n // 3, n // 2)
    e = err_report(*got, *ref)
    assert e["acc_rms"] <= 1e-3 and e["pot_rms"] <= 2e-4, e
    assert abs(got[0][0] - ref[0][0]) <= 1e-9 * abs(ref[0][0])  # the core: direct FP64
    sl = slice(n // 3, n // 3 + n // 2)
    for g, r, h in zip(got, again, half):
        assert np.array_equal(g, r) and np.array_equal(g[sl], h[sl])
        assert not h[: n // 3].any()


# a batch's sets are cut into parts as they are alone: 8 and none, 8 and 2, 4 and 8
@pytest.mark.parametrize("model", [inputs.single_polytrope, inputs.red_giant])
@pytest.mark.parametrize("n1, n2", [(1003, 190007), (22999, 100003), (30011, 517)])
def test_batch_of_mixed_parts(model, n1, n2):
    a, b = (model(n, seed=n % 89) for n in (n1, n2))
    f = ("x", "y", "z", "m", "range2")
    both = [np.concatenate([getattr(a, k), getattr(b, k)]) for k in f]
    with Context(0) as ctx:
        ctx.set_theta(0.5)
        got = ctx.batch_forces([0, n1, n1 + n2], *both, 0, "tree")
        heavy = ctx.tree_stats()[1]
        one = ctx.forces(*(getattr(a, k) for k in f), 0, "tree")
        two = ctx.forces(*(getattr(b, k) for k in f), 0, "tree")
    alone = [np.concatenate([u, v]) for u, v in zip(one, two)]
    # the same bits, but for the rows of groups handed to the direct sum, whose
    # source chunks follow from the call's count of them
    other = np.flatnonzero(np.any([g != w for g, w in zip(got, alone)], axis=0))
    assert len(other) <= 32 * heavy
    amag = np.sqrt(sum(w ** 2 for w in alone[:3]))
    for g, w in zip(got[:3], alone[:3]):
        assert (np.abs(g - w)[other] <= 1e-11 * np.median(amag)).all()
    assert np.allclose(got[3], alone[3], rtol=1e-12)


def test_captured_call_with_groups_of_tiny_h():
    """Groups whose largest H^2 is a subnormal float, which the walking order cannot tell
    from the unused entries of a captured call's group list, and coincident particles:
    as the eager call."""
    import torch
    n = 3000
    s = inputs.single_polytrope(n, 1.5, seed=12)
    a = [getattr(s, k).copy() for k in ("x", "y", "z", "m", "range2")]
    a[4][:] = 1e-40
    for v in a[:3]:
        v[100:200] = v[100]
    X = [torch.from_numpy(v).cuda() for v in a]
    out = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(4)]
    with Context(0) as ctx:
        ctx.set_theta(0.5)
        ctx.forces_device(n, *X, *out, nkernel=0, precision="tree")
        ctx.sync()
        want = [t.cpu().numpy() for t in out]
        with ctx.capture() as cap:
            ctx.forces_device(n, *X, *out, nkernel=0, precision="tree")
        for t in out:
            t.zero_()
        torch.cuda.synchronize()
        cap.graph.launch(1)
        ctx.sync()
        assert all(np.array_equal(w, t.cpu().numpy()) for w, t in zip(want, out))


def test_no_direct_sum_plan():
    """The walk has no row tiles: a tree call plans no work items, and one of other rows of
    the same set gives the same bits."""
    s = inputs.single_polytrope(20011, 1.5, seed=2)
    a = (s.x, s.y, s.z, s.m, s.range2)
    with Context(0) as ctx:
        full = ctx.forces(*a, 0, "tree")
        assert ctx.plan_info()["nitems"] == 0
        part = ctx.forces(*a, 0, "tree", 4000, 5000)
        direct = ctx.forces(*a, 0, "f32split")
        assert ctx.plan_info()["nitems"] > 0
        again = ctx.forces(*a, 0, "tree")
        with Context(0) as other:
            assert all(np.array_equal(u, v) for u, v in zip(direct, other.forces(*a, 0, "f32split")))
    for u, v, w in zip(full, part, again):
        assert np.array_equal(u, w) and np.array_equal(u[4000:9000], v[4000:9000])


def test_memory_of_a_small_set_beside_a_large_one():
    """The parts of a small set's walk cost its own results' memory, not the batch's."""
    import torch
    n, small = 400000, 300
    s = inputs.single_polytrope(n + small, 1.5, seed=1)
    X = [torch.from_numpy(getattr(s, k)).cuda() for k in ("x", "y", "z", "m", "range2")]
    out = [torch.zeros(n + small, dtype=torch.float64, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()

    def used(offsets):
        free = torch.cuda.mem_get_info()[0]
        with Context(0) as ctx:
            ctx.set_theta(0.7)
            ctx.batch_forces_device(offsets, *X, *out, nkernel=0, precision="tree")
            ctx.sync()
            return free - torch.cuda.mem_get_info()[0]

    used([0, n])  # loads the kernels
    one = used([0, n])
    assert used([0, n, n + small]) - one < 0.2 * one
