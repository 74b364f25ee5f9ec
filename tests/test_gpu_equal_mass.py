"""The split kernel's equal-mass tiles: models of one mass, of one mass but for
single particles, and lengths near both ends of the range in which the mass is
factored out, against the FP64 kernel."""
import numpy as np
import pytest

from starsmasher_b200 import inputs

from conftest import err_report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 257, 1023, 5000])
@pytest.mark.parametrize("odd", [0, 1, 40])
def test_masses(gpu_ctx, n, odd):
    s = inputs.single_polytrope(n, 1.5, seed=n + odd)
    m = s.m.copy()
    m[np.random.default_rng(odd).choice(n, odd, replace=False)] *= 1.75
    ref = gpu_ctx.forces(s.x, s.y, s.z, m, s.range2, 0, "fp64")
    e = err_report(*gpu_ctx.forces(s.x, s.y, s.z, m, s.range2, 0, "f32split"), *ref)
    assert e["acc_max"] <= 1e-6 and e["pot_max"] <= 1e-6, e


# mass-free terms reach 1/r^3: past 1e-12 < r < 1e12 the kernel multiplies per pair
@pytest.mark.parametrize("scale", [1e-11, 1e-8, 1e8, 1e11, 1e12])
def test_length_units(gpu_ctx, scale):
    s = inputs.single_polytrope(4000, 1.5, seed=3)
    a = (s.x * scale, s.y * scale, s.z * scale, s.m, s.range2 * scale ** 2)
    ref = gpu_ctx.forces(*a, 0, "fp64")
    e = err_report(*gpu_ctx.forces(*a, 0, "f32split"), *ref)
    assert e["acc_max"] <= 1e-6 and e["pot_max"] <= 1e-6, e


@pytest.mark.parametrize("n", [30000, 140000])
def test_rounding_of_the_mass(gpu_ctx, n):
    """Potentials per unit mass of a model whose mass FP32 rounds by nearly 2^-24, against
    those of unit masses: the far tiles, most of the sums, must not share that rounding."""
    s = inputs.single_polytrope(n, 1.5, seed=4)
    one = np.ones(n)
    m = 1.0 + 0.98 * 2.0 ** -24
    a = gpu_ctx.forces(s.x, s.y, s.z, one, s.range2, 0, "f32split")[3]
    b = gpu_ctx.forces(s.x, s.y, s.z, m * one, s.range2, 0, "f32split")[3] / m
    assert abs(np.mean(b / a) - 1.0) <= 0.4 * 2.0 ** -24
