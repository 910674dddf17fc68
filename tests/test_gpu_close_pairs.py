"""FP64 gravity of particles closer than the square root of the smallest normal
number: their softened force is finite, in the walk and in the direct sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sep", [1e-100, 1e-153, 1e-155, 1e-160, 3e-162])
@pytest.mark.parametrize("n", [2, 64, 7000])
def test_close_pair(oc, n, sep):
    from sph_3_b200 import Config, Context
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3))
    pos[0] = 0.0
    pos[1] = [sep, -sep, 0.5 * sep]
    m = rng.random(n) + 0.5
    eps = np.full(n, 0.05)
    rows = np.arange(min(n, 64))
    with Context(Config(precision="fp64", theta=0.0)) as ctx:
        ctx.set_particles(pos, m, eps=eps)
        ctx.compute("gravity")
        acc, phi = ctx.get_field("acc_g")[rows], ctx.get_field("phi")[rows]
        direct, _ = ctx.gravity_direct_rows(rows)
    ref = oc.grav_direct_rows(pos, m, 1.0, eps, rows=rows)
    assert np.all(np.isfinite(phi))
    # n terms of either sign, a few roundings each
    tol = 1e-13 * np.sqrt(n) * np.sqrt(np.mean(ref ** 2))
    assert np.max(np.abs(acc - ref)) <= tol
    assert np.max(np.abs(direct - ref)) <= tol
