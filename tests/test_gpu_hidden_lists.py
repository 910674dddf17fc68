"""Pair lists are handed out after a density pass only: lists that FP64 forces from
a given density make for themselves are not the caller's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_lists_from_forces(precision):
    from sph_3_b200 import Config, Context
    from sph_3_b200._lib import Sph3Error
    n = 3000
    rng = np.random.default_rng(1)
    pos, h = rng.random((n, 3)), np.full(n, 0.04)
    rows = np.arange(20)
    with Context(Config(precision=precision, gravity=False)) as ctx:
        ctx.set_particles(pos, np.full(n, 1.0 / n), vel=rng.normal(size=(n, 3)), u=np.ones(n), h=h)
        for f in ("rho", "P", "c"):
            ctx.set_field(f, np.ones(n))
        ctx.compute("acc_sph", "dudt")
        with pytest.raises(Sph3Error):
            ctx.pair_lists(rows)
        ctx.compute("density", "acc_sph")
        lists = ctx.pair_lists(rows)
        ctx.set_field("h", h)
        ctx.compute("acc_sph")
        with pytest.raises(Sph3Error):
            ctx.pair_lists(rows)
        ctx.compute("density")
        for a, b in zip(ctx.pair_lists(rows), lists):
            assert np.array_equal(a, b)
