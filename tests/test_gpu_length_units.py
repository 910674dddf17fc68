"""FP64 neighbour counts and densities do not depend on the unit of length, also
where squared distances overflow FP32 (a cloud of 10 pc is 3e19 cm across) or
fall below its normal range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(oc, n, unit):
    from sph_3_b200 import Config, Context
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3)) * unit
    h = unit * (20.0 / n) ** (1 / 3) * (0.3 + rng.random(n))
    rows = np.arange(0, n, max(1, n // 400))
    cnt = oc.count_within(pos, h, rows=rows)
    # the window takes every count: the search stops at its first
    with Context(Config(precision="fp64", gravity=False, h_mode="refstep", n_ngb=100000, n_ngb_tol=99999)) as ctx:
        ctx.set_particles(pos, np.full(n, 1.0 / n), h=h)
        ctx.compute("h")
        assert np.array_equal(ctx.get_field("nngb")[rows], cnt)
        ctx.compute("density")
        rho = oc.density_rows(pos, np.full(n, 1.0 / n), h, rows=rows)
        assert np.max(np.abs(ctx.get_field("rho")[rows] / rho - 1.0)) < 1e-12


@pytest.mark.parametrize("unit", [1.0, 1e18, 1e19, 1e21])
@pytest.mark.parametrize("n", [5, 333, 9001])  # one warp and teams of warps per group; odd batches
def test_counts(oc, n, unit):
    _check(oc, n, unit)


@pytest.mark.parametrize("n,unit", [(333, 1e-21), (9001, 1e-21), (9001, 1e-22), (9001, 1e-24)])
def test_small_units(oc, n, unit):
    _check(oc, n, unit)
