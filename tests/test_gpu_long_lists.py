"""FP64 forces from a given density where the caller's h gives more pairs than a
list holds: the lists are given up early (few candidates tested) and the walk gives
the bits it gives without lists; distances on the support's very edge too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(pos, vel, m, h, cap, visc):
    from sph_3_b200 import Config, Context
    n = len(m)
    with Context(Config(precision="fp64", gravity=False, list_cap=cap, visc=visc)) as ctx:
        ctx.set_particles(pos, m, vel=vel, h=h)
        for f, v in (("rho", 1.0 + 0.1 * np.sin(np.arange(n))), ("P", np.full(n, 0.4)), ("c", np.full(n, 0.8))):
            ctx.set_field(f, v)
        ctx.counters(clear=True)
        ctx.compute("acc_sph", "dudt")
        assert ctx.status() == 0, ctx.status_names()
        return [ctx.get_field(f) for f in ("acc_sph", "dudt", "vsig")], ctx.counters()


@pytest.mark.parametrize("visc", ["signal", "mg83", "balsara"])
@pytest.mark.parametrize("n", [600, 7000, 40000])  # teams of 8, teams of 4, a warp per group
def test_overflowing_lists(oc, n, visc):
    rng = np.random.default_rng(n)
    pos, vel, m = rng.random((n, 3)), rng.normal(size=(n, 3)), np.full(n, 1.0 / n)
    h = 0.5 * (3 * 300 / (4 * np.pi * n)) ** (1 / 3) * (0.8 + 0.4 * rng.random(n))
    walked, _ = _run(pos, vel, m, h, 0, visc)
    full, all_pairs = _run(pos, vel, m, h, 1024, visc)
    cut, few_pairs = _run(pos, vel, m, h, 8, visc)
    for a, b, c in zip(walked, full, cut):
        assert np.array_equal(a, b) and np.array_equal(a, c)
    assert few_pairs["density_pairs"] < all_pairs["density_pairs"] // 2
    rows = np.arange(0, n, max(1, n // 200))
    a_ref, _ = oc.hydro_rows(pos, vel, 1.0 + 0.1 * np.sin(np.arange(n)), np.full(n, 0.4), np.full(n, 0.8), h, m,
                             {"signal": 0, "mg83": 1, "balsara": 0}[visc], 1.0, 2.0, 0.1, rows=rows)
    if visc != "balsara":
        assert np.max(np.abs(walked[0][rows] - a_ref)) <= 1e-10 * np.sqrt(np.mean(a_ref ** 2))


@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_walk_on_the_edge(oc, ulps):
    k, s = 12, 1.0 / 16.0
    g = np.arange(k) * s
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    n = k ** 3
    h = np.full(n, s if ulps == 0 else np.nextafter(s, 1.0 if ulps > 0 else 0.0))
    m, vel = np.full(n, 1.0 / n), np.random.default_rng(1).normal(size=(n, 3))
    (acc, dudt, _), cnt = _run(pos, vel, m, h, 0, "signal")
    a_ref, du_ref = oc.hydro_rows(pos, vel, 1.0 + 0.1 * np.sin(np.arange(n)), np.full(n, 0.4), np.full(n, 0.8), h, m,
                                  0, 1.0, 2.0, 0.1)
    # an in-support pair at q = 2 adds exactly 0, so the pair sets are compared through the lists
    for x, ref in ((acc, a_ref), (dudt, du_ref)):
        assert np.max(np.abs(x - ref)) <= 1e-10 * np.sqrt(np.mean(ref ** 2))
    (acc2, dudt2, _), _ = _run(pos, vel, m, h, 512, "signal")
    assert np.array_equal(acc, acc2) and np.array_equal(dudt, dudt2)
