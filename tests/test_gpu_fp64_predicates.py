"""The FP64 path settles most distance tests in FP32 and only a narrow band
around the radius exactly: lattices whose distances equal the radii to the last
bit, radii one ulp either side, and clustered sets whose h is tiny against the
root cube give the oracle's pair sets and neighbour counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(k, s):
    g = np.arange(k) * s
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)


def _cluster(n):
    rng = np.random.default_rng(n)
    pos = rng.normal(scale=1e-4, size=(n, 3))
    pos[0], pos[1] = -1.0, 1.0  # the root cube is 20,000 times the cluster
    return pos


@pytest.mark.parametrize("case", ["equal", "above", "below", "cluster"])
@pytest.mark.parametrize("k", [8, 14, 22])
def test_pairs_and_counts(oc, case, k):
    from sph_3_b200 import Config, Context
    s = 1.0 / 16.0
    if case == "cluster":
        pos = _cluster(k ** 3)
        n = pos.shape[0]
        h = np.full(n, 4e-5)
    else:
        pos = _lattice(k, s)
        n = pos.shape[0]
        # |r| <= h_i + h_j with |r| = s, 2 s, ... : exactly on the radius, or one ulp off it
        h = np.full(n, {"equal": s, "above": np.nextafter(s, 1.0), "below": np.nextafter(s, 0.0)}[case])
    m = np.full(n, 1.0 / n)
    u = np.full(n, 0.5)
    with Context(Config(precision="fp64", gravity=False, list_cap=512, leaf_size=16)) as ctx:
        ctx.set_particles(pos, m, u=u, h=h)
        ctx.compute("density", "acc_sph", "dudt")
        pairs = sum(oc.neighbours(pos, h, i).size for i in range(n)) if n <= 3000 else None
        if pairs is not None:
            assert ctx.counters()["hydro_pairs"] == pairs
        rows = np.arange(0, n, max(1, n // 200))
        rho = oc.density_rows(pos, m, h, rows=rows)
        assert np.max(np.abs(ctx.get_field("rho")[rows] / rho - 1.0)) < 1e-12
    # counts d < 2h of the search: the reference's rule stops at once where the count is in the window
    rows = np.arange(0, n, max(1, n // 200))
    cnt = oc.count_within(pos, h, rows=rows)
    with Context(Config(precision="fp64", gravity=False, h_mode="refstep", n_ngb=100000, n_ngb_tol=99999)) as ctx:
        ctx.set_particles(pos, m, h=h)
        ctx.compute("h")
        assert np.array_equal(ctx.get_field("nngb")[rows], cnt)
