"""The walks at the set sizes where several warps share a group (teams of 8, 4
and 2, chosen by the particle count): results on either side of each limit and
for the smallest sets, against the oracle; a row-restricted pass gives the
bits of the full one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 33, 700, 2500, 2501, 6000, 6001, 14001, 18001, 20001, 35001]


def _ic(n):
    from sph_3_b200.ic import evrard
    ic = evrard(n, seed=n)
    ic["vel"] = np.random.default_rng(n).normal(scale=0.3, size=(n, 3))
    return ic


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / (np.sqrt(np.mean(b ** 2)) + 1e-300)) if b.size else 0.0


@pytest.mark.parametrize("n", SIZES + [45001, 50001, 90001, 110001])
@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_passes_against_oracle(oc, n, prec):
    from sph_3_b200 import Config, Context
    ic = _ic(n)
    tol = 1e-10 if prec == "fp64" else 1e-5
    n_ngb = min(64, max(6, n // 4))
    with Context(Config(precision=prec, n_ngb=n_ngb, h_max_iter=64)) as ctx:
        r = np.linalg.norm(ic["pos"], axis=1)
        h = 0.5 * (3 * n_ngb * 2 * np.pi * np.maximum(r, 0.05) / (4 * np.pi * n)) ** (1 / 3) + 1e-3
        ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"], h=h)
        rows = np.unique(np.random.default_rng(1).integers(0, n, min(n, 96)))
        if n > 100:
            ctx.compute("h")
            got = ctx.get_field("nngb")
            assert np.all(np.abs(got - n_ngb) <= 5)
            hh = ctx.get_field("h")
            cnt = oc.count_within(ic["pos"], hh, rows=rows)
            # FP32 distances may move a particle across 2h
            assert np.max(np.abs(cnt - got[rows])) <= (0 if prec == "fp64" else 1)
        else:
            hh = h
        ctx.compute("density", "divcurl")
        rho = oc.density_rows(ic["pos"], ic["m"], hh, rows=rows)
        assert _rel(ctx.get_field("rho")[rows], rho) < tol
        full = ctx.get_field("rho")
        dv, cv = oc.div_curl_rows(ic["pos"], ic["vel"], full, ic["m"], hh, rows=rows)
        assert _rel(ctx.get_field("divV")[rows], dv) < 100 * tol
        assert _rel(ctx.get_field("curlV")[rows], cv) < 100 * tol
        ctx.compute("density")
        assert _rel(ctx.get_field("rho")[rows], rho) < tol
        ctx.compute("gravity")
        acc, phi = ctx.gravity_direct_rows(rows)
        err = np.linalg.norm(ctx.get_field("acc_g")[rows] - acc, axis=1)
        assert np.median(err) <= 1e-3 * np.sqrt(np.mean(np.sum(acc ** 2, axis=1))) + 1e-300
        assert _rel(ctx.get_field("phi")[rows], phi) < 5e-3
        assert ctx.status() == 0, ctx.status_names()


@pytest.mark.parametrize("n", [1500, 5000, 12000, 30000])
@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_rows_keep_the_bits_and_lists_the_pairs(oc, n, prec):
    from sph_3_b200 import Config, Context
    ic = _ic(n)
    b, e = n // 3, n // 3 + 200
    out = []
    whole_h = None
    for rows in (None, (b, e)):
        with Context(Config(precision=prec)) as ctx:
            ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"])
            ctx.compute("boot_h")
            ctx.compute("h", rows=rows)
            vals = [ctx.get_field("h", rows=(b, e))]
            # a restricted h search leaves the other rows' h undefined
            whole_h = ctx.get_field("h") if whole_h is None else whole_h
            ctx.set_field("h", whole_h)
            ctx.compute("density", rows=rows)
            vals.append(ctx.get_field("rho", rows=(b, e)))
            ctx.compute("gravity", rows=rows)
            vals.append(ctx.get_field("acc_g", rows=(b, e)))
            out.append(vals)
            if rows is None and prec == "mixed":
                h = ctx.get_field("h")
                for r, got in zip(range(b, b + 20), ctx.pair_lists(np.arange(b, b + 20))):
                    ref = oc.neighbours(ic["pos"], h, r)
                    assert np.setxor1d(got, ref).size <= 1 and np.all(np.diff(got) > 0)
    for x, y in zip(*out):
        assert np.array_equal(x, y)
