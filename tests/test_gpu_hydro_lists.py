"""The list passes of the hydro step at the particle counts and list lengths
where their lanes run out (four or eight lanes per particle), and the FP64
passes that make their own lists: against the oracle, and a restricted pass or
one without lists gives the same bits in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(oc, n, seed=0):
    from sph_3_b200.ic import evrard
    ic = evrard(n, seed=seed + n)
    rng = np.random.default_rng(n)
    ic["vel"] = rng.normal(scale=0.3, size=(n, 3))
    r = np.linalg.norm(ic["pos"], axis=1)
    h = 0.5 * (3 * 50 * 2 * np.pi * np.maximum(r, 0.05) / (4 * np.pi * n)) ** (1 / 3) * (0.5 + rng.random(n))
    rho = oc.density_rows(ic["pos"], ic["m"], h)
    return ic, h, rho, (2.0 / 3.0) * rho * ic["u"], np.sqrt(10.0 / 9.0 * ic["u"])


def _load(ctx, ic, h, rho, P, c):
    ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], h=h)
    for f, v in (("rho", rho), ("P", P), ("c", c)):
        ctx.set_field(f, v)


@pytest.mark.parametrize("visc", ["signal", "mg83"])
@pytest.mark.parametrize("n", [1, 2, 5, 33, 257, 3001])
def test_fp64_forces_from_given_density(oc, n, visc):
    from sph_3_b200 import Config, Context
    st = _state(oc, n)
    ic, h, rho, P, c = st
    out = []
    for cap in (1024, 128, 0):  # all lists; some particles walked; all walked
        with Context(Config(precision="fp64", gravity=False, list_cap=cap, visc=visc)) as ctx:
            _load(ctx, *st)
            ctx.compute("acc_sph", "dudt")
            out.append([ctx.get_field(f) for f in ("acc_sph", "dudt", "vsig")])
            assert ctx.status() == 0, ctx.status_names()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            assert np.array_equal(x, y)
    with Context(Config(precision="fp64", gravity=False, visc=visc)) as ctx:
        _load(ctx, *st)
        b, e = n // 3, n // 3 + max(1, n // 4)
        ctx.compute("acc_sph", "dudt", rows=(b, e))
        for f, x in zip(("acc_sph", "dudt"), out[0]):
            assert np.array_equal(ctx.get_field(f, rows=(b, e)), x[b:e])
    a_ref, du_ref = oc.hydro_rows(ic["pos"], ic["vel"], rho, P, c, h, ic["m"], {"signal": 0, "mg83": 1}[visc], 1.0,
                                  2.0, 0.1)
    for x, ref in zip(out[0], (a_ref, du_ref)):
        assert np.max(np.abs(x - ref)) <= 1e-10 * (np.sqrt(np.mean(ref ** 2)) + 1e-300)


@pytest.mark.parametrize("n", [1, 2, 5, 33, 257, 3001, 12001])
def test_mixed_list_pass(oc, n):
    from sph_3_b200 import Config, Context
    ic, h, rho, P, c = _state(oc, n)
    for cap in (1024, 8):
        with Context(Config(precision="mixed", gravity=False, list_cap=cap)) as ctx:
            ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"], h=h)
            ctx.compute("density", "acc_sph", "dudt")
            rows = np.arange(0, n, max(1, n // 300))
            a_ref, du_ref = oc.hydro_rows(ic["pos"], ic["vel"], rho, P, c, h, ic["m"], 0, 1.0, 2.0, 0.1, rows=rows)
            for f, ref in (("acc_sph", a_ref), ("dudt", du_ref)):
                err = np.abs(ctx.get_field(f)[rows] - ref)
                # the FP32 pair terms cancel in the acceleration: 1e-5 of its rms at the median, 1e-3 at most
                rms = np.sqrt(np.mean(ref ** 2)) + 1e-300
                assert np.median(err) <= 1e-5 * rms and np.max(err) <= 1e-3 * rms
            assert ctx.status() == 0, ctx.status_names()
