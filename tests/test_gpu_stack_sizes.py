"""The deepest walk stack a configuration may ask for, in sets small enough that
several warps share a group: a block takes no more warps than its stacks leave
room for, and the results are those of the default stack."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,walk_warps", [(1000, 4), (10000, 1), (100000, 8)])
def test_deepest_stack(n, walk_warps, precision):
    from sph_3_b200 import Config, Context
    from sph_3_b200.ic import evrard
    ic = evrard(n, seed=n)
    out = []
    for cap in (768, 4096):
        for mode in ("newton", "refstep"):
            with Context(Config(precision=precision, stack_cap=cap, walk_warps=walk_warps, h_mode=mode,
                                visc="balsara")) as ctx:
                ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"],
                                  h=0.5 * (3 * 50 * 2 * np.pi * np.maximum(np.linalg.norm(ic["pos"], axis=1), 0.05)
                                           / (4 * np.pi * n)) ** (1 / 3))
                ctx.compute("h", "density")
                ctx.compute("density", "divcurl", "gravity", "acc_sph", "dudt")
                # the reference's rule may turn back and forth over its window for good
                allowed = ["H_NOT_CONVERGED"] if mode == "refstep" else []
                assert [x for x in ctx.status_names() if x not in allowed] == []
                out.append([ctx.get_field(f) for f in ("h", "rho", "divV", "curlV", "acc_g", "phi", "acc_sph",
                                                       "dudt")])
    # sums over another number of warps, in the pass's precision
    tol = 1e-5 if precision == "mixed" else 1e-12
    for a, b in zip(out[:2], out[2:]):
        assert np.array_equal(a[0], b[0])
        for x, y in zip(a[1:], b[1:]):
            assert np.sqrt(np.mean((x - y) ** 2)) <= tol * np.sqrt(np.mean(x ** 2))
