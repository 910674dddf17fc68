"""The mixed hydro pair terms round as they always did: accelerations, du/dt and
signal velocities of a small set, by the walk and by the list pass, against bits
recorded on a B200 (tests/golden/hydro_mixed_bits.npz, written by running this file
with the output's name).  A change of rounding here travels through the h rule's
windows into whole runs, so it has to be meant."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 60  # one leaf: the pairs are met in Morton order
FORMS = (("acc_sph", "dudt"), ("acc_sph",), ("dudt",))


def _run(visc, lists):
    from sph_3_b200 import Config, Context
    rng = np.random.default_rng(7)
    pos = rng.normal(size=(N, 3))
    vel = rng.normal(size=(N, 3))
    m, u, h = rng.random(N) + 0.5, rng.random(N) + 0.5, 0.5 + 0.5 * rng.random(N)
    rho, P, c, bal = (rng.random(N) + 0.5 for _ in range(4))
    out = {}
    with Context(Config(precision="mixed", visc=visc, gravity=False)) as ctx:
        ctx.set_particles(pos, m, vel=vel, u=u, h=h)
        if lists:
            ctx.compute("density")
        for f, v in (("rho", rho), ("P", P), ("c", c), ("balsara", bal)):
            ctx.set_field(f, v)
        for what in FORMS:
            ctx.compute(*what)
            for f in what + (("vsig",) if "acc_sph" in what else ()):
                out["%s_%s_%s_%s" % (visc, "list" if lists else "walk", "".join(w[0] for w in what), f)] = \
                    ctx.get_field(f).astype(np.float32)
    return out


@pytest.mark.parametrize("lists", [False, True])
@pytest.mark.parametrize("visc", ["signal", "mg83", "balsara"])
def test_bits(golden, visc, lists):
    ref = golden("hydro_mixed_bits")
    for k, v in _run(visc, lists).items():
        assert np.any(v != 0) and np.array_equal(v, ref[k]), k


if __name__ == "__main__":
    import sys
    bits = {}
    for visc in ("signal", "mg83", "balsara"):
        for lists in (False, True):
            bits.update(_run(visc, lists))
    np.savez_compressed(sys.argv[1], **bits)
