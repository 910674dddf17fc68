"""The mixed hydro list pass and the mixed density with div and curl add a
particle's pairs one by one in list order.

Clouds of one and the same cluster, small enough that a walk takes its particles
in Morton order and all of them are neighbours.  In the first clouds a single
particle has mass, which gives every pair's term alone; in the others the masses
are powers of two over twenty binades, so that every product of a mass and a
term is exact and the FP32 sum in list order is known to the last bit, and no
other order gives it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = 60


def _in_order(terms, mass, order):
    """float32 sums over j, in `order`, of mass[c, j] * terms[j, i]: [c, i]"""
    out = np.zeros((mass.shape[0], terms.shape[1]), np.float32)
    for j in order:
        out += (mass[:, j, None] * terms[None, j, :]).astype(np.float32)
    return out


@pytest.mark.parametrize("clouds", [80, 700, 1150])  # either side of the sizes where lanes or warps share the work
def test_list_order(clouds):
    from sph_3_b200 import Config, Context
    rng = np.random.default_rng(clouds)
    one = rng.normal(scale=0.1, size=(K, 3))
    pos = np.tile(one, (clouds, 1))
    mass = np.zeros((clouds, K))
    mass[:K] = np.eye(K)
    mass[K:] = 2.0 ** rng.integers(-10, 11, size=(clouds - K, K))
    n = K * clouds
    with Context(Config(precision="mixed", visc="signal", gravity=False)) as ctx:
        ctx.set_clouds([K] * clouds)
        # an expanding set: no viscosity, so a pair's factor is its mass times P_i/rho_i^2 + P_j/rho_j^2
        ctx.set_particles(pos, mass.reshape(-1), vel=pos, u=np.ones(n), h=np.full(n, 0.6))
        ctx.compute("density", "divcurl")
        order = ctx.morton_order()[0][:K]
        assert sorted(order) == list(range(K))
        rho = ctx.get_field("rho").reshape(clouds, K).astype(np.float32)
        for f, v in (("rho", 1.0), ("P", 0.5), ("c", 1.0)):
            ctx.set_field(f, np.full(n, v))
        both = []
        for what in (("acc_sph", "dudt"), ("acc_sph",), ("dudt",)):
            ctx.compute(*what)
            both.append((ctx.get_field("acc_sph"), ctx.get_field("dudt")))
    for acc, dudt in both:
        acc = acc.reshape(clouds, K, 3).astype(np.float32)
        dudt = dudt.reshape(clouds, K).astype(np.float32)
        for got in (acc[..., 0], acc[..., 1], acc[..., 2], dudt):
            assert np.array_equal(got[K:], _in_order(got[:K], mass[K:], order))
    if n > 36000:  # a team's warps add up their shares apart
        assert np.array_equal(rho[K:], _in_order(rho[:K], mass[K:], order))
