"""The octree build at the sizes where its kernels change: tiles of 512
particles in the topology pass, moments in one launch or two, leaf sizes at
both ends, equal keys, several clouds.  Node and leaf counts against a NumPy
restatement of the tree's definition; theta = 0 gravity (which visits every
particle through the tree) against the FP64 direct sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _count(keys, max_level, leaf_size):
    """(nodes, leaves) of one cloud's sorted keys: a run of more than leaf_size
    keys is split on the first 3-bit digit its keys differ in."""
    nodes = leaves = 0
    todo = [(0, len(keys))]
    while todo:
        s, e = todo.pop()
        nodes += 1
        x = int(keys[s]) ^ int(keys[e - 1]) if e > s else 0
        lvl = max_level if x == 0 else max_level - 1 - (x.bit_length() - 1) // 3
        if e - s <= leaf_size or lvl >= max_level:
            leaves += 1
            continue
        dg = (keys[s:e] >> np.uint64(3 * (max_level - lvl - 1))) & np.uint64(7)
        cut = np.flatnonzero(np.diff(dg.astype(np.int64))) + 1
        bounds = [0, *cut.tolist(), e - s]
        todo += [(s + a, s + b) for a, b in zip(bounds[:-1], bounds[1:])]
    return nodes, leaves


def _run(pos, leaf_size=16, max_level=16, counts=None, rows=64):
    from oracle import morton
    from sph_3_b200 import Config, Context
    n = pos.shape[0]
    rng = np.random.default_rng(n)
    m = rng.random(n) + 0.5
    with Context(Config(precision="fp64", theta=0.0, leaf_size=leaf_size, max_level=max_level)) as ctx:
        if counts is not None:
            ctx.set_clouds(counts)
        ctx.set_particles(pos, m)
        c = ctx.counters()
        nodes = leaves = beg = 0
        for cnt in counts if counts is not None else [n]:
            a, b = _count(np.sort(morton.keys(pos[beg:beg + cnt], max_level)), max_level, leaf_size)
            nodes, leaves, beg = nodes + a, leaves + b, beg + cnt
        assert (c["tree_nodes"], c["tree_leaves"]) == (nodes, leaves)
        ctx.compute("gravity")
        got = ctx.get_field("acc_g")
        r = np.unique(rng.integers(0, n, min(n, rows)))
        ref, _ = ctx.gravity_direct_rows(r)
        scale = np.sqrt(np.mean(ref ** 2)) + 1e-300
        # the same FP64 pair terms in another order: n terms, 1e-16 each
        assert np.max(np.abs(got[r] - ref)) <= 1e-15 * max(n, 100) * scale
        assert ctx.status() == 0, ctx.status_names()


@pytest.mark.parametrize("n", [1, 2, 16, 17, 31, 33, 511, 512, 513, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("leaf_size", [1, 16, 64])
def test_sizes_and_leaf_sizes(n, leaf_size):
    _run(np.random.default_rng(n).random((n, 3)), leaf_size)


@pytest.mark.parametrize("max_level", [4, 16, 21])
def test_equal_keys(max_level):
    # 64 places, 30 particles each: leaves at the deepest level hold more than leaf_size
    pos = np.floor(np.random.default_rng(1).random((1920, 3)) * 4.0) / 4.0
    pos += 1e-9 * np.random.default_rng(2).random(pos.shape)
    _run(pos, 8, max_level)


@pytest.mark.parametrize("counts", [(1, 0, 511, 1, 513), (0, 600, 0), (512, 512, 512)])
def test_clouds(counts):
    _run(np.random.default_rng(3).random((sum(counts), 3)), 16, 16, counts)


@pytest.mark.parametrize("n", [99999, 100001])
def test_moments_in_one_launch_and_two(n):
    """Evrard spheres either side of the limit: Barnes-Hut gravity (all moments)
    against the direct sum, to the multipole error."""
    from sph_3_b200 import Config, Context
    from sph_3_b200.ic import evrard
    ic = evrard(n, seed=2)
    with Context(Config(precision="fp64")) as ctx:
        ctx.set_particles(ic["pos"], ic["m"], vel=ic["vel"], u=ic["u"])
        ctx.compute("gravity")
        r = np.random.default_rng(1).choice(n, 512, replace=False)
        ref, phi = ctx.gravity_direct_rows(r)
        err = np.linalg.norm(ctx.get_field("acc_g")[r] - ref, axis=1) / np.linalg.norm(ref, axis=1)
        assert np.median(err) < 1e-3 and err.max() < 1e-2
        assert np.max(np.abs(ctx.get_field("phi")[r] / phi - 1.0)) < 1e-3
