"""The context's Morton sort at the sizes where its way changes: all-pairs
ranking up to 16,384 keys of at most 62 bits, radix passes with tiles of 1024,
2048 and 4096 keys above, an odd or even number of passes, remainders of every
chunk and tile, and many equal keys (ties keep the caller's order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(pos, max_level, counts=None):
    from oracle import morton
    from sph_3_b200 import Config, Context
    n = pos.shape[0]
    with Context(Config(max_level=max_level)) as ctx:
        if counts is not None:
            ctx.set_clouds(counts)
        ctx.set_particles(pos, np.full(n, 1.0 / n))
        order, keys = ctx.morton_order()
        o_ref, k_ref = morton.order(pos, max_level, counts)
        assert np.array_equal(keys, k_ref)
        assert np.array_equal(order, o_ref)
        assert ctx.status() == 0, ctx.status_names()


def _points(n, seed, ties):
    pos = np.random.default_rng(seed).random((n, 3))
    if ties:  # at most 64 different places: long runs of equal keys
        pos = np.floor(pos * 4.0) / 4.0
    return pos


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 255, 256, 257, 2047, 2049, 16383, 16384, 16385, 17408, 17409])
def test_sizes(n, ties):
    # equal places make leaves of more than leaf_size particles at the deepest level
    _check(_points(n, n, ties), 16)


@pytest.mark.parametrize("n,max_level", [(400000, 16), (400001, 16), (1600001, 16), (20011, 6), (20011, 19),
                                         (5003, 4), (5003, 20)])
def test_tiles_and_passes(n, max_level):
    _check(_points(n, 3, False), max_level)


@pytest.mark.parametrize("n", [9000, 30000])
def test_63_bit_keys_in_the_last_cells(n):
    # level 21: keys of 63 bits, the largest in the far corner of the root cube
    pos = _points(n, 5, False)
    pos[: n // 2] = 1.0 - 1e-3 * pos[: n // 2] ** 4
    pos[7] = pos[11] = 1.0 - 1e-9
    _check(pos, 21)


@pytest.mark.parametrize("counts", [(1, 0, 31, 700, 2048), (9000, 12000, 3)])
def test_several_clouds(counts):
    _check(_points(sum(counts), 9, False), 16, counts)
