"""The reference-order gravity sums at the sizes where their blocks change
(rows per block, whole and partial source tiles, slices and partial arrays
that start or end inside a tile, pairs near |r| = 2 eps), bit for bit against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n, seed=0):
    rng = np.random.default_rng(seed + n)
    pos = rng.random((n, 3))
    return pos, rng.random(n) + 0.5, 0.02 + 0.05 * rng.random(n)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 127, 128, 129, 513, 2959, 2961, 6001])
def test_full_field(oc, n):
    from sph_3_b200 import libsx
    pos, m, eps = _case(n)
    assert np.array_equal(libsx.getAcc_g_smth(pos, m, 1.3, eps), oc.getAcc_g_smth(pos, m, 1.3, eps))


@pytest.mark.parametrize("nbeg,nend", [(0, 1), (1, 700), (127, 129), (640, 1000), (999, 1000)])
def test_slices_and_partial_arrays(oc, nbeg, nend):
    from sph_3_b200 import libsx
    pos, m, eps = _case(1000)
    assert np.array_equal(libsx.getAcc_g_smth_mpi(nbeg, nend, pos, m, 1.0, eps),
                          oc.getAcc_g_smth_mpi(nbeg, nend, pos, m, 1.0, eps))
    assert np.array_equal(libsx.getAcc_g_smth_mimj_mpi(nbeg, nend, pos, m, 1.0, eps),
                          oc.getAcc_g_smth_mimj_mpi(nbeg, nend, pos, m, 1.0, eps))


def test_pairs_at_the_edges_of_the_kernel(oc):
    """Distances of exactly eps, 2 eps and their neighbouring doubles: the
    pieces of the kernel are chosen by the rounded quotient."""
    from sph_3_b200 import libsx
    e = 0.05
    x = [0.0]
    for c in (e, 2.0 * e):
        lo = hi = c
        for _ in range(6):
            x += [lo, hi]
            lo, hi = np.nextafter(lo, 0.0), np.nextafter(hi, 1.0)
    pos = np.zeros((len(x), 3))
    pos[:, 0] = x
    m = np.ones(len(x))
    eps = np.full(len(x), e)
    assert np.array_equal(libsx.getAcc_g_smth(pos, m, 1.0, eps), oc.getAcc_g_smth(pos, m, 1.0, eps))
