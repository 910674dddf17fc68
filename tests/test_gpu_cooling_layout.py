"""Cooling tables whose dimensions exercise the device layout and the copies of
the species rows: one point in a dimension, N_M that is not a multiple of four,
ion-fraction arrays that do not start on 16 bytes, ragged particle counts, bit
for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 2, 1, 2, 1, 2), (3, 7, 5, 3, 4, 1), (5, 64, 4, 2, 12, 6), (4, 33, 9, 3, 17, 5),
                                  (2, 16, 3, 2, 3, 9)])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000])
def test_rows_and_columns(oc, dims, n):
    import torch
    from sph_3_b200 import cooling
    tab = cooling.seeded_table(seed=sum(dims), dims=dims)
    units = cooling.Units(unit_density_cgs=1e-24, unit_time_s=3e13, unit_u_cgs=1e12, unit_length_cm=3.086e21)
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * 4 - 2).astype(np.float32)
    rho = (10.0 ** (rng.random(n) * 8 - 4)).astype(np.float32)
    u = (10.0 ** (rng.random(n) * 6 - 3)).astype(np.float32)
    typ = (rng.random(n) < 0.2).astype(np.int32)
    ref_u, ref_ion = oc.hcooling(tab, units.as_tuple(), 1e-3, u, rho, pos, typ=typ)
    t = cooling.CoolTable(tab)
    got_u, got_ion = cooling.hcooling(t, units, 1e-3, u, rho, pos, typ=typ)
    gas = typ == 0
    assert np.array_equal(got_u, ref_u)
    assert np.array_equal(got_ion[gas], ref_ion[gas])
    # an ion-fraction array that starts 4 bytes past a 16-byte boundary
    import ctypes
    from sph_3_b200 import _lib
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    us, rs, ts, xs = dev(u), dev(rho), dev(typ), [dev(pos[:, k]) for k in range(3)]
    room = torch.zeros(n * dims[4] + 1, dtype=torch.float32, device="cuda")
    cu = units.to_c()
    P = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    _lib.check(_lib.load().sph3_hcooling(t.handle, ctypes.byref(cu), ctypes.c_float(1e-3), n, P(ts), P(us), P(rs),
                                         P(xs[0]), P(xs[1]), P(xs[2]), ctypes.c_void_p(room.data_ptr() + 4), None,
                                         ctypes.c_void_p(0)), "hcooling")
    torch.cuda.synchronize()
    ion = room.cpu().numpy()[1:].reshape(n, dims[4])
    assert np.array_equal(ion[gas], ref_ion[gas]) and not ion[~gas].any()
    t.close()
