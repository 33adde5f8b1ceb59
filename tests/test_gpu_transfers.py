"""Fields in and out in the reference layout, and the per-plane profile, at
sizes around the 32 x 32 tiles that the transfers move: exact."""
import numpy as np
import pytest

from conftest import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("shape", [(1, 1, 1), (31, 3, 33), (32, 2, 32), (33, 5, 31),
                                   (64, 1, 65), (7, 40, 100), (100, 33, 1)])
def test_fields_round_trip(shape, storage):
    from multiphase_lbm_b200 import capi
    fluid, rho = random_case(shape, seed=sum(shape), rho0=0.3, amp=0.25)
    lat = capi.Lattice(shape, storage=storage)
    lat.set_params(capi.default_params(G=-5.0, rhos=0.2, rho_shift=1.0))
    lat.upload(fluid, rho)
    lat.initialize()
    want = np.where(fluid, rho, np.float32(0.2))
    f64 = storage == 2
    assert np.array_equal(lat.field("fluid"), fluid)
    assert np.array_equal(lat.field("rho"), want)
    assert np.array_equal(lat.field("rho", f64=True), want.astype(np.float64))
    psi = lat.field("psi", f64=f64)
    assert np.allclose(psi, 1 - np.exp(-want.astype(np.float64)), atol=2e-7)
    nf, nl = lat.plane_profile()
    m = fluid.astype(bool)
    assert np.array_equal(nf, m.sum((1, 2)))
    assert np.array_equal(nl, (m & (rho > np.float32(0.2726))).sum((1, 2)))
    # the velocity through the transfer against the momentum of the populations
    lat.iterate(0, 1, write_velocity=True)
    u = lat.field("velocity", f64=f64)
    assert u.shape == shape + (3,) and np.array_equal(
        u[~m], np.zeros_like(u[~m]))
    d64 = lat.field("velocity", f64=True)
    assert np.array_equal(d64.astype(np.float32), u.astype(np.float32))
    f = lat.field("f", f64=True)[m]
    e = np.zeros(57, np.int32)
    capi.lib().mlbm_d3q19(e.ctypes.data, None)
    d = lat.field("rho", f64=True)[m]
    # tau = 1: f = feq(rho, u), whose first moment is rho u
    j = f @ e.reshape(19, 3).astype(np.float64)
    tol = 2e-3 if storage == 1 else 2e-6
    assert np.allclose(j / d[:, None], d64[m], atol=tol)
