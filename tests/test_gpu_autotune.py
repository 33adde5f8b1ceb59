"""The autotuners time only kernels whose shape they set: a lattice or batch
that advances as moments (tau = 1, no kernel asked for) has none."""
import pytest

from conftest import random_case

pytestmark = pytest.mark.gpu

SHAPE = (40, 18, 11)


@pytest.mark.parametrize("storage,kernel,tau,steps", [
    (2, "AUTO", 1.0, False), (2, "AUTO", 0.8, True), (2, "TWO_PASS", 1.0, True),
    (0, "AUTO", 1.0, False), (0, "AUTO", 0.8, False), (0, "TWO_PASS", 1.0, True)])
def test_lattice(storage, kernel, tau, steps):
    from multiphase_lbm_b200 import capi
    fluid, rho = random_case(SHAPE, seed=1, rho0=1.2, amp=0.3)
    lat = capi.Lattice(SHAPE, storage=storage)
    lat.set_step_kernel(getattr(capi, "KERNEL_" + kernel))
    lat.set_update_shape(2, 7)
    lat.set_params(capi.default_params(G=-5.0, rhos=0.2, tau=tau))
    lat.upload(fluid, rho)
    lat.initialize()
    rows, planes, done = lat.autotune(0, trial_steps=1)
    if steps:
        assert done == 40 and rows in (1, 2, 4, 8) and planes in (2, 4, 8, 16, 32)
    else:
        assert done == 0
        assert (rows, planes) == ((2, 7) if storage == 2 else (0, 0))
    lat.close()


@pytest.mark.parametrize("storage,tau,steps", [(2, 1.0, False), (2, 0.8, True),
                                               (0, 1.0, False), (1, 0.8, False)])
def test_batch(storage, tau, steps):
    from multiphase_lbm_b200 import batch, capi
    fluid, rho = random_case(SHAPE, seed=1, rho0=1.2, amp=0.3)
    b = batch.Batch(storage=storage)
    did = b.add(fluid, rho, capi.default_params(G=-5.0, rhos=0.2, tau=tau))
    b.set_tuning(2, 8, 3, 0, graphs=True)
    got = b.autotune(1)
    assert (b.domain_step(did) > 0) == steps
    if not steps:
        assert (got["rows_density"], got["rows_update"], got["planes"]) == (2, 8, 3)
    b.close()
