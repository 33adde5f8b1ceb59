"""New fluid masks in a lattice that has stepped: its fluid-only buffers are
kept where the new fluid nodes fit them."""
import numpy as np
import pytest

from conftest import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("tau", [1.0, 0.8])
def test_one_pass_step_after_masks_of_other_sizes(storage, tau):
    """Many fluid nodes, then few -- where the one-pass step first takes its
    second buffer -- then many again, more than at that moment."""
    from multiphase_lbm_b200 import capi
    shape = (40, 24, 18)
    params = capi.default_params(G=-5.0, rhos=0.2, tau=tau, rho_shift=1.0)
    lat, ref = (capi.Lattice(shape, storage=storage) for _ in range(2))
    ref.set_step_kernel(capi.KERNEL_TWO_PASS)
    for l in (lat, ref):
        l.set_params(params)
    for kernel, solid in ((capi.KERNEL_COMPACT, 0.05), (capi.KERNEL_BAND, 0.9),
                          (capi.KERNEL_BAND, 0.2), (capi.KERNEL_BAND, 0.02)):
        fluid, rho = random_case(shape, seed=7, solid_frac=solid, rho0=1.2, amp=0.3)
        lat.set_step_kernel(kernel)
        for l in (lat, ref):
            l.upload(fluid, rho)
            l.initialize()
            l.iterate(0, 6)  # one two-pass step, then five that swap the buffers
        assert np.array_equal(lat.field("f"), ref.field("f")), (kernel, solid)
    lat.close()
    ref.close()


@pytest.mark.parametrize("storage", [0, 2])
@pytest.mark.parametrize("kernel", ["AUTO", "TWO_PASS"])
@pytest.mark.parametrize("restore", [False, True])
def test_nodes_that_became_solid_have_no_velocity(storage, kernel, restore):
    from multiphase_lbm_b200 import capi
    shape = (40, 24, 18)
    lat, other = (capi.Lattice(shape, storage=storage) for _ in range(2))
    for l, solid in ((lat, 0.02), (other, 0.4)):
        fluid, rho = random_case(shape, seed=1, solid_frac=solid, rho0=1.2, amp=0.3)
        l.set_step_kernel(getattr(capi, "KERNEL_" + kernel))
        l.set_params(capi.default_params(G=-5.0, rhos=0.2))
        l.upload(fluid, rho)
        l.initialize()
        l.iterate(0, 3, write_velocity=True)
    if restore:
        lat.restore(other.checkpoint(3))
    else:
        lat.upload(fluid, rho)
        lat.initialize()
        lat.iterate(0, 3)
    for l in (lat, other):
        l.iterate(3, 1, write_velocity=True)
    assert np.array_equal(lat.field("velocity"), other.field("velocity"))
    assert not other.field("velocity")[fluid == 0].any()
    lat.close()
    other.close()
