"""Device memory of the moment step: it is taken where there is room, and given
back where another buffer of the lattice needs it.  The limits are a lattice's
own (mlbm_test_memory_limit), so that no test fills the device."""
import pytest

from conftest import sphere_case

pytestmark = pytest.mark.gpu

SHAPE = (64, 40, 33)
KW = dict(G=-5.0, rhos=0.2, rho_shift=1.0, inlet_width=2, outlet_width=1,
          rho_inlet=0.17, rho_outlet=1.9)


def _lattice(capi, storage, kernel=0, tau=1.0):
    fluid, rho = sphere_case(SHAPE, seed=9, rmin=2.0, rmax=5.0, porosity=0.5,
                             rho0=1.2, amp=0.4)
    lat = capi.Lattice(SHAPE, storage=storage)
    lat.set_step_kernel(kernel)
    lat.set_params(capi.default_params(tau=tau, **KW))
    lat.upload(fluid, rho)
    lat.initialize()
    return lat


def _grown(capi, storage, kernel, tau=1.0):
    """Device bytes that a first step adds."""
    lat = _lattice(capi, storage, kernel, tau)
    before = lat.test_memory_limit()
    lat.iterate(0, 1)
    grown = lat.test_memory_limit() - before
    lat.close()
    return grown


def _same(a, b, fields=("rho", "f")):
    for field in fields:
        assert a.field(field).tobytes() == b.field(field).tobytes(), field


@pytest.mark.parametrize("storage", [0, 1])
def test_tau_leaves_1_where_only_one_form_fits(storage):
    from multiphase_lbm_b200 import capi
    mom, compact = _grown(capi, storage, 0), _grown(capi, storage, capi.KERNEL_COMPACT)
    assert mom > 0 and compact > 0
    a, b = _lattice(capi, storage), _lattice(capi, storage, capi.KERNEL_TWO_PASS)
    # room for the larger form, and for the tables beside it
    a.test_memory_limit(a.test_memory_limit() + max(mom, compact))
    step = 0
    for tau in (1.0, 0.8, 1.0):
        for lat in (a, b):
            lat.set_params(capi.default_params(tau=tau, **KW))
            lat.iterate(step, 5)
        step += 5
    a.test_memory_limit()
    _same(a, b)
    a.close()
    b.close()


@pytest.mark.parametrize("storage", [0, 2])
def test_velocity_where_it_fits_only_without_the_moments(storage):
    from multiphase_lbm_b200 import capi
    mom = _grown(capi, storage, 0)
    a, b = _lattice(capi, storage), _lattice(capi, storage, capi.KERNEL_TWO_PASS)
    vel = SHAPE[0] * SHAPE[1] * SHAPE[2] * 12  # nx is a multiple of 32
    other = _grown(capi, storage, capi.KERNEL_COMPACT) if storage != 2 else 0
    held = a.test_memory_limit()
    a.iterate(0, 4)
    b.iterate(0, 4)
    a.test_memory_limit(held + max(mom, vel + other))
    a.iterate(4, 3, write_velocity=True)
    b.iterate(4, 3, write_velocity=True)
    a.test_memory_limit()
    _same(a, b, ("rho", "f", "velocity"))
    a.close()
    b.close()


@pytest.mark.parametrize("storage", [0, 2])
def test_a_download_where_it_fits_only_without_the_moments(storage):
    from multiphase_lbm_b200 import capi
    mom = _grown(capi, storage, 0)
    a, b = _lattice(capi, storage), _lattice(capi, storage, capi.KERNEL_TWO_PASS)
    a.iterate(0, 4)
    b.iterate(0, 4)
    held = a.test_memory_limit()
    nodes = SHAPE[0] * SHAPE[1] * SHAPE[2]
    a.test_memory_limit(held + 19 * 4 * nodes - mom // 2)
    _same(a, b, ("f",))
    a.test_memory_limit()
    a.iterate(4, 4)  # from populations
    b.iterate(4, 4)
    _same(a, b)
    a.close()
    b.close()


@pytest.mark.parametrize("storage", [1, 2])
def test_refused_moments_leave_the_population_kernels(storage):
    """FP16: the fluid-only layout is the smaller one; FP64 needs nothing."""
    from multiphase_lbm_b200 import capi
    mom = _grown(capi, storage, 0)
    a, b = _lattice(capi, storage), _lattice(capi, storage, capi.KERNEL_TWO_PASS)
    held = a.test_memory_limit()
    a.test_memory_limit(held + mom - 1)
    for lat in (a, b):
        lat.iterate(0, 5)
        lat.iterate(5, 4)
    a.test_memory_limit()
    _same(a, b)
    a.close()
    b.close()
