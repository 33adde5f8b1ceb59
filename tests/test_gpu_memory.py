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


def _batch(capi, storage, tau1=1.0):
    from multiphase_lbm_b200 import batch
    b = batch.Batch(storage=storage)
    ids, alone = [], []
    for i in range(2):
        fluid, rho = sphere_case(SHAPE, seed=9 + i, rmin=2.0, rmax=5.0, porosity=0.5,
                                 rho0=1.2, amp=0.4)
        p = capi.default_params(tau=tau1 if i else 1.0, **KW)
        ids.append(b.add(fluid, rho, p))
        lat = capi.Lattice(SHAPE, storage=storage)
        lat.set_step_kernel(capi.KERNEL_TWO_PASS)
        lat.set_params(p)
        lat.upload(fluid, rho)
        lat.initialize()
        alone.append(lat)
    return b, ids, alone


def _run(b, ids, alone, step, n):
    b.iterate(n)
    for did, lat in zip(ids, alone):
        lat.iterate(step, n)
        _same(b.lattice(did), lat, ("rho",))
    return step + n


@pytest.mark.parametrize("storage", [1, 2])
def test_a_batch_whose_moments_are_refused_keeps_none(storage):
    from multiphase_lbm_b200 import capi
    mom = _grown(capi, storage, 0)
    layout = _grown(capi, storage, capi.KERNEL_COMPACT) if storage == 1 else 0
    b, ids, alone = _batch(capi, storage)
    first, second = (b.lattice(i) for i in ids)
    held = first.test_memory_limit()
    # the second domain's packing differs by less than its moments' half
    second.test_memory_limit(second.test_memory_limit() + layout + (mom - layout) // 2)
    step = _run(b, ids, alone, 0, 5)
    step = _run(b, ids, alone, step, 9)
    assert first.test_memory_limit() == held + layout
    b.remove(ids.pop())
    alone.pop().close()
    _run(b, ids, alone, step, 3)  # alone again, it is held as moments
    assert first.test_memory_limit() == held + layout + mom
    b.close()


@pytest.mark.parametrize("storage", [0, 1])
def test_a_batch_that_leaves_tau_1_makes_room(storage):
    """The second domain is refused its populations' layout: the first one's
    moments go, and the call fails; it goes on once there is room."""
    from multiphase_lbm_b200 import capi
    layout = _grown(capi, storage, capi.KERNEL_COMPACT)
    b, ids, alone = _batch(capi, storage)
    first, second = (b.lattice(i) for i in ids)
    held = first.test_memory_limit()
    step = _run(b, ids, alone, 0, 4)
    for lat in (second, alone[1]):
        lat.set_params(capi.default_params(tau=0.8, **KW))
    second.test_memory_limit(held)
    with pytest.raises(capi.MlbmError, match="NOMEM"):
        b.iterate(3)
    assert first.test_memory_limit() == held + layout
    second.test_memory_limit()
    step = _run(b, ids, alone, step, 3)
    assert b.domain_step(ids[0]) == step
    b.close()


def test_a_domain_that_does_not_fit_takes_the_batchs_moments_first():
    import ctypes as C

    import numpy as np

    from multiphase_lbm_b200 import batch, capi
    b, ids, alone = _batch(capi, 2)
    first = b.lattice(ids[0])
    held = first.test_memory_limit()
    step = _run(b, ids, alone, 0, 4)
    grown = first.test_memory_limit()
    assert grown > held
    # 1280^3 FP64 nodes take 370 GB: refused before an array is read
    one = np.ones(1, np.float32)
    did = C.c_int32()
    p = capi.default_params(**KW)
    st = batch.blib().mlbm_batch_add(b.h, 1280, 1280, 1280, C.byref(p),
                                     one.ctypes.data, one.ctypes.data, 0, C.byref(did))
    assert st == 3  # MLBM_ERR_NOMEM
    assert first.test_memory_limit() == held
    _run(b, ids, alone, step, 4)
    assert first.test_memory_limit() == grown
    b.close()


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_a_small_transfer_needs_no_room_for_a_field(storage):
    """A restored lattice has no transfer buffer yet: the profile's few bytes
    per plane, and the fluid mask, fit where a field does not."""
    import numpy as np

    from multiphase_lbm_b200 import capi
    ref = _lattice(capi, storage)
    ref.iterate(0, 2)
    lat = capi.Lattice(SHAPE, storage=storage)
    lat.restore(ref.checkpoint(2))
    nodes = SHAPE[0] * SHAPE[1] * SHAPE[2]
    lat.test_memory_limit(lat.test_memory_limit() + 16 * SHAPE[0])
    for got, want in zip(lat.plane_profile(), ref.plane_profile()):
        assert np.array_equal(got, want)
    lat.test_memory_limit(lat.test_memory_limit() + nodes - 16 * SHAPE[0])
    assert np.array_equal(lat.field("fluid"), ref.field("fluid"))
    lat.close()
    ref.close()


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("shape,solid", [((40, 24, 17), 0.0), ((33, 20, 16), 0.4),
                                         ((5, 3, 1), 0.0)])
def test_stated_bytes_cover_what_is_held(shape, solid, storage):
    """A server that admits by mlbm_lattice_bytes: at most that is held by a
    domain that is uploaded, stepped at tau = 1 and read, and a batch says what
    its domains hold."""
    from conftest import random_case

    from multiphase_lbm_b200 import batch, capi
    fluid, rho = random_case(shape, seed=4, solid_frac=solid, rho0=1.2, amp=0.3)
    b = batch.Batch(storage=storage)
    ids = [b.add(fluid, rho, capi.default_params(G=-5.0)) for _ in range(2)]
    b.iterate(3)
    for did in ids:
        b.lattice(did).stats()
        b.lattice(did).field("rho", f64=storage == 2)
    held = [b.lattice(did).test_memory_limit() for did in ids]
    assert max(held) <= capi.lattice_bytes(shape, storage)
    if solid == 0.0 and shape[2] > 1:  # not by much above it, either
        assert max(held) >= 0.9 * (capi.lattice_bytes(shape, storage) - 70_000)
    assert b.nbytes() == sum(held)
    b.close()


@pytest.mark.parametrize("storage", [0, 2])
def test_buffers_given_back_and_taken_again_between_batch_calls(storage):
    """The only domain's moments make room for one that does not fit after all;
    its own steps then take new buffers, which the batch goes on with."""
    import ctypes as C

    import numpy as np

    from multiphase_lbm_b200 import batch, capi
    b, ids, alone = _batch(capi, storage)
    b.remove(ids.pop())
    alone.pop().close()
    step = _run(b, ids, alone, 0, 12)  # a graph of 8 steps is kept
    one = np.ones(1, np.float32)
    did = C.c_int32()
    p = capi.default_params(**KW)
    n = 1280 if storage == 2 else 1287  # 370 GB, 196 GB
    assert batch.blib().mlbm_batch_add(b.h, n - n % 32, n, n, C.byref(p), one.ctypes.data,
                                       one.ctypes.data, 0, C.byref(did)) == 3
    for lat in (b.lattice(ids[0]), alone[0]):
        lat.iterate(step, 3)
    step += 3
    _run(b, ids, alone, step, 12)
    b.close()
