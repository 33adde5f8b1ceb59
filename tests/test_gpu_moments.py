"""The moment step (tau = 1: the state of a step is rho and u of every node)
against the dense two-pass kernels, which hold populations: the same bits.

Both form f* = feq(rho, u) with the same operations in the same order, so
every comparison is exact.
"""
import numpy as np
import pytest

from conftest import random_case, sphere_case

pytestmark = pytest.mark.gpu

DRAIN = dict(G=-5.0, rhos=0.223144, tau=1.0, inlet_width=2, outlet_width=1,
             rho_inlet=0.17, rho_outlet=1.90, rho_shift=1.0)


def _lattice(capi, shape, fluid, rho, kernel, storage, **kw):
    lat = capi.Lattice(shape, storage=storage)
    lat.set_step_kernel(kernel)
    lat.set_params(capi.default_params(**kw))
    lat.upload(fluid, rho)
    lat.initialize()
    return lat


def _same(a, b, f64):
    for field in ("rho", "f", "velocity"):
        assert np.array_equal(a.field(field, f64=f64), b.field(field, f64=f64)), field


# one plane, odd and even z (the last plane alone in its pair, next to a
# periodic image), single rows and columns, edges of the 32 x 8 x 4 tiles
SHAPES = [(33, 9, 1), (16, 8, 2), (31, 7, 3), (32, 8, 4), (33, 9, 5), (65, 17, 9),
          (1, 6, 7), (2, 2, 2), (9, 1, 6), (3, 40, 33)]


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_moment_step_bit_identical(shape, storage):
    from multiphase_lbm_b200 import capi
    fluid, rho = random_case(shape, seed=sum(shape), rho0=1.2, amp=0.4)
    kw = dict(DRAIN) if shape[0] >= 8 else dict(DRAIN, inlet_width=0, outlet_width=0)
    a = _lattice(capi, shape, fluid, rho, capi.KERNEL_AUTO, storage, **kw)
    b = _lattice(capi, shape, fluid, rho, capi.KERNEL_TWO_PASS, storage, **kw)
    step = 0
    for n in (1, 1, 4, 7):
        for lat in (a, b):
            lat.iterate(step, n, write_velocity=True)
        step += n
        _same(a, b, storage == 2)
    assert a.stats()["n_fluid"] == int(fluid.sum())


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_moment_step_changes_of_form(storage):
    """tau away from 1 and back, another kernel in between, a save and
    restore, slabs moved by a new initial state, injection, all-solid."""
    from multiphase_lbm_b200 import capi
    shape = (40, 19, 13)
    fluid, rho = sphere_case(shape, seed=5, rmin=2.0, rmax=4.0, porosity=0.6,
                             rho0=1.2, amp=0.4)
    kw = dict(DRAIN, rho_increment=0.01, rho_inject_period=3, inject_position=0.5,
              inject_density=1)
    a = _lattice(capi, shape, fluid, rho, capi.KERNEL_AUTO, storage, **kw)
    b = _lattice(capi, shape, fluid, rho, capi.KERNEL_TWO_PASS, storage, **kw)
    step = 0

    def both(n, **opt):
        nonlocal step
        for lat in (a, b):
            lat.iterate(step, n, write_velocity=True, **opt)
        step += n
        _same(a, b, storage == 2)

    both(5, inject_type=1)
    for tau in (0.8, 1.0):
        for lat in (a, b):
            lat.set_params(capi.default_params(**dict(kw, tau=tau)))
        both(3)
    a.set_step_kernel(capi.KERNEL_TWO_PASS)
    both(2, reverse=-1)
    a.set_step_kernel(capi.KERNEL_AUTO)
    both(4, inject_type=2)
    image = a.checkpoint(step)
    a.close()
    a = capi.Lattice(shape, storage=storage)
    assert a.restore(image) == step
    both(3)
    for lat in (a, b):
        lat.set_params(capi.default_params(**dict(kw, inlet_width=5, rho_inlet=0.3)))
        lat.upload(fluid, rho)
        lat.initialize()
    both(6)
    for lat in (a, b):
        lat.upload(np.zeros_like(fluid), rho)
        lat.initialize()
    both(2)


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_batched_moments_bit_identical(storage):
    """Domains of a batch, one added later, one removed, one advanced on its
    own in between (an even number of steps), one whose tau leaves 1 (the
    whole batch then holds populations), against the domains alone."""
    from multiphase_lbm_b200 import batch, capi
    shapes = [(33, 9, 5), (16, 24, 8), (40, 17, 13)]
    b = batch.Batch(storage=storage)
    cases, ids, alone, at = [], [], [], []
    for i, shape in enumerate(shapes):
        fluid, rho = random_case(shape, seed=i, rho0=1.2, amp=0.4)
        cases.append((shape, fluid, rho, dict(DRAIN, rho_inlet=0.2 + 0.1 * i)))
        alone.append(_lattice(capi, shape, fluid, rho, capi.KERNEL_TWO_PASS, storage,
                              **cases[-1][3]))
        at.append(0)

    def run(n):
        b.iterate(n)
        for i in range(len(ids)):
            if ids[i] is not None:
                alone[i].iterate(at[i], n)
                at[i] += n
                for field in ("rho", "f"):
                    got = b.lattice(ids[i]).field(field, f64=storage == 2)
                    assert np.array_equal(got, alone[i].field(field, f64=storage == 2))

    for i in range(2):
        ids.append(b.add(cases[i][1], cases[i][2], capi.default_params(**cases[i][3])))
    run(1)
    run(13)  # a graph replay and single steps
    ids.append(b.add(cases[2][1], cases[2][2], capi.default_params(**cases[2][3])))
    run(10)
    b.lattice(ids[0]).iterate(at[0], 2)
    alone[0].iterate(at[0], 2)
    at[0] += 2
    run(9)
    b.remove(ids[1])
    ids[1] = None
    run(3)
    for lat in (b.lattice(ids[2]), alone[2]):
        lat.set_params(capi.default_params(**dict(cases[2][3], tau=0.9)))
    run(4)
    b.close()
