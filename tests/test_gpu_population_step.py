"""The step that holds populations (tau other than 1) over the fluid-only
layout: one node per thread in the gather/push phase, pairs in the local one,
alone and batched, against the dense two-pass kernels bit for bit."""
import numpy as np
import pytest

from conftest import sphere_case

pytestmark = pytest.mark.gpu


def _case(shape, storage):
    fluid, rho = sphere_case(shape, seed=sum(shape) + storage, rmin=1.5, rmax=3.5,
                             porosity=0.6, rho0=1.5, amp=0.3)
    kw = dict(G=-5.0, rhos=0.223144, tau=0.8, rho_shift=1.0)
    if shape[0] >= 8:
        kw.update(inlet_width=2, outlet_width=1, rho_inlet=0.17, rho_outlet=1.9,
                  rho_inject_period=4)
    return fluid, rho, kw


def _fields(lat):
    return [lat.field(n) for n in ("rho", "f", "psi")]


# planes with odd fluid counts (a hole after each), fewer nodes than a block,
# blocks that end within a warp, rows over several mask words, one-node edges
@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("shape", [(5, 3, 2), (11, 7, 9), (33, 5, 7), (70, 3, 2),
                                   (300, 6, 6), (1, 9, 8), (40, 32, 25)])
def test_matches_dense_kernels(shape, storage):
    from multiphase_lbm_b200 import batch, capi
    fluid, rho, kw = _case(shape, storage)
    outs = []
    for kind in (capi.KERNEL_COMPACT, capi.KERNEL_TWO_PASS):
        lat = capi.Lattice(shape, storage=storage)
        lat.set_step_kernel(kind)
        lat.set_params(capi.default_params(**kw))
        lat.upload(fluid, rho)
        lat.initialize()
        got = []
        for first, n in ((0, 1), (1, 1), (2, 7)):  # ends in either phase
            lat.iterate(first, n)
            got += _fields(lat)
        lat.iterate(9, 1, write_velocity=True)
        got += _fields(lat)
        outs.append(got + [lat.field("velocity")])
        lat.close()
    for u, v in zip(*outs):
        assert np.array_equal(u, v)
    # batched beside a domain of another size, one step further on
    b = batch.Batch(storage=storage)
    f2, r2, k2 = _case((24, 9, 5), storage)
    b.add(f2, r2, capi.default_params(**k2))
    b.iterate(1)
    did = b.add(fluid, rho, capi.default_params(**kw))
    b.iterate(9)
    b.iterate(1)
    for u, v in zip(_fields(b.lattice(did)), outs[1][-4:-1]):
        assert np.array_equal(u, v)
    b.close()
