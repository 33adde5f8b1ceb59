"""Tables that a lattice builds on first use, against its own stream: a
non-blocking stream is not ordered with the default stream, so what its
kernels read has to come in on it, whatever the default stream does meanwhile."""
import numpy as np
import pytest

from conftest import sphere_case

pytestmark = pytest.mark.gpu

BUSY = 600_000_000  # cycles: some 0.3 s of the default stream


def _lattice(capi, shape, fluid, rho, storage, kernel, **kw):
    lat = capi.Lattice(shape, storage=storage)
    lat.set_step_kernel(kernel)
    lat.set_params(capi.default_params(G=-5.0, rhos=0.2, rho_shift=1.0, **kw))
    lat.upload(fluid, rho)
    lat.initialize()
    return lat


@pytest.mark.parametrize("storage", [0, 1])
def test_fluid_only_tables_come_in_on_the_lattices_stream(storage):
    import torch

    from multiphase_lbm_b200 import capi
    shape = (70, 36, 28)
    fluid, rho = sphere_case(shape, seed=3, rmin=2.0, rmax=4.0, porosity=0.6,
                             rho0=1.2, amp=0.4)
    want = _lattice(capi, shape, fluid, rho, storage, capi.KERNEL_TWO_PASS, tau=0.8)
    want.iterate(0, 6)
    stream = torch.cuda.Stream()  # non-blocking
    for rep in range(2):  # the first one loads the kernels
        lat = _lattice(capi, shape, fluid, rho, storage, capi.KERNEL_COMPACT, tau=0.8)
        torch.cuda.synchronize()  # set-up ran on the default stream
        lat.set_stream(stream.cuda_stream)
        busy = torch.cuda.Event()
        if rep:
            torch.cuda._sleep(BUSY)
        busy.record()
        lat.iterate(0, 6)
        if rep:  # built and launched without the default stream
            assert not busy.query()
        torch.cuda.synchronize()
        assert np.array_equal(lat.field("f"), want.field("f"))
        lat.close()
    want.close()


def test_ring_jobs_come_in_on_the_slabs_stream():
    import torch

    from multiphase_lbm_b200 import capi, slab
    shape = (40, 24, 20)
    fluid, rho = sphere_case(shape, seed=5, rmin=2.0, rmax=4.0, porosity=0.6,
                             rho0=1.2, amp=0.4)
    want = _lattice(capi, shape, fluid, rho, 0, capi.KERNEL_TWO_PASS, tau=0.8)
    want.iterate(0, 7)
    m = fluid.astype(bool)
    params = capi.default_params(G=-5.0, rhos=0.2, rho_shift=1.0, tau=0.8)
    stream = torch.cuda.Stream()
    for rep in range(2):  # the first one loads the kernels
        with torch.cuda.stream(stream):
            slabs = [slab.Slab(fluid, rho, params, 10 * i, 10) for i in range(2)]
        torch.cuda.synchronize()
        busy = torch.cuda.Event()
        if rep:
            torch.cuda._sleep(BUSY)
        busy.record()
        run = slab.SlabRun(slabs, slab.RingExchange(slabs))
        run.run(0, 7)
        if rep:
            assert not busy.query()
        torch.cuda.synchronize()
        assert np.array_equal(slab.gather(slabs, "f")[m], want.field("f")[m])
        run.close()
    want.close()


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("tau", [1.0, 0.8])
def test_a_step_after_a_new_initial_state_can_be_captured(storage, tau):
    """The buffers and tables of the first run serve the next: nothing is
    allocated or waited for, which a capture would refuse."""
    import torch

    from multiphase_lbm_b200 import capi
    shape = (40, 24, 17)
    fluid, rho = sphere_case(shape, seed=8, rmin=2.0, rmax=4.0, porosity=0.6,
                             rho0=1.2, amp=0.4)
    want = _lattice(capi, shape, fluid, rho, storage, capi.KERNEL_TWO_PASS, tau=tau,
                    inlet_width=2, rho_inlet=0.3)
    want.iterate(0, 5)
    stream = torch.cuda.Stream()
    lat = _lattice(capi, shape, fluid, rho, storage, capi.KERNEL_AUTO, tau=tau,
                   inlet_width=2, rho_inlet=0.3)
    torch.cuda.synchronize()
    lat.set_stream(stream.cuda_stream)
    lat.iterate(0, 3)
    lat.initialize()
    lat.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        lat.iterate(0, 4)
    graph.replay()
    torch.cuda.synchronize()
    lat.iterate(4, 1)
    torch.cuda.synchronize()
    assert lat.field("f", f64=storage == 2).tobytes() == \
        want.field("f", f64=storage == 2).tobytes()
    del graph
    # slabs of another width: the lists follow them
    for l in (lat, want):
        l.set_params(capi.default_params(G=-5.0, rhos=0.2, rho_shift=1.0, tau=tau,
                                         inlet_width=5, rho_inlet=0.3))
        l.initialize()
        l.iterate(0, 5)
    torch.cuda.synchronize()
    assert lat.field("f").tobytes() == want.field("f").tobytes()
    lat.close()
    want.close()


def test_creating_a_lattice_does_not_wait_for_the_default_stream():
    import torch

    from multiphase_lbm_b200 import capi
    capi.Lattice((40, 24, 17)).close()  # the first one loads the library
    torch.cuda.synchronize()
    busy = torch.cuda.Event()
    torch.cuda._sleep(BUSY)
    busy.record()
    lat = capi.Lattice((40, 24, 17))
    assert not busy.query()
    torch.cuda.synchronize()
    lat.close()
