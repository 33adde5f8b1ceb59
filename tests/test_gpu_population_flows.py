"""The kernels that hold populations (tau other than 1) in the flows that a
program runs them in: lattices one after another over reused memory, random
runs with statistics and a save, steps captured into a CUDA graph, batches that
domains join, leave and resume in, slabs.  Against the dense two-pass kernels,
launched plainly, bit for bit."""
import numpy as np
import pytest

from conftest import sphere_case

pytestmark = pytest.mark.gpu

KW = dict(G=-5.0, rhos=0.223144, inlet_width=3, outlet_width=1, rho_inlet=0.17,
          rho_outlet=1.90, rho_shift=1.0)


def _lattice(capi, fluid, rho, kernel, storage, tau):
    lat = capi.Lattice(fluid.shape, storage=storage)
    lat.set_step_kernel(kernel)
    lat.set_params(capi.default_params(tau=tau, **KW))
    lat.upload(fluid, rho)
    lat.initialize()
    return lat


def _case(shape, seed):
    return sphere_case(shape, seed=seed, rmin=2.0, rmax=4.0, porosity=0.6, rho0=1.2,
                       amp=0.4)


@pytest.mark.parametrize("storage", [0, 1])
def test_lattices_over_reused_memory(storage):
    from multiphase_lbm_b200 import capi
    cases = [_case((40, 36, 28), 40 + i) for i in range(3)]
    want = []
    for fluid, rho in cases:
        ref = _lattice(capi, fluid, rho, capi.KERNEL_TWO_PASS, storage, 0.8)
        ref.iterate(0, 3)
        want.append(ref.field("f"))
        ref.close()
    for rep in range(8):
        lat = _lattice(capi, *cases[rep % 3], capi.KERNEL_AUTO, storage, 0.8)
        lat.iterate(0, 3)
        assert np.array_equal(lat.field("f"), want[rep % 3]), rep
        lat.close()


def test_random_runs_with_statistics_and_a_save():
    from multiphase_lbm_b200 import capi
    rng = np.random.default_rng(17)
    for cycle in range(24):
        shape = tuple(int(v) for v in rng.choice([16, 24, 32, 40], 3))
        storage, tau = int(rng.integers(0, 2)), float(rng.choice([0.8, 0.95, 1.2]))
        fluid, rho = _case(shape, int(rng.integers(1 << 20)))
        plan = [int(v) for v in rng.integers(1, 60, int(rng.integers(1, 4)))]
        save_at = int(rng.integers(0, len(plan)))
        finals = []
        for kernel in (capi.KERNEL_AUTO, capi.KERNEL_TWO_PASS):
            lat = _lattice(capi, fluid, rho, kernel, storage, tau)
            step = 0
            for i, n in enumerate(plan):
                lat.iterate(step, n)
                step += n
                lat.stats()
                if i == save_at:
                    image = lat.checkpoint(step)
                    lat.close()
                    lat = capi.Lattice(shape, storage=storage)
                    lat.set_step_kernel(kernel)
                    assert lat.restore(image) == step
            finals.append(lat.field("f").tobytes())
            lat.close()
        assert finals[0] == finals[1], (cycle, shape, storage, tau, plan)


@pytest.mark.parametrize("storage", [0, 1])
def test_captured_steps(storage):
    import torch

    from multiphase_lbm_b200 import capi
    fluid, rho = _case((40, 36, 28), 77)
    stream = torch.cuda.Stream()
    a = _lattice(capi, fluid, rho, capi.KERNEL_AUTO, storage, 0.8)
    torch.cuda.synchronize()  # set-up ran on the default stream
    a.set_stream(stream.cuda_stream)
    a.iterate(0, 2)
    a.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        a.iterate(2, 2)
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    b = _lattice(capi, fluid, rho, capi.KERNEL_TWO_PASS, storage, 0.8)
    b.iterate(0, 12)
    assert np.array_equal(a.field("f"), b.field("f"))
    del graph
    a.close()
    b.close()


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_batch_domains_join_leave_and_resume(storage):
    from multiphase_lbm_b200 import batch, capi
    shapes = [(32, 48, 16), (48, 32, 32), (64, 16, 48), (33, 17, 9)]
    taus = [0.8, 1.0, 1.2, 0.9]
    cases = [_case(s, 10 + i) for i, s in enumerate(shapes)]
    b = batch.Batch(storage=storage)
    at = [0] * 4

    def add(i):
        return b.add(*cases[i], capi.default_params(tau=taus[i], **KW))

    def run(n, ids):
        b.iterate(n)
        for i in ids:
            at[i] += n

    ids = {i: add(i) for i in (0, 1)}
    run(11, ids)                      # odd: the next domains join in phase 1
    ids.update({i: add(i) for i in (2, 3)})
    run(13, ids)
    image = b.lattice(ids[0]).checkpoint(at[0])
    b.remove(ids.pop(0))
    run(10, ids)
    ids[0] = b.add_checkpoint(image)
    run(9, ids)
    for i, did in ids.items():
        lat = _lattice(capi, *cases[i], capi.KERNEL_TWO_PASS, storage, taus[i])
        lat.iterate(0, at[i])
        for field in ("rho", "f"):
            got = b.lattice(did).field(field, f64=storage == 2)
            assert got.tobytes() == lat.field(field, f64=storage == 2).tobytes(), i
        assert b.domain_step(did) == at[i]
        lat.close()
    b.close()


@pytest.mark.parametrize("storage,parts,transport", [(0, 2, "ring"), (0, 3, "local"),
                                                     (1, 3, "ring"), (1, 1, "ring")])
def test_slabs(storage, parts, transport):
    import torch

    from multiphase_lbm_b200 import capi, slab
    fluid, rho = _case((40, 36, 32), 5)
    m = fluid.astype(bool)
    whole = _lattice(capi, fluid, rho, capi.KERNEL_TWO_PASS, storage, 0.8)
    run = slab.decompose(fluid, rho, capi.default_params(tau=0.8, **KW), parts, storage,
                         transport=transport)
    whole.iterate(0, 7, write_velocity=True)
    run.run(0, 6)
    run.step(6, write_velocity=True)
    torch.cuda.synchronize()
    for which in ("f", "rho", "velocity"):
        assert np.array_equal(whole.field(which)[m], slab.gather(run.slabs, which)[m])
    run.close()
    whole.close()
