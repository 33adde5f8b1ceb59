"""Which step kernels run: a kernel that the caller asks for is the one that
advances the lattice, at tau = 1 too; AUTO takes the moment step there.

The launches are read from torch's profiler, which may leave later launches of
the process slower: this file is named to be collected after the others."""
import pytest

from conftest import random_case

pytestmark = pytest.mark.gpu


def _launched(run, copies=False):
    """Names of the library's kernels that `run` launches, with repeats (and
    of everything else on the device, with `copies`)."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    if not names:
        pytest.skip("the profiler records no launches here")
    return names if copies else [n for n in names if "mlbm" in n]


@pytest.mark.parametrize("storage,kernel,tau,want", [
    (0, "AUTO", 1.0, "k_mom_collide"), (1, "AUTO", 1.0, "k_mom_collide"),
    (2, "AUTO", 1.0, "k_mom_collide"), (0, "AUTO", 0.8, "k_cupdate"),
    (2, "AUTO", 0.8, "k_update_zm"), (0, "COMPACT", 1.0, "k_cupdate"),
    (1, "COMPACT", 1.0, "k_cupdate"), (0, "TWO_PASS", 1.0, "k_update_zm"),
    (2, "TWO_PASS", 1.0, "k_update_zm"), (0, "BAND", 1.0, "k_band")])
def test_the_kernel_asked_for_runs(storage, kernel, tau, want):
    from multiphase_lbm_b200 import capi
    shape = (40, 18, 11)
    fluid, rho = random_case(shape, seed=1, rho0=1.2, amp=0.3)
    lat = capi.Lattice(shape, storage=storage)
    lat.set_step_kernel(getattr(capi, "KERNEL_" + kernel))
    lat.set_params(capi.default_params(G=-5.0, rhos=0.2, tau=tau))
    lat.upload(fluid, rho)
    lat.initialize()
    lat.iterate(0, 1)
    names = _launched(lambda: lat.iterate(1, 3))
    updates = [n for n in names for k in ("k_mom_collide", "k_cupdate", "k_update_zm",
                                          "k_band") if k in n]
    assert len(updates) == 3 and all(want in n for n in updates), names
    lat.close()


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_only_a_joining_domain_steps_by_itself(storage):
    """A batch held as moments takes in a domain: one step of that domain by its
    own launches, beside the batched launches of the others."""
    from multiphase_lbm_b200 import batch, capi
    b = batch.Batch(storage=storage)

    def add(i):
        fluid, rho = random_case((20 + i, 9, 6), seed=i, rho0=1.2, amp=0.3)
        return b.add(fluid, rho, capi.default_params(G=-5.0, rhos=0.2))

    for i in range(5):
        add(i)
    b.iterate(2)
    add(5)
    names = _launched(lambda: b.iterate(3))
    alone = [n for n in names if "k_mom_collide" in n]
    batched = [n for n in names if "k_batch_mom_collide" in n]
    assert len(alone) == 1 and len(batched) == 3, names
    b.close()


@pytest.mark.parametrize("tau", [1.0, 0.8])
def test_the_same_parameters_again_change_nothing(tau):
    """A program that sets a domain's parameters before every call keeps the
    batch's tables and graph: no table goes to the device again."""
    from multiphase_lbm_b200 import batch, capi
    b = batch.Batch(storage=0)
    fluid, rho = random_case((20, 9, 6), seed=1, rho0=1.2, amp=0.3)
    p = capi.default_params(G=-5.0, rhos=0.2, tau=tau)
    did = b.add(fluid, rho, p)
    b.iterate(12)

    def again(q):
        b.lattice(did).set_params(q)
        b.iterate(12)

    assert not [n for n in _launched(lambda: again(p), True) if "HtoD" in n]
    if tau == 1.0:  # nor after steps of its own, which leave it held as moments
        b.lattice(did).iterate(24, 3)
        assert not [n for n in _launched(lambda: again(p), True) if "HtoD" in n]
    q = capi.default_params(G=-4.9, rhos=0.2, tau=tau)
    assert [n for n in _launched(lambda: again(q), True) if "HtoD" in n]
    b.close()
