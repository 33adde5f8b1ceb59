"""A lattice's set-up against work of other streams."""
import numpy as np
import pytest

from conftest import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_new_domains_while_the_default_stream_is_busy(storage):
    """A batch works on a stream of its own, which the default stream does not
    order itself with: what creating a domain clears there must be done before
    the domain's own set-up starts, however long the default stream is busy."""
    import torch

    from multiphase_lbm_b200 import batch, capi
    shape = (24, 20, 18)
    fluid, rho = random_case(shape, seed=3, rho0=1.2, amp=0.3)
    params = capi.default_params(G=-5.0, rhos=0.2, rho_shift=1.0)
    alone = capi.Lattice(shape, storage=storage)
    alone.set_step_kernel(capi.KERNEL_TWO_PASS)
    alone.set_params(params)
    alone.upload(fluid, rho)
    alone.initialize()
    alone.iterate(0, 6)
    want = alone.field("rho", f64=storage == 2)
    for _ in range(2):
        b = batch.Batch(storage=storage)
        torch.cuda._sleep(40_000_000)  # about 20 ms on the default stream
        did = b.add(fluid, rho, params)
        b.iterate(6)
        b.synchronize()
        torch.cuda.synchronize()
        assert np.array_equal(b.lattice(did).field("rho", f64=storage == 2), want)
        b.iterate(1)
        b.close()
