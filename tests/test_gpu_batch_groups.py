"""Batches of domains held as moments at the numbers of domains where their
launches change: one launch of up to 16 or of up to 128 domains, and several.
Every domain has the bits of the same domain advanced alone; a domain without
fluid takes part."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,count", [(0, 1), (0, 16), (1, 17), (0, 128),
                                           (1, 129), (2, 130)])
def test_domains_match_alone(storage, count):
    from multiphase_lbm_b200 import batch, capi
    rng = np.random.default_rng(count)
    b = batch.Batch(storage=storage)
    want = {}
    for i in range(count):
        shape = (6 + i % 5, 5 + i % 3, 4 + i % 4)
        fluid = (rng.random(shape) < 0.7).astype(np.uint8)
        if i == count // 2 and count > 1:
            fluid[:] = 0
        rho = (1.5 + 0.2 * rng.random(shape)).astype(np.float32)
        p = dict(G=-5.0 - 0.01 * i, tau=1.0, rhos=0.2, rho_inject_period=1 + i % 5)
        did = b.add(fluid, rho, capi.default_params(**p))
        if i in (0, 15, 16, 127, 128, count - 1):
            want[did] = (shape, fluid, rho, p)
    b.iterate(1)
    b.iterate(12)  # steps by graph replays and by themselves
    for did, (shape, fluid, rho, p) in want.items():
        lat = capi.Lattice(shape, storage=storage)
        lat.set_params(capi.default_params(**p))
        lat.upload(fluid, rho)
        lat.initialize()
        lat.iterate(0, 13)
        for name in ("rho", "f"):
            assert np.array_equal(b.lattice(did).field(name), lat.field(name)), (did, name)
        lat.close()
    b.close()
