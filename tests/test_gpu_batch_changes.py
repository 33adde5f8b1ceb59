"""Domains of a batch that change between its iterate calls: advanced on
their own by any step kernel, given other parameters.  Every domain has the
bits of the same domain advanced alone by the dense two-pass kernels."""
import pytest

from conftest import random_case

pytestmark = pytest.mark.gpu

DRAIN = dict(G=-5.0, rhos=0.223144, inlet_width=2, outlet_width=1, rho_inlet=0.17,
             rho_outlet=1.90, rho_shift=1.0)
SHAPES = [(33, 9, 5), (16, 24, 8)]


class Pair:
    """A batch and the same domains alone."""

    def __init__(self, storage, taus):
        from multiphase_lbm_b200 import batch, capi
        self.capi, self.storage = capi, storage
        self.b = batch.Batch(storage=storage)
        self.kw, self.ids, self.alone, self.at = [], [], [], []
        for i, (shape, tau) in enumerate(zip(SHAPES, taus)):
            fluid, rho = random_case(shape, seed=i, rho0=1.2, amp=0.4)
            kw = dict(DRAIN, tau=tau)
            self.kw.append(kw)
            self.ids.append(self.b.add(fluid, rho, capi.default_params(**kw)))
            lat = capi.Lattice(shape, storage=storage)
            lat.set_step_kernel(capi.KERNEL_TWO_PASS)
            lat.set_params(capi.default_params(**kw))
            lat.upload(fluid, rho)
            lat.initialize()
            self.alone.append(lat)
            self.at.append(0)

    def lattice(self, i):
        return self.b.lattice(self.ids[i])

    def set(self, i, **kw):
        self.kw[i] = dict(self.kw[i], **kw)
        for lat in (self.lattice(i), self.alone[i]):
            lat.set_params(self.capi.default_params(**self.kw[i]))

    def own(self, i, n):
        """Advance domain i on its own."""
        for lat in (self.lattice(i), self.alone[i]):
            lat.iterate(self.at[i], n)
        self.at[i] += n

    def run(self, n):
        self.b.iterate(n)
        for i, lat in enumerate(self.alone):
            lat.iterate(self.at[i], n)
            self.at[i] += n
            for field in ("rho", "f"):
                got = self.lattice(i).field(field, f64=self.storage == 2)
                want = lat.field(field, f64=self.storage == 2)
                # bits: a change of rho_shift in FP16 storage moves every
                # density, and may drive a domain to infinities and NaN
                assert got.tobytes() == want.tobytes(), (i, field)

    def close(self):
        self.b.close()
        for lat in self.alone:
            lat.close()


# AUTO, TWO_PASS, COMPACT, BAND; FP64 has the first two
@pytest.mark.parametrize("storage,kernel", [(s, k) for s in (0, 1) for k in (0, 2, 3, 6)]
                         + [(2, 0), (2, 2)])
@pytest.mark.parametrize("taus", [(1.0, 1.0), (1.0, 0.8), (0.8, 0.8)])
def test_an_odd_number_of_steps_alone(storage, kernel, taus):
    """An odd number of own steps leaves the domain in the other AA phase,
    and a kernel of its own may leave it in another layout or buffer."""
    t = Pair(storage, taus)
    t.run(2)
    t.lattice(0).set_step_kernel(kernel)
    t.own(0, 3)
    t.run(10)  # a graph replay and single steps
    t.own(0, 1)
    t.run(1)
    if taus[1] == 1.0:  # tau leaves 1: the whole batch holds populations
        t.set(1, tau=0.9)
        t.run(3)
        t.own(0, 1)
        t.set(1, tau=1.0)
    t.run(2)
    t.close()


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("taus", [(1.0, 1.0), (1.0, 0.8)])
def test_changed_parameters(storage, taus):
    """What mlbm_set_params on a domain's lattice changes holds from the next
    batch step on, as it does for a lattice alone."""
    t = Pair(storage, taus)
    t.run(10)
    t.set(0, G=-4.5)
    t.run(10)
    t.set(1, rho_inlet=0.3)
    t.set(0, rho_outlet=1.7)
    t.run(3)
    t.set(0, rho_increment=0.01, rho_inject_period=2, inject_position=0.6)
    t.run(11)
    t.set(1, rho_shift=0.5)
    t.run(2)
    if taus[1] != 1.0:
        t.set(1, tau=1.1)
        t.run(9)
    t.close()
