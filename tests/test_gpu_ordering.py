"""Entries that return before their work has run, followed at once by one that
sets host or device state of its own: the results are those of the same calls
with a wait between them, bit for bit."""
import numpy as np
import pytest

from amdkiit_b200 import configs
from amdkiit_b200.engine import FP64, MIXED, Engine, Ensemble
from amdkiit_b200.inputs import XC_PBE
from amdkiit_b200.slab import LocalExchange, Slab, apply_local_h, density, gram
from tests.helpers import start_coefficients

pytestmark = pytest.mark.gpu


def _engine(system, prec):
    e = Engine(system, prec)
    g = e.gvectors()
    e.set_wfn(start_coefficients(g["hg"][: e.ngpw], 2 * np.pi / system.alat, e.nstate))
    e.ortho()
    return e


def _stages(e):
    """One CG iteration up to the gradient by its single entries."""
    e.density()
    e.potential()
    e.energy()
    e.apply_h()
    e.gradient()


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_cg_step_followed_by_an_iteration(prec):
    """amdk_pcg(a) and amdk_scf_iteration(b) straight after it: each update
    takes its own step number (a = 1 restarts the direction, b = 12 carries it
    on with another factor), eager and replayed from graphs."""
    s = configs.small_water(xc=XC_PBE)
    got = []
    for wait in (True, False):
        e = _engine(s, prec)
        for it in (1, 2):
            e.scf_iteration(it, 1e-7)
        for a, b in ((1, 12), (12, 1), (1, 25)):
            _stages(e)
            e.pcg(a)
            if wait:
                e.get_wfn()
            e.scf_iteration(b, 1e-7)
        _stages(e)
        e.pcg(1)
        if wait:
            e.get_wfn()
        e.pcg(12)  # the direction of the first carried on
        got.append(e.get_wfn())
        e.close()
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_ensemble_after_work_on_the_members_streams(prec):
    """An ensemble iteration (its own stream) starts after what its members'
    entries have queued: the CG update and the rotation of an ortho."""
    systems = [configs.cluster(n, L, 500 + n, ecut=30.0) for n, L in ((3, 13.5), (2, 14.0))]
    got = []
    for wait in (True, False):
        members = [_engine(s, prec) for s in systems]
        ens = Ensemble(members)
        for it in (1, 2, 3):
            ens.iteration([it] * 2, 1e-7)
        for it in (4, 5):
            for e in members:
                _stages(e)
                e.pcg(it)
                e.ortho()
                if wait:
                    e.get_wfn()
            ens.iteration([it] * 2, 1e-7)
        got.append([e.get_wfn() for e in members])
        ens.close()
        for e in members:
            e.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_slab_calls_follow_the_default_stream(prec):
    """The slab entries called without a stream run on the context's own, which
    does not wait for the default stream by itself: inputs written there, and
    the exchange's copies there, are complete before a kernel reads them, also
    when the default stream is 10 ms behind."""
    import torch

    class Exchange(LocalExchange):
        def __init__(self, late):
            self.late = late

        def __call__(self, sends, send_counts, recv_counts):
            if self.late:
                torch.cuda._sleep(20_000_000)
            return super().__call__(sends, send_counts, recv_counts)

    s = configs.small_water()
    e = _engine(s, prec)
    slabs = [Slab(e, 2, r) for r in range(2)]
    c0 = e.get_wfn()
    start = [torch.from_numpy(np.ascontiguousarray(c0[:, x.local_g])).cuda() for x in slabs]
    vs = [torch.randn(x.grid, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(x.rank))
          for x in slabs]
    torch.cuda.synchronize()
    got = []
    for late in (False, True):
        c0s = [torch.zeros_like(c) for c in start]
        c2s, rhos = [torch.zeros_like(c) for c in start], [torch.zeros_like(v) for v in vs]
        torch.cuda.synchronize()
        ex = Exchange(late)
        if late:
            torch.cuda._sleep(20_000_000)
        for c, x in zip(c0s, start):
            c.copy_(x)
        if not late:
            torch.cuda.synchronize()
        out = [gram(slabs, ex, c0s, c0s, e.nstate)[0]]
        if late:
            for c in c0s:
                torch.cuda._sleep(20_000_000)
                c.mul_(1.0)
        apply_local_h(slabs, ex, c0s, vs, c2s)
        density(slabs, ex, c0s, rhos)
        torch.cuda.synchronize()
        got.append([x.cpu().numpy() for x in out + c2s + rhos])
    for x in slabs:
        x.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
