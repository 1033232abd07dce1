"""The plane kernels in their less travelled forms, against the oracle: V(r)psi
that takes a plane's column groups in turn and sums their shares of the rays in
a scratch plane per block (160 points, FP64), with a potential per spin and over
the ray segments of a slab decomposition, where the number of blocks differs
from the one-GPU, closed-shell launch.

Bars as in the parity tests of these paths: 1e-10 of the array's maximum in
FP64, 1e-5 mixed."""
import dataclasses
import math

import numpy as np
import pytest

from amdkiit_b200 import configs
from amdkiit_b200.engine import FP64, MIXED, Engine
from amdkiit_b200.slab import LocalExchange, Slab, apply_local_h, density
from oracle.oracle import Oracle
from tests.helpers import load_fixture, start_coefficients

pytestmark = pytest.mark.gpu

BAR = {FP64: 1e-10, MIXED: 1e-5}


def _ecut(n, box):
    """The cutoff (Ry) whose grid in this box is n^3."""
    return ((n - 0.9) * math.pi / (2.0 * box)) ** 2


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def _oracle(system):
    o = Oracle(system, 0)
    o.set_wfn(start_coefficients(o.gvectors()["hg"][: o.ngpw], o.d("tpiba"), o.nstate, 21))
    assert o.ortho() == 0
    for r in ("eval_density", "rhor2g", "eval_pot", "cal_vpot_ex", "pp_energy", "vpsi"):
        o.call(r)
    return o


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("n", [144, 160])
def test_two_spins(n, prec):
    s = load_fixture("o2_triplet")
    s = dataclasses.replace(s, ecut=_ecut(n, s.alat))
    o = _oracle(s)
    local = o.c2()
    o.call("fnonloc")
    e = Engine(s, prec)
    assert e.nr == (n, n, n)
    e.set_wfn(o.c0())
    e.density()
    e.potential()
    e.energy()
    e.apply_h()
    errs = {"rho": _rel(e.get("rho"), o.real_grid("rho")), "rho2": _rel(e.get("rho2"), o.real_grid("rho2")),
            "v_pot": _rel(e.get("v_pot"), o.real_grid("v_pot")), "v_pot2": _rel(e.get("v_pot2"), o.real_grid("v_pot2")),
            "c2": float(np.abs(e.get("c2") - o.c2()).max() / np.abs(local).max())}
    e.close()
    assert max(errs.values()) < BAR[prec], errs


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("n,nranks", [(72, 3), (90, 3), (96, 2), (160, 1), (160, 3)])
def test_ray_segments(n, nranks, prec):
    import torch
    box = 13.0 if n < 100 else 24.0
    o = _oracle(configs.cluster(2, box, 40 + n, ecut=_ecut(n, box)))
    c0, v = o.c0(), o.real_grid("v_pot")
    e = Engine(configs.cluster(2, box, 40 + n, ecut=_ecut(n, box)), prec)
    assert e.nr == (n, n, n)
    slabs = [Slab(e, nranks, r) for r in range(nranks)]
    c0s = [torch.from_numpy(np.ascontiguousarray(c0[:, s.local_g])).cuda() for s in slabs]
    vs = [torch.from_numpy(np.ascontiguousarray(v[:, :, s.plane0:s.plane0 + s.nplane])).cuda() for s in slabs]
    c2s, rhos = [torch.zeros_like(c) for c in c0s], [torch.zeros_like(x) for x in vs]
    apply_local_h(slabs, LocalExchange(), c0s, vs, c2s)
    density(slabs, LocalExchange(), c0s, rhos)
    torch.cuda.synchronize()
    c2, rho = np.zeros_like(c0), np.zeros_like(v)
    for s, c, r in zip(slabs, c2s, rhos):
        c2[:, s.local_g] = c.cpu().numpy()
        rho[:, :, s.plane0:s.plane0 + s.nplane] = r.cpu().numpy()
    for s in slabs:
        s.close()
    errs = {"c2": _rel(c2, o.c2()), "rho": _rel(rho, o.real_grid("rho"))}
    e.close()
    assert max(errs.values()) < BAR[prec], errs
