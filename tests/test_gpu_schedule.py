"""The density against its own schedule: the (plane, column group, pair) units
of a batch are split evenly over the resident blocks, each block adding its
pairs of one (plane, group) in its registers (in FP32 at most 32 pairs, then
into the FP64 partial grid), so the pair batch changes which terms are added
where, and later batches add to the grid.

Bars: FP64 1e-13 of the maximum (64 terms of 1.1e-16 rounding); mixed 4e-6 (at
most 32 terms of 6e-8 on either side)."""
import numpy as np
import pytest

from amdkiit_b200 import configs
from amdkiit_b200.engine import FP64, MIXED, Engine
from tests.helpers import load_fixture, start_coefficients

pytestmark = pytest.mark.gpu

BAR = {FP64: 1e-13, MIXED: 4e-6}


def _rho(system, prec, batch):
    e = Engine(system, prec, pair_batch=batch)
    g = e.gvectors()
    e.set_wfn(start_coefficients(g["hg"][: e.ngpw], 2 * np.pi / system.alat, e.nstate, 7))
    e.density()
    rho = e.get("rho")
    e.close()
    return rho


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_density_of_64_pairs_in_batches(prec):
    """64 pairs at once (the mixed sums are carried over at 32), 33 and 31, 5 at
    a time with 4 left, one at a time."""
    s = configs.water32(ecut=30.0)
    ref = _rho(s, prec, 0)
    for batch in (33, 5, 1):
        rho = _rho(s, prec, batch)
        err = np.abs(rho - ref).max() / np.abs(ref).max()
        assert err < BAR[prec], (batch, err)


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_two_spins_in_batches(prec):
    """O2 triplet, 6 pairs of which the third straddles the spins: in batches of
    4, 2 and 1 the spin-2 density is formed from the rays again and V(r)psi
    counts the pairs from the batch's first.  Bars of the densities as above; of
    H|psi>, whose potentials magnify the difference at low densities, 1e-10 and
    1e-5, as in the parity tests."""
    s = load_fixture("o2_triplet")
    ref = None
    for batch in (0, 4, 2, 1):
        e = Engine(s, prec, pair_batch=batch)
        g = e.gvectors()
        e.set_wfn(start_coefficients(g["hg"][: e.ngpw], 2 * np.pi / s.alat, e.nstate, 7))
        e.ortho()
        e.density()
        e.potential()
        e.energy()
        e.apply_h()
        got = [e.get(k) for k in ("rho", "rho2", "c2")]
        e.close()
        if ref is None:
            ref = got
            continue
        for k, a, b in zip(("rho", "rho2", "c2"), got, ref):
            err = np.abs(a - b).max() / np.abs(b).max()
            assert err < (BAR[prec] if k != "c2" else 1e-10 if prec == FP64 else 1e-5), (k, batch, err)
