"""Grid lengths without a compile-time transform: the band pairs go through the
slab passes and the density-sphere fields through the shared-memory FFT, whose
kernels also carry the conjugate at -G, the GGA gradient fields and the real
part of V(r).  One H|psi> stage by stage against the oracle, the sphere
transform against numpy.

Bars: 1e-10 of the maximum in FP64 and 1e-5 mixed, as in the parity tests; the
transform alone 1e-11."""
import dataclasses
import math

import numpy as np
import pytest

from amdkiit_b200 import configs
from amdkiit_b200.engine import FP64, MIXED, Engine
from amdkiit_b200.inputs import XC_PBE, XC_PZ
from oracle.oracle import Oracle
from tests.helpers import start_coefficients

pytestmark = pytest.mark.gpu

BAR = {FP64: 1e-10, MIXED: 1e-5}


def _system(n, xc=XC_PZ):
    box = 12.0 if n < 100 else 20.0
    s = configs.cluster(2, box, 40 + n, ecut=((n - 0.9) * math.pi / (2.0 * box)) ** 2)
    return dataclasses.replace(s, xc=xc)


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("n,xc", [(40, XC_PBE), (50, XC_PZ), (54, XC_PBE), (150, XC_PBE)])
def test_stages_match_oracle(n, xc, prec):
    s = _system(n, xc)
    o, e = Oracle(s, 0), Engine(s, prec)
    assert e.nr == (n, n, n)
    o.set_wfn(start_coefficients(o.gvectors()["hg"][: o.ngpw], o.d("tpiba"), o.nstate))
    assert o.ortho() == 0
    for r in ("eval_density", "rhor2g", "eval_pot", "cal_vpot_ex", "pp_energy", "vpsi", "fnonloc"):
        o.call(r)
    e.set_wfn(o.c0())
    e.density()
    e.potential()
    e.energy()
    e.apply_h()
    errs = {"rho": _rel(e.get("rho"), o.real_grid("rho")),
            "rho_g": _rel(e.get("rho_g"), o.arr("rho_g", (e.ngrho,), np.complex128)),
            "v_pot": _rel(e.get("v_pot"), o.real_grid("v_pot")), "c2": _rel(e.get("c2"), o.c2())}
    e.close()
    assert max(errs.values()) < BAR[prec], errs


@pytest.mark.parametrize("n", [40, 50, 54, 150])
def test_sphere_transform_matches_numpy(n):
    e = Engine(_system(n), FP64)
    g = e.gvectors()
    rng = np.random.default_rng(n)
    coef = (rng.standard_normal(e.ngrho) + 1j * rng.standard_normal(e.ngrho)) / (1.0 + g["hg"])
    coef[0] = coef[0].real
    k = g["inyh"] - (n // 2 + 1)
    full = np.zeros((n, n, n), complex)
    full[-k[:, 2] % n, -k[:, 1] % n, -k[:, 0] % n] = coef.conj()
    full[k[:, 2] % n, k[:, 1] % n, k[:, 0] % n] = coef
    _, grid = e.fft_sphere(-1, coef=coef)
    ref = np.fft.ifftn(full) * n**3
    assert np.abs(grid - ref).max() < 1e-11 * np.abs(ref).max()
    back, _ = e.fft_sphere(+1, grid=ref)
    assert np.abs(back - coef).max() < 1e-11 * np.abs(coef).max()
    e.close()


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("box,ecut,nr", [((9.0, 11.0, 12.0), 42.0, (40, 48, 50)), ((12.0, 8.5, 15.0), 40.0, (50, 36, 64))])
def test_three_different_lengths(box, ecut, nr, prec):
    """An orthorhombic cell: every axis with a length of its own, known at
    compile time or not, through the slab passes."""
    s = configs.cluster(1, 9.0, 77, ecut=ecut)
    s = dataclasses.replace(s, a_cell=np.diag(box), alat=box[0], xc=XC_PBE)
    o, e = Oracle(s, 0), Engine(s, prec)
    assert e.nr == nr
    o.set_wfn(start_coefficients(o.gvectors()["hg"][: o.ngpw], o.d("tpiba"), o.nstate))
    assert o.ortho() == 0
    for r in ("eval_density", "rhor2g", "eval_pot", "cal_vpot_ex", "pp_energy", "vpsi", "fnonloc"):
        o.call(r)
    e.set_wfn(o.c0())
    e.density()
    e.potential()
    e.energy()
    e.apply_h()
    errs = {"rho": _rel(e.get("rho"), o.real_grid("rho")), "v_pot": _rel(e.get("v_pot"), o.real_grid("v_pot")),
            "c2": _rel(e.get("c2"), o.c2())}
    e.close()
    assert max(errs.values()) < BAR[prec], errs
