"""The transforms at every specialised grid length, against the general ones.

The plane kernels of the band pairs (V(r)psi and the density, whole planes or
column groups, one launch shape per length and precision) against the slab
transforms of the same library (AMDK_NO_PENCIL=1), which share no code with
them beyond the register DFTs; the density-sphere transform against numpy.fft.
An odd cutoff and a cluster off the cell's centre leave the sphere short of the
slab the kernels are compiled for.

Bars: FP64 1e-11 of the array's maximum (a transform of 160^3 points accumulates
about 20 rounding errors of 1.1e-16 per element, the sums over eight bands
little more), mixed 1e-5 (the same with 6e-8)."""
import math

import numpy as np
import pytest

from amdkiit_b200 import configs
from amdkiit_b200.engine import FP64, MIXED, Engine
from tests.helpers import start_coefficients

pytestmark = pytest.mark.gpu

LENGTHS = [36, 48, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 160]
BAR = {FP64: 1e-11, MIXED: 1e-5}


def _system(n, short):
    """A two-molecule cluster (8 bands) whose grid is n^3; short: the smallest
    cutoff sphere that still takes that grid."""
    box = 13.0 if n < 100 else 24.0
    smaller = [m for m in range(2, n, 2) if _smooth(m)][-1]
    reach = smaller + 0.2 if short else n - 0.9
    return configs.cluster(2, box, 40 + n, ecut=(reach * math.pi / (2.0 * box)) ** 2)


def _smooth(m):
    for f in (2, 3, 5):
        while m % f == 0:
            m //= f
    return m == 1


def _run(system, prec):
    e = Engine(system, prec)
    g = e.gvectors()
    e.set_wfn(start_coefficients(g["hg"][: e.ngpw], 2 * np.pi / system.alat, e.nstate))
    e.ortho()
    e.density()
    e.potential()
    e.energy()
    e.apply_h()
    out = {k: e.get(k) for k in ("rho", "v_pot", "c2")}
    nr = e.nr
    e.close()
    return nr, out


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("n", LENGTHS)
def test_plane_kernels_match_the_slab_transforms(n, prec, monkeypatch):
    system = _system(n, short=(n % 3 == 0) != (prec == MIXED))
    nr, got = _run(system, prec)
    assert nr == (n, n, n)
    monkeypatch.setenv("AMDK_NO_PENCIL", "1")
    _, ref = _run(system, prec)
    for k in got:
        err = np.abs(got[k] - ref[k]).max() / np.abs(ref[k]).max()
        assert err < BAR[prec], f"{k} at {n}: {err:.2e}"


@pytest.mark.parametrize("n", LENGTHS)
def test_sphere_transform_matches_numpy(n):
    e = Engine(_system(n, short=False), FP64)
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
