"""The band products in the forms that the other tests leave out: both
triangles of the overlap with its G = 0 term, matrices with an odd leading
dimension (copied into padded rows for TMA), and overlaps so small that the
Cholesky's pivots are scaled for their reciprocal square root."""
import dataclasses

import numpy as np
import pytest

from amdkiit_b200 import configs
from amdkiit_b200.engine import FP64, MIXED, Engine
from oracle.oracle import Oracle
from tests.helpers import start_coefficients

pytestmark = pytest.mark.gpu


def _start(e, s):
    g = e.gvectors()
    return start_coefficients(g["hg"][: e.ngpw], 2 * np.pi / s.alat, e.nstate)


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def _hydrogens(n):
    """n H2 molecules, so n doubly occupied bands, in a 16 bohr box."""
    rng = np.random.default_rng(n)
    centres = np.array([[x, y, z] for z in (2.5, 8.0, 13.5) for y in (2.5, 8.0, 13.5) for x in (2.5, 8.0, 13.5)])[:n]
    d = rng.standard_normal((n, 3))
    d *= 0.7 / np.linalg.norm(d, axis=1)[:, None]
    s = configs.water1(ecut=16.0)
    return dataclasses.replace(s, a_cell=np.diag([16.0] * 3), alat=16.0, species=[configs.gth_hydrogen()],
                               positions=[np.concatenate([centres + d, centres - d])], name=f"h2_{n}")


@pytest.mark.parametrize("system,prec", [
    (configs.cluster(3, 13.5, 503, ecut=30.0), FP64), (configs.cluster(18, 18.4, 718, ecut=16.0), FP64),
    (configs.cluster(18, 18.4, 718, ecut=16.0), MIXED), (configs.cluster(40, 22.0, 740, ecut=16.0), FP64)],
    ids=["12", "72", "72-mixed", "160"])
def test_overlap_of_both_triangles(system, prec):
    """S = 2 Re C0^T C0 - Re c0(0) Re c0(0)^T below the diagonal as well.  Bars:
    FP64 1e-12, as for the upper triangle; mixed 1e-5 (28-bit operands, the 10
    leading digit products of 16: about 2^-21)."""
    e = Engine(system, prec)
    c = _start(e, system)
    e.set_wfn(c)
    e.ortho()
    S = 2.0 * (c.conj() @ c.T).real - np.outer(c[:, 0].real, c[:, 0].real)
    got = e.get("overlap")
    e.close()
    assert _rel(got, S) < (1e-12 if prec == FP64 else 1e-5)


@pytest.mark.parametrize("nbands", [1, 3, 9, 27])
def test_odd_band_counts(nbands):
    """One CG iteration's products with an odd number of bands against the
    oracle: the rotations and C2 -= C0 Lambda take padded matrices.  Bar 1e-10,
    as in the stage by stage parity test."""
    s = _hydrogens(nbands)
    o, e = Oracle(s, 0), Engine(s, FP64)
    assert e.nstate == nbands
    c = _start(e, s)
    o.set_wfn(c)
    e.set_wfn(c)
    assert o.ortho() == 0
    e.ortho()
    errs = {"ortho": _rel(e.get_wfn(), o.c0())}
    for r in ("eval_density", "rhor2g", "eval_pot", "cal_vpot_ex", "pp_energy", "vpsi", "fnonloc", "forces"):
        o.call(r)
    e.density()
    e.potential()
    e.energy()
    e.apply_h()
    e.gradient()
    errs["gradient"] = _rel(e.get("c2"), o.c2())
    o.call("pcg", 1)
    e.pcg(1)
    assert o.ortho() == 0
    e.ortho()
    errs["c0"] = _rel(e.get_wfn(), o.c0())
    e.close()
    assert max(errs.values()) < 1e-10, errs


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("ecut,n", [(16.0, 54), (20.0, 60)])
def test_odd_projector_count_above_the_fused_limit(ecut, n, prec):
    """33 projectors: C2 += P D as one product of padded D, with the default
    batch and in batches of an odd number of pairs (band offsets into D), on a
    run-time length and on the plane kernels.  Bars 1e-10 FP64, 1e-5 mixed, as
    in the parity tests."""
    s = configs.cluster(33, 20.5, 733, ecut=ecut)
    o = Oracle(s, 0)
    o.set_wfn(start_coefficients(o.gvectors()["hg"][: o.ngpw], o.d("tpiba"), o.nstate))
    assert o.ortho() == 0
    for r in ("eval_density", "rhor2g", "eval_pot", "cal_vpot_ex", "pp_energy", "vpsi", "fnonloc"):
        o.call(r)
    for batch in (0, 7):
        e = Engine(s, prec, pair_batch=batch)
        assert e.nr == (n, n, n)
        e.set_wfn(o.c0())
        e.density()
        e.potential()
        e.energy()
        e.apply_h()
        err = _rel(e.get("c2"), o.c2())
        e.close()
        assert err < (1e-10 if prec == FP64 else 1e-5), (batch, err)


@pytest.mark.parametrize("power", [-480, -150, 150])
def test_orthonormalisation_does_not_depend_on_the_scale(power):
    """C0 times 2^power gives the same orthonormal C0: the powers of two go
    through every product exactly, and only the pivots' reciprocal square roots
    see another argument (below 2^-900 a scaled one): under 1 ulp each, times
    the overlap's condition number (below 3 here), 72 bands.  Bar 1e-11."""
    s = configs.cluster(18, 18.4, 718, ecut=16.0)
    e = Engine(s, FP64)
    c = _start(e, s)
    out = []
    for f in (1.0, 2.0 ** power):
        e.set_wfn(c * f)
        e.ortho()
        out.append(e.get_wfn())
    e.close()
    assert _rel(out[1], out[0]) < 1e-11


def test_reciprocal_square_root_of_a_pivot():
    """One band: U^-1 is the pivot's reciprocal square root (the hardware's
    approximation and two Newton steps), so C0 U^-1 over C0 shows it.  Over the
    binades from 2^-1000 to 2^200 it is within 1 ulp, the bound of CUDA's own
    rsqrt: 2^-52, and 2^-53 for the product's rounding."""
    s = _hydrogens(1)
    e = Engine(s, FP64)
    c = _start(e, s)
    rng = np.random.default_rng(5)
    worst = 0.0
    for power in np.concatenate([rng.uniform(-500.0, 100.0, 200), rng.uniform(-451.0, -449.0, 40)]):
        x = c * 2.0 ** power
        e.set_wfn(x)
        e.ortho()
        exact = np.longdouble(1.0) / np.sqrt(np.longdouble(e.get("overlap")[0, 0]))
        y = e.get_wfn()
        big = np.abs(x.real) > 0.1 * np.abs(x.real).max()
        ratio = np.longdouble(y.real[big]) / (np.longdouble(x.real[big]) * exact)
        worst = max(worst, float(np.abs(ratio - 1).max()))
    e.close()
    assert worst <= 2.0 ** -52 + 2.0 ** -53, worst
