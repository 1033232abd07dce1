"""The calls whose time matters to a program that uses this package.

Most of the work is the self-consistent-field (SCF) loop of one system
resident on a GPU: load a wavefunction, orthonormalise it, take conjugate
gradient (CG) iterations, read the wavefunction, energies and forces back
(`Engine`; an MD or geometry step is this loop at new positions).  Besides it
a program drives several small systems together (`Ensemble`), and applies the
transforms to its own GPU arrays (`slab`: density, local H|psi>, band-space
products), on one GPU or as the ranks of a decomposed system.

Systems come from `amdkiit_b200.configs`, at their own cutoffs or, for drawn
cases, over the range between the tests' 12-30 Ry and the configurations'
70 Ry.  The wavefunction of a case is seeded noise damped by 1/(1 + |G|^2), the
package's own start (`amdkiit_b200.guess`), made on the GPU; positions are
the configuration's, displaced by up to 0.05 bohr as an MD step would.

Mixed-precision engines work to single precision, and their program keeps
single-precision results: `run` hands them on as float32/complex64.
"""
import dataclasses
import math

import numpy as np
import torch

from amdkiit_b200 import configs
from amdkiit_b200.engine import FP64, MIXED, Engine, Ensemble
from amdkiit_b200.inputs import XC_PBE, XC_PZ, XC_TETER93, System
from amdkiit_b200.slab import LocalExchange, Slab, apply_local_h, density, gram

PRECISION = {"fp64": FP64, "mixed": MIXED}
XC = {"pz": XC_PZ, "pbe": XC_PBE, "teter": XC_TETER93}


def listed():
    return [
        # one molecule, closed shell: the quick check and the start of every study; 64^3 grid, 4 bands
        {"name": "scf_water1_fp64", "kind": "scf", "system": "water1", "ecut": 70.0, "precision": "fp64", "steps": 20},
        # an open-shell molecule (spin-polarised): O2 triplet, 12 bands of two spins, 7 of one and 5 of the other
        {"name": "scf_o2_triplet_fp64", "kind": "scf", "system": "o2", "ecut": 70.0, "grid": 60, "precision": "fp64",
         "steps": 20},
        # a cluster of five molecules, an odd cutoff: 20 bands
        {"name": "scf_cluster5_mixed", "kind": "scf", "system": "cluster", "mols": 5, "box": 15.3, "ecut": 63.0,
         "xc": "pbe", "precision": "mixed", "steps": 20},
        # a solid with s and p projectors (256 of them): 72^3 grid, 128 bands
        {"name": "scf_si64_mixed", "kind": "scf", "system": "si64", "ecut": 30.0, "precision": "mixed", "steps": 16},
        # the benchmark system, 32 molecules of liquid water: 100^3 grid, 128 bands, in both precisions
        {"name": "scf_water32_fp64", "kind": "scf", "system": "water32", "ecut": 70.0, "precision": "fp64", "steps": 16},
        {"name": "scf_water32_mixed", "kind": "scf", "system": "water32", "ecut": 70.0, "precision": "mixed", "steps": 16},
        # the largest configuration, 128 molecules: 160^3 grid, 512 bands
        {"name": "scf_water128_fp64", "kind": "scf", "system": "water128", "ecut": 70.0, "precision": "fp64", "steps": 3},
        # several small systems on one GPU, as in a screening of clusters
        {"name": "ensemble_clusters_mixed", "kind": "ensemble", "members": 6, "ecut": 70.0, "precision": "mixed", "steps": 12},
        # local H|psi> on the program's own GPU arrays, the system held as four ranks
        {"name": "local_h_water32_fp64", "kind": "local_h", "system": "water32", "ecut": 70.0, "precision": "fp64", "ranks": 4},
        # the density of the largest configuration on the program's own GPU arrays, 64 pairs of bands at a time
        {"name": "density_water128_mixed", "kind": "density", "system": "water128", "ecut": 70.0, "precision": "mixed",
         "ranks": 1, "pairs": 64},
        # overlap and Lambda-type matrices of a band set on the GPU
        {"name": "gram_water32_fp64", "kind": "gram", "system": "water32", "ecut": 70.0, "precision": "fp64", "ranks": 1},
    ]


def draw(rng):
    kind = rng.choice(["scf", "scf", "scf", "scf", "ensemble", "local_h", "density", "gram"])
    case = {"kind": kind, "precision": rng.choice(["fp64", "mixed"])}
    if kind == "ensemble":
        return dict(case, members=rng.randint(2, 6), ecut=round(rng.uniform(25.0, 70.0), 1), steps=rng.randint(6, 14))
    system = rng.choice(["water1", "o2", "cluster", "cluster", "si64", "water32"] if kind == "scf" else
                        ["cluster", "si64", "water32"])
    case["system"] = system
    case["ecut"] = round(math.exp(rng.uniform(math.log(12.0), math.log(30.0))) if system == "si64" else
                         math.exp(rng.uniform(math.log(22.0), math.log(70.0))), 1)
    if system == "o2":
        case["grid"] = rng.choice([36, 48, 60, 64, 72])  # the open-shell branch is for these lengths
    if system == "cluster":
        mols = round(math.exp(rng.uniform(math.log(2.0), math.log(20.0))))
        case.update(mols=mols, box=round(9.5 + 4.0 * mols ** (1.0 / 3.0) * rng.uniform(0.95, 1.2), 2),
                    xc=rng.choice(["pz", "pbe"]))
    if kind == "scf":
        return dict(case, steps=rng.randint(8, 16))
    return dict(case, ranks=1 if kind == "gram" else rng.choice([1, 2, 3, 5, 8]))


def _o2_box(ecut, grid):
    """The cell (bohr) whose grid at this cutoff is `grid`."""
    return round((grid - 0.9) * math.pi / (2.0 * math.sqrt(ecut)), 4)


def _o2(ecut, grid):
    """An O2 molecule (bond 2.28 bohr), multiplicity 3."""
    box, half = _o2_box(ecut, grid), 1.14
    pos = np.array([[box / 2, box / 2, box / 2 - half], [box / 2, box / 2, box / 2 + half]])
    return System(a_cell=np.diag([box] * 3), alat=box, symmetry=1, ecut=ecut, species=[configs.gth_oxygen()],
                  positions=[pos], xc=XC_TETER93, name="o2", multiplicity=3)


def _system(case, rng):
    name, ecut = case["system"], case["ecut"]
    if name == "o2":
        system = _o2(ecut, case["grid"])
    elif name == "cluster":
        system = configs.cluster(case["mols"], case["box"], 1000 + case["mols"], ecut)
        system = dataclasses.replace(system, xc=XC[case["xc"]])
    else:
        system = configs.BY_NAME[name](ecut=ecut)
    return dataclasses.replace(system, positions=[p + rng.uniform(-0.05, 0.05, p.shape) for p in system.positions])


def _bands(engine, seed, nstate=None):
    """Seeded noise / (1 + |G|^2), G = 0 real: (nstate, ngpw) complex128 on the GPU."""
    tpiba = 2.0 * math.pi / engine.system.alat
    hg = torch.from_numpy(engine.gvectors()["hg"][:engine.ngpw] * tpiba * tpiba).cuda()
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.randn(nstate or engine.nstate, engine.ngpw, dtype=torch.complex128, device="cuda", generator=g)
    c /= 1.0 + hg
    c[:, 0].imag.zero_()
    return c


def _single(x):
    return x.astype(np.float32)


class _Scf:
    """An engine, the wavefunction to start from and the buffers to read it back into, in pinned host memory."""

    def __init__(self, system, precision, seed):
        self.engine = Engine(system, precision)
        self.single = precision == MIXED
        c = _bands(self.engine, seed)
        self.start = torch.empty(c.shape, dtype=c.dtype, pin_memory=True).copy_(c)
        self.c0 = torch.empty(c.shape, dtype=c.dtype, pin_memory=True)
        self.c0_single = torch.empty(c.shape, dtype=torch.complex64) if self.single else None

    def load(self):
        self.engine.set_wfn(self.start.numpy())
        self.engine.ortho()

    def results(self, energies, gemax):
        self.engine.get_wfn(self.c0.numpy())
        forces = self.engine.ionic_forces()
        scalars = np.array(list(energies.values()) + [gemax])
        if self.single:
            return [_single(scalars), self.c0_single.copy_(self.c0), _single(forces)]
        return [scalars, self.c0, forces]


class _Arrays:
    """The ranks of a system held by this process, with its arrays on the GPU: bands [nstate][local G], V(r) and
    rho(r) by slabs of x planes, and the output arrays."""

    def __init__(self, case, seed):
        self.kind = case["kind"]
        rng = np.random.default_rng(seed)
        self.engine = Engine(_system(case, rng), PRECISION[case["precision"]])
        self.single = case["precision"] == "mixed"
        self.slabs = [Slab(self.engine, case["ranks"], r) for r in range(case["ranks"])]
        self.exchange = LocalExchange()
        self.nstate, self.pairs = self.engine.nstate, _pairs(case, self.engine.nstate)
        c = _bands(self.engine, seed)
        self.full = c
        own = [torch.from_numpy(s.local_g).long().cuda() for s in self.slabs]
        self.c0 = [c if len(own) == 1 else c[:, o].contiguous() for o in own]
        if self.kind == "local_h":
            self.v = _potential(self.engine.nr, seed)
            self.vs = [self.v[:, :, s.plane0:s.plane0 + s.nplane].contiguous() for s in self.slabs]
            self.c2 = [torch.zeros_like(c) for c in self.c0]
        elif self.kind == "density":
            self.rho = [torch.zeros(s.grid, dtype=torch.float64, device="cuda") for s in self.slabs]
        else:
            c2 = _bands(self.engine, seed + 1)
            self.c2 = [c2 if len(own) == 1 else c2[:, o].contiguous() for o in own]


def _pairs(case, nstate):
    return min(case.get("pairs", nstate), (nstate + 1) // 2)


def _potential(nr, seed):
    """A smooth V(r) in Hartree: -1 to +0.6, as the potential of a molecule or a liquid."""
    n1, n2, n3 = nr
    x, y, z = (2.0 * math.pi * torch.arange(n, dtype=torch.float64, device="cuda") / n for n in nr)
    r = np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi, 6)
    return (-0.2 - 0.3 * torch.cos(z + r[0])[:, None, None] * torch.cos(2 * x + r[1])[None, None, :]
            + 0.3 * torch.sin(y + r[2])[None, :, None] * torch.sin(3 * z + r[3])[:, None, None]
            + 0.2 * torch.cos(y + r[4])[None, :, None] * torch.cos(x + r[5])[None, None, :]).contiguous()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    precision = PRECISION[case["precision"]]
    if case["kind"] == "scf":
        return {"steps": case["steps"], "scf": _Scf(_system(case, rng), precision, seed)}
    if case["kind"] == "ensemble":
        members = []
        for k in range(case["members"]):
            system = configs.cluster(1 + (3 * k) % 8, 12.0 + (0.7 * k) % 4.0, 1600 + k, case["ecut"])
            system = dataclasses.replace(
                system, positions=[p + rng.uniform(-0.05, 0.05, p.shape) for p in system.positions])
            members.append(_Scf(system, precision, seed + 100 * k))
        return {"steps": case["steps"], "members": members, "ensemble": Ensemble([m.engine for m in members])}
    return {"arrays": _Arrays(case, seed)}


def run(state):
    if "scf" in state:
        scf = state["scf"]
        scf.load()
        for i in range(1, state["steps"] + 1):
            energies, gemax, _ = scf.engine.scf_iteration(i, 1e-6)
        return scf.results(energies, gemax)
    if "ensemble" in state:
        members = state["members"]
        for m in members:
            m.load()
        for i in range(1, state["steps"] + 1):
            energies, gemax, _ = state["ensemble"].iteration([i] * len(members), 1e-6)
        return [m.results(e, float(g)) for m, e, g in zip(members, energies, gemax)]
    a = state["arrays"]
    if a.kind == "local_h":
        apply_local_h(a.slabs, a.exchange, a.c0, a.vs, a.c2)
        return [c.to(torch.complex64) for c in a.c2] if a.single else a.c2
    if a.kind == "density":
        for p0 in range(0, (a.nstate + 1) // 2, a.pairs):
            n = min(a.pairs, (a.nstate + 1) // 2 - p0)
            density(a.slabs, a.exchange, a.c0, a.rho, band0=2 * p0, npairs=n, accumulate=p0 > 0)
        return [r.float() for r in a.rho] if a.single else a.rho
    s = gram(a.slabs, a.exchange, a.c0, a.c0, a.nstate)
    lam = gram(a.slabs, a.exchange, a.c2, a.c0, a.nstate)
    return [s[0], lam[0]]


def exact(case, seed):
    """The band transforms and products in 64 bits by torch.fft and matmul; the engine's tables give only the order
    of the G vectors (the layout of the arrays) and the occupations' closed-shell 2."""
    if case["kind"] in ("scf", "ensemble"):
        return None  # a whole plane-wave DFT program: pseudopotentials, Ewald sums, functionals, CG
    a = _Arrays(case, seed)
    c, (n1, n2, n3) = a.full, a.engine.nr
    if case["kind"] == "gram":
        def product(x, y):
            return 2.0 * (x.real @ y.real.T + x.imag @ y.imag.T) - torch.outer(x[:, 0].real, y[:, 0].real)
        return [product(c, c), product(a.c2[0], c)]
    g = a.engine.gvectors()
    k = torch.from_numpy(g["inyh"][:a.engine.ngpw] - np.array([n1 // 2 + 1, n2 // 2 + 1, n3 // 2 + 1])).long().cuda()
    hg = torch.from_numpy(g["hg"][:a.engine.ngpw] * (2.0 * math.pi / a.engine.system.alat) ** 2).cuda()

    def at(m):
        return (m[:, 2] % n3, m[:, 1] % n2, m[:, 0] % n1)

    def real_space(band):
        f = torch.zeros(n3, n2, n1, dtype=torch.complex128, device="cuda")
        f[at(-k)] = band.conj()
        f[at(k)] = band
        return torch.fft.ifftn(f).real * (n1 * n2 * n3)

    planes = [slice(s.plane0, s.plane0 + s.nplane) for s in a.slabs]
    if case["kind"] == "density":
        rho = torch.zeros(n3, n2, n1, dtype=torch.float64, device="cuda")
        for band in c:
            rho += 2.0 / a.engine.info.omega * real_space(band) ** 2
        return [rho[:, :, p].contiguous() for p in planes]
    c2 = torch.empty_like(c)
    for b, band in enumerate(c):
        vpsi = torch.fft.fftn(a.v * real_space(band))[at(k)] / (n1 * n2 * n3)
        c2[b] = -2.0 * (0.5 * hg * band + vpsi)
    return [c2[:, torch.from_numpy(s.local_g).long().cuda()] for s in a.slabs]


def _sizes(case):
    """(bands, plane-wave half-sphere G vectors, density G vectors, grid points, nonlocal projectors) of a system."""
    if case["system"] == "si64":
        box, bands, proj = 20.52, 128, 256
    elif case["system"] == "o2":
        box, bands, proj = _o2_box(case["ecut"], case["grid"]), 12, 2
    else:
        mols = {"water1": 1, "water32": 32, "water128": 128}.get(case["system"], case.get("mols", 0))
        box = {"water1": 12.0, "water32": 18.63, "water128": 29.58}.get(case["system"], case.get("box", 0.0))
        bands, proj = 4 * mols, mols
    sphere = 4.0 / 3.0 * math.pi * (math.sqrt(case["ecut"]) * box / (2.0 * math.pi)) ** 3
    return bands, 0.5 * sphere, 4.0 * sphere, (4.0 * math.sqrt(case["ecut"]) * box / (2.0 * math.pi)) ** 3, proj


def _fft_flops(points, ng):
    """One complex 3D transform between the plane-wave sphere and the grid, the empty lines left out: of the three
    passes of 5/3 N log2 N the sphere needs pi/16 of the x lines, half of the y lines and every z line."""
    return 5.0 * points * math.log2(points) / 3.0 * (math.pi / 16.0 + 0.5 + 1.0)


def _work_scf(bands, ng, ngrho, points, proj, steps):
    wfn = 16.0 * bands * ng
    pairs = 0.5 * bands
    # an iteration: C0 and the CG direction read and written, C2 written and read, the projectors, the density and the
    # potential; then the wavefunction in and out of the pass
    per = {"bytes": 6.0 * wfn + 16.0 * proj * ng + 4.0 * 8.0 * points + 6.0 * 16.0 * ngrho,
           "flops": 3.0 * pairs * _fft_flops(points, ng) + 5.0 * 5.0 * points * math.log2(points)
           + (2.0 * (1.0 + 2.0 + 2.0 + 1.0) * bands + 4.0 * 2.0 * proj) * bands * ng}
    return {"bytes": steps * per["bytes"] + 2.0 * wfn, "flops": steps * per["flops"]}


def work(case):
    if case["kind"] == "ensemble":
        total = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["members"]):
            one = {"system": "cluster", "mols": 1 + (3 * k) % 8, "box": 12.0 + (0.7 * k) % 4.0, "ecut": case["ecut"]}
            for key, value in _work_scf(*_sizes(one), case["steps"]).items():
                total[key] += value
        return total
    bands, ng, ngrho, points, proj = _sizes(case)
    if case["kind"] == "scf":
        return _work_scf(bands, ng, ngrho, points, proj, case["steps"])
    wfn = 16.0 * bands * ng
    if case["kind"] == "local_h":
        return {"bytes": 2.0 * wfn + 8.0 * points, "flops": 2.0 * 0.5 * bands * _fft_flops(points, ng)}
    if case["kind"] == "density":
        return {"bytes": wfn + 8.0 * points, "flops": 0.5 * bands * (_fft_flops(points, ng) + 4.0 * points)}
    return {"bytes": 3.0 * wfn + 2.0 * 8.0 * bands * bands, "flops": 2.0 * 2.0 * ng * bands * bands * 1.5}
