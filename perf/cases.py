"""Performance cases: what a program does with this package, on synthetic inputs.

Every case is one call path of the SQ step on one processor block of a
periodic cell: the density / energy step in its three forms, the nonlocal
forces, the adjoint, the projector tables, and the pseudocharge density with
the local forces.  Cells, spacings, truncation radii, Chebyshev orders and
temperatures are those of the package's own systems (configs/gen_configs.py);
potentials, atomic positions and radial tables are smooth synthetic ones made
from the seed.  A block smaller than the cell is what one process of a larger
run holds.

``exact`` restates each path in plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sqdft_b200 import sq
from sqdft_b200.case import AtomType, Case
from sqdft_b200.pseudocharge import LocalAtoms, LocalGrid, projector_replicas, pseudocharge_replicas

HARTREE_EV = 27.211384523
# weights of the 12th-order central differences: second derivative, first derivative
LAP = [-5369 / 1800, 12 / 7, -15 / 56, 10 / 189, -1 / 112, 2 / 1925, -1 / 16632]
GRAD = [0.0, 6 / 7, -15 / 56, 5 / 63, -1 / 56, 1 / 385, -1 / 5544]
FD = 6
RC_TILDA = 0.5
# per species: valence, projector radius, reach of its pseudocharge, local
# channel, largest channel, projector amplitude and width, denominator h^3
SPECIES = {
    "Al": dict(z=3.0, rc=2.58, rb=6.0, lloc=1, lmax=1, amp=0.30, width=1.15, den=0.0571, core=1.8),
    "Li": dict(z=1.0, rc=3.00, rb=8.0, lloc=0, lmax=1, amp=0.28, width=1.30, den=-0.0421, core=1.5),
    "H": dict(z=1.0, rc=1.30, rb=8.0, lloc=0, lmax=0, amp=0.0, width=1.0, den=1.0, core=1.1),
}
FCC = [(0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0)]
SYSTEMS = {
    "al": dict(lattice=7.78, basis=[("Al", FCC)], depth={"Al": 0.35}),
    "lih": dict(lattice=7.72, basis=[("Li", FCC), ("H", [((x + .5) % 1, y, z) for x, y, z in FCC])],
                depth={"Li": 0.5, "H": 0.9}),
}


def listed():
    return [
        # The smallest call: a 4-atom cell on 8^3, 9^3 windows, where launches and latency count.
        _c("sq_fp64_w9", "sq", cells=1, per_cell=8, block=[8, 8, 8], nloc=4, npl=16, kt=5.0),
        # The reference's regression system: 10^3 grid, 17^3 windows, order 28.
        _c("sq_fp64_w17", "sq", cells=1, per_cell=10, block=[10, 10, 10], nloc=8, npl=28, kt=4.0),
        # A whole 4-atom cell at production spacing: 16^3 grid, 27^3 windows, order 64.
        _c("sq_fp64_w27", "sq", cells=1, per_cell=16, block=[16, 16, 16], nloc=13, npl=64, kt=5.0),
        # The 108-atom cell (48^3, 31^3 windows, order 96): one process's block, in the parity form ...
        _c("sq_fp64_w31", "sq", cells=3, per_cell=16, block=[16, 12, 6], nloc=15, npl=96, kt=5.0),
        # ... in the FP32-mixed form at its 1e-3 Ha stop ...
        _c("sq_mixed_w31", "sq", form=1, cells=3, per_cell=16, block=[16, 12, 6], nloc=15, npl=96, kt=5.0),
        # ... and in the Lanczos-quadrature form.
        _c("sq_quad_w31", "sq", form=2, cells=3, per_cell=16, block=[16, 12, 6], nloc=15, npl=96, kt=5.0),
        # Two species with three projectors beside none: 64-atom LiH, 33^3 windows, order 128.
        _c("sq_fp64_w33_lih", "sq", system="lih", cells=2, per_cell=20, block=[10, 8, 5], nloc=16, npl=128, kt=3.0),
        # A finer grid (h = 0.389) with its wider window, ragged block: 39^3 windows.
        _c("sq_fp64_w39", "sq", cells=1, per_cell=20, block=[9, 7, 7], nloc=19, npl=96, kt=5.0),
        # Nonlocal forces after the step, same block as the 31^3 cases.
        _c("forces_w31", "forces", cells=3, per_cell=16, block=[16, 12, 6], nloc=15, npl=96, kt=5.0),
        # The adjoint (gradients for the potential and the atoms): 32-atom cell, 27^3 windows, order 64.
        _c("vjp_w27", "vjp", cells=2, per_cell=16, block=[8, 8, 8], nloc=13, npl=64, kt=5.0),
        # Pseudocharge density and local forces of the 500-atom cell, 80^3 grid.
        _c("local_g80", "local", cells=5, per_cell=16, block=[80, 80, 80], nloc=1, npl=4, kt=10.0),
        # Its projector tables, made anew for every MD step.
        _c("projectors_g80", "projectors", cells=5, per_cell=16, block=[80, 80, 80], nloc=15, npl=4, kt=10.0),
    ]


def _c(name, kind, **kw):
    d = dict(name=name, kind=kind, system="al", form=0)
    d.update(kw)
    d["block"] = "x".join(str(b) for b in d["block"])
    return d


def draw(rng):
    """One more case: any path, species and form; window half-width 4..21, order
    16..128, a ragged block whose work stays below the largest listed case's."""
    kind = rng.choice(["sq", "sq", "sq", "sq", "forces", "forces", "vjp", "local", "projectors"])
    system = rng.choice(["al", "al", "lih"])
    per_cell = rng.randint(10, 20) if system == "lih" else rng.randint(8, 18)
    kt = round(rng.uniform(4.5, 10.0), 2)
    if kind in ("local", "projectors"):
        cells = rng.randint(1, 4)
        per_cell += per_cell % 2
        n = cells * per_cell
        block = [rng.randint(max(2, n // 2), n) for _ in range(3)]
        return dict(kind=kind, system=system, form=0, cells=cells, per_cell=per_cell,
                    block="x".join(map(str, block)), nloc=rng.randint(4, 16), npl=16, kt=kt)
    nloc = round(math.exp(rng.uniform(math.log(4), math.log(21.99))) - 0.5)
    # an order that resolves the occupation on the grid's spectral range (about 10 / h^2)
    h = SYSTEMS[system]["lattice"] / per_cell
    npl = min(128, 4 * max(rng.randint(4, 32), math.ceil(0.15 * 5 / h ** 2 / (kt / HARTREE_EV))))
    # at most about 110 atoms whose projectors reach a window
    atoms = sum(len(b) for _, b in SYSTEMS[system]["basis"])
    while nloc > 4 and atoms * ((2 * nloc + 1) / per_cell + 6.5 / SYSTEMS[system]["lattice"]) ** 3 > 110:
        nloc -= 1
    w = (2 * nloc + 1) ** 3
    # node-sweep points of the case: a share of the 31^3 block's (1152 nodes, about 110 sweeps)
    cap = math.exp(rng.uniform(math.log(0.02), 0.0)) * 1152 * 31 ** 3 * 110
    sweeps = {"sq": 64 + npl / 2, "forces": npl * 1.1, "vjp": npl * 6.0}[kind]
    nodes = max(8, min(4096, int(cap / (w * sweeps))))
    side = max(2, round(nodes ** (1 / 3)))
    block = [max(1, min(side + rng.randint(-1, 1), side)), side, 1]
    block[2] = max(1, nodes // (block[0] * block[1]))
    cells = max(1, -(-max(block) // per_cell))
    form = rng.choice([0, 0, 1, 2]) if kind == "sq" else rng.choice([0, 1]) if kind == "forces" else 0
    return dict(kind=kind, system=system, form=form, cells=cells, per_cell=per_cell,
                block="x".join(map(str, block)), nloc=nloc, npl=npl, kt=kt)


# -- inputs ---------------------------------------------------------------------

def _radial_grid():
    i = np.arange(1069)
    return 116.75 * np.expm1(0.0125 * i) / math.expm1(0.0125 * 1068)


def _erf(x):
    return torch.erf(torch.from_numpy(np.asarray(x, np.float64))).numpy()


def _rvloc(s, r):
    """r V_loc(r) and its derivative: -z erf(r / core)."""
    return -s["z"] * _erf(r / s["core"]), -s["z"] * 2 / math.sqrt(math.pi) / s["core"] * np.exp(-(r / s["core"]) ** 2)


def _projector_table(s):
    r = _radial_grid()
    t = np.zeros((19, r.size))
    t[0] = r
    t[1], t[10] = _rvloc(s, r)
    g = np.exp(-(r / s["width"]) ** 2)
    for l in range(4):  # channel potentials r V_l and radial functions r U_l, with derivatives
        on = 1.0 if l <= s["lmax"] and l != s["lloc"] else 0.0
        t[2 + l] = t[1] + on * r * g
        t[11 + l] = t[10] + on * g * (1 - 2 * (r / s["width"]) ** 2)
        t[6 + l] = on * s["amp"] * r * r ** l
        t[15 + l] = on * s["amp"] * (l + 1) * r ** l
    return t


def _local_table(s):
    r = _radial_grid()
    v, dv = _rvloc(s, r)
    a = 1.1
    uu = s["z"] / (math.pi ** 1.5 * a ** 3) * np.exp(-(r / a) ** 2)
    return np.stack([r, v, dv, uu, -2 * r / a ** 2 * uu])


def _atoms(case, seed):
    """Positions and types, type by type: displaced lattice sites."""
    sysd = SYSTEMS[case["system"]]
    rng = np.random.default_rng(seed)
    cells, lat = case["cells"], sysd["lattice"]
    corner = np.array([(x, y, z) for z in range(cells) for y in range(cells) for x in range(cells)], float)
    xyz, typ = [], []
    for t, (_, basis) in enumerate(sysd["basis"]):
        p = (corner[:, None, :] + np.array(basis)[None]).reshape(-1, 3) * lat
        d = rng.normal(0, 0.1, p.shape)
        if case["kind"] == "projectors":  # small moves keep every atom's grid node, and so the tables' size
            d = np.clip(d, -0.2 * lat / case["per_cell"], 0.2 * lat / case["per_cell"])
        xyz.append(np.mod(p + d, cells * lat))
        typ += [t] * len(p)
    return np.concatenate(xyz), np.array(typ, np.int32), rng


def _wells(points, centres, width, domain):
    """exp(-d^2/width^2) of grid points to centres along one axis, minimum image."""
    d = np.abs(points[:, None] - centres[None])
    d = np.minimum(d, domain - d)
    return np.exp(-(d / width) ** 2)


def _case(case, seed):
    sysd = SYSTEMS[case["system"]]
    n = case["cells"] * case["per_cell"]
    h = sysd["lattice"] / case["per_cell"]
    domain = n * h
    block = [int(b) for b in case["block"].split("x")]
    xyz, typ, rng = _atoms(case, seed)
    start = [int(rng.integers(0, n - b + 1)) if b < n and case["kind"] != "projectors" else 0 for b in block]
    nl = case["nloc"]
    types = []
    for t, (name, _) in enumerate(sysd["basis"]):
        s = SPECIES[name]
        den = np.array([s["den"] / h ** 3 if l <= s["lmax"] and l != s["lloc"] else 0.0 for l in range(4)])
        types.append(AtomType(natm=int((typ == t).sum()), lmax=s["lmax"], lloc=s["lloc"],
                              nlocc=math.ceil(s["rc"] / h), rc=s["rc"], denom=den, z=s["z"],
                              nproj=sum(2 * l + 1 for l in range(s["lmax"] + 1) if l != s["lloc"]),
                              tables=_projector_table(s)))
    rt, ra, rx = projector_replicas(xyz, typ, [t.rc for t in types], [domain] * 3, [n] * 3, start, block, nl)
    # Veff: a well at every atom and a few long waves, on the periodic grid, then the block with its halo
    veff = np.full((n, n, n), 0.05)
    g = np.arange(n) * h
    for t, (name, _) in enumerate(sysd["basis"]):
        c = xyz[typ == t]
        wx, wy, wz = (_wells(g, c[:, d], 1.6, domain) for d in range(3))
        yx = (wy[:, None, :] * wx[None, :, :]).reshape(n * n, -1)
        veff -= sysd["depth"][name] * (wz @ yx.T).reshape(n, n, n)
    for _ in range(3):
        k = 2 * math.pi / domain * rng.integers(-2, 3, 3)
        ph = rng.uniform(0, 2 * math.pi)
        veff += 0.01 * np.cos((k[2] * g)[:, None, None] + (k[1] * g)[None, :, None] + (k[0] * g)[None, None, :] + ph)
    ix = [(np.arange(block[d] + 2 * nl) + start[d] - nl) % n for d in range(3)]
    veff = np.ascontiguousarray(veff[np.ix_(ix[2], ix[1], ix[0])])
    z = np.array([t.z for t in types])
    electrons = float(z[typ].sum()) * np.prod(block) / n ** 3
    return Case(n_int=(n,) * 3, np_=tuple(block), pnode_s=tuple(start), nloc=nl, fdn=FD, npl=case["npl"], fermi_alg=1,
                n_atm=len(typ), scf_iter=1, delta=h, bet=HARTREE_EV / case["kt"], lanczos_tol=1e-6, fermi_tol=1e-6,
                ncharge=-electrons, lambda_f=0.0, temperature=0.0, rcut=nl * h, coeff_lap=np.array(LAP) / h ** 2,
                coeff_grad=np.array(GRAD) / h, veff=veff, types=types, rep_type=rt, rep_atom=ra, rep_xyz=rx,
                atoms_xyz=xyz, atom_type=typ)


def _given_bounds(c, seed):
    """Spectral bounds and Fermi-Dirac coefficients a force or adjoint call is handed."""
    rng = np.random.default_rng(seed + 1)
    top = -0.5 * 3 * (c.coeff_lap[0] + 2 * sum(c.coeff_lap[k] * (-1) ** k for k in range(1, FD + 1)))
    n = c.n_nodes
    lo = c.veff.min() - 2.0 - 0.05 * rng.random(n)
    hi = top + c.veff.max() + 2.0 + 0.05 * rng.random(n)
    chi, zee = (hi + lo) / 2, (hi - lo) / 2
    k = np.arange(c.npl + 1)
    x = np.cos(math.pi * (k + 0.5) / (c.npl + 1))
    f = 1 / (1 + np.exp(np.minimum(c.bet * (zee[:, None] * x + chi[:, None] - 0.2), 700.0)))
    ci = 2.0 / (c.npl + 1) * f @ np.cos(math.pi * np.outer(k + 0.5, k) / (c.npl + 1))
    ci[:, 0] /= 2
    return chi, zee, ci


def _local_inputs(case, seed):
    c = _case(dict(case, nloc=1), seed)
    names = [name for name, _ in SYSTEMS[case["system"]]["basis"]]
    rt, ra, rx, rb = pseudocharge_replicas(c.atoms_xyz, c.atom_type, [SPECIES[k]["rb"] for k in names],
                                           [c.n_int[0] * c.delta] * 3, c.n_int, c.pnode_s, c.np_)
    loc = LocalAtoms(tables=[_local_table(SPECIES[k]) for k in names], Z=np.array([SPECIES[k]["z"] for k in names]),
                     rep_type=rt, rep_atom=ra, rep_xyz=rx, rep_box=rb, rc_tilda=RC_TILDA)
    grid = LocalGrid(np_=c.np_, pnode_s=c.pnode_s, fdn=FD, delta=c.delta, coeff_lap=c.coeff_lap,
                     coeff_grad=c.coeff_grad, n_atm=c.n_atm)
    # the fields the forces read: an electrostatic potential with its halo, Vc, b, b_tilda
    rng = np.random.default_rng(seed + 1)
    sh = tuple(grid.np_[::-1])
    ax = [np.arange(s + 2 * FD) * c.delta for s in sh]
    w = 2 * math.pi / (c.n_int[0] * c.delta)
    phi = sum(rng.normal() * 0.1 * np.cos(w * (k + 1) * ax[0] + rng.uniform(0, 6))[:, None, None]
              * np.cos(w * ax[1] + rng.uniform(0, 6))[None, :, None]
              * np.cos(w * k * ax[2] + rng.uniform(0, 6))[None, None, :] for k in range(3))
    fields = [np.ascontiguousarray(phi)] + [rng.normal(0, 0.05, sh) for _ in range(3)]
    return grid, loc, fields


def prepare(case, seed):
    if case["kind"] == "local":
        grid, loc, fields = _local_inputs(case, seed)
        return dict(kind="local", ctx=sq.LocalContext(grid, loc), fields=fields)
    c = _case(case, seed)
    ctx = sq.Context(c, precision=case["form"])
    s = dict(kind=case["kind"], ctx=ctx)
    if case["kind"] == "projectors":
        return s
    ctx.nonlocal_projectors()
    if case["kind"] == "sq":
        if case["form"]:
            ctx.set_mixed_lanczos(1e-3, 0.5)
        s["veff"] = c.veff
    else:
        chi, zee, ci = _given_bounds(c, seed)
        if case["kind"] == "forces":
            s["args"] = (chi, zee, ci)
        else:
            ctx.moments_at(chi, zee)
            s["g_mu"] = _weights(ci, seed)
    return s


def _weights(ci, seed):
    """Moment weights of a density loss with weights in [0, 1]."""
    return 2 * np.random.default_rng(seed + 2).random(len(ci))[:, None] * ci


def run(state):
    ctx = state["ctx"]
    if state["kind"] == "sq":
        ctx.set_veff(state["veff"])  # every SCF iteration brings a new potential
        return _arrays(ctx.spectral_quadrature(1, 0.0))
    if state["kind"] == "forces":
        return ctx.forces_nonlocal(*state["args"])
    if state["kind"] == "vjp":
        return ctx.moments_vjp(state["g_mu"], atoms=True)
    if state["kind"] == "projectors":
        return ctx.nonlocal_projectors(copy_out=True)
    cd = ctx.charge_density()
    floc, fcorr = ctx.forces_local(*state["fields"])
    return _arrays(dict(cd, floc=floc, fcorr=fcorr))


def _arrays(d):
    """Scalars as 64-bit arrays."""
    return {k: np.asarray(v, np.float64) for k, v in d.items()}


# -- floors and tolerances --------------------------------------------------------

def work(case):
    """Bytes: inputs read once, outputs written once.  Flops of a window point
    and matvec: three 12th-order arms with shared coefficients, Veff, the
    recurrence and the projectors on the share of points their boxes cover."""
    block = [int(b) for b in case["block"].split("x")]
    nodes = math.prod(block)
    sysd = SYSTEMS[case["system"]]
    h = sysd["lattice"] / case["per_cell"]
    n = case["cells"] * case["per_cell"]
    sp = [(SPECIES[name], len(b)) for name, b in sysd["basis"]]
    if case["kind"] == "local":
        # per replica and point of its box: two radial values, two Laplacians, four gradients per axis
        reps = sum(k * case["cells"] ** 3 * math.prod((b + 2 * math.ceil(s["rb"] / h)) / n for b in block) for s, k in sp)
        vol = sum(k * (2 * math.ceil(s["rb"] / h) + 1) ** 3 for s, k in sp) / sum(k for _, k in sp)
        vol = min(vol, nodes)
        return dict(bytes=8.0 * nodes * 8, flops=reps * vol * (2 * 2 * 36 + 12 * 18 + 120.0))
    balls = [((2 * math.ceil(s["rc"] / h) + 1) ** 3 * sum(2 * l + 1 for l in range(s["lmax"] + 1) if l != s["lloc"]), k)
             for s, k in sp]
    cover = sum(v * k for v, k in balls) / case["per_cell"] ** 3  # projector values per grid point
    ext = math.prod(b + 2 * case["nloc"] for b in block)
    if case["kind"] == "projectors":
        return dict(bytes=8.0 * ext * cover, flops=ext * cover * 60.0)
    npl, w = case["npl"], (2 * case["nloc"] + 1) ** 3
    # Lanczos steps to the stop grow with the window edge and the spacing's spectral range (31^3 at h = 0.486: 64)
    steps = min(500.0, 2.1 * (2 * case["nloc"] + 1))
    sweeps = {"sq": [steps + npl / 2, 0.38 * steps + npl / 2, max(npl / 2 + 1, 0.9 * steps)][case["form"]],
              "forces": npl, "vjp": 3 * npl}[case["kind"]]
    io = ext * 8.0 * (1 + cover) + nodes * 8.0 * (2 * npl + 5)
    return dict(bytes=io, flops=nodes * w * sweeps * (48.0 + 4 * cover))


def tolerance(case):
    """Measured between the package's two node kernels (another order of every
    sum) and between forms, times about four."""
    if case["kind"] == "local":
        return {"rel": 1e-7, "max": 1e-7}  # Ecorr is what is left of terms 10^5 times its size
    if case["kind"] == "projectors":
        return {"rel": 1e-12, "max": 1e-10}
    if case["kind"] == "sq":
        # a rounding can move a node's Lanczos count by one, and its bounds by the stop (1e-6 or 1e-3 Ha);
        # the mixed form's bounds carry the rounding of FP32 vectors
        return [{"rel": 1e-7, "max": 1e-4}, {"rel": 1e-4, "max": 3e-2}, {"rel": 1e-4, "max": 3e-2}][case["form"]]
    if case["kind"] == "forces" and case["form"] == 1:
        return {"rel": 1e-4, "max": 1e-3}
    return {"rel": 1e-10, "max": 1e-9}


# -- 64-bit restatement -----------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _spline(tab, y, dy, r):
    """Cubic Hermite interpolation of rows y, dy of a radial table."""
    x = tab[0]
    j = (torch.searchsorted(x, r.contiguous()) - 1).clamp(0, x.numel() - 2)
    dx = 1.0 / (x[j + 1] - x[j])
    s = (y[j + 1] - y[j]) * dx
    t = r - x[j]
    a2 = dx * (3 * s - 2 * dy[j] - dy[j + 1])
    a3 = dx * dx * (-2 * s + dy[j] + dy[j + 1])
    return ((a3 * t + a2) * t + dy[j]) * t + y[j]


def _round(x):
    return int(math.floor(abs(x) + 0.5) * (1 if x >= 0 else -1))


def _ball(c, r, dev, shift=(0.0, 0.0, 0.0)):
    """Projector values [q, z, y, x] of replica r on its ball."""
    t = c.types[c.rep_type[r]]
    tab = torch.as_tensor(t.tables, device=dev)
    off = torch.arange(-t.nlocc, t.nlocc + 1, device=dev, dtype=torch.float64)
    d = [(off + _round(c.rep_xyz[r, k] / c.delta)) * c.delta - (c.rep_xyz[r, k] + shift[k]) for k in range(3)]
    z, y, x = torch.meshgrid(d[2], d[1], d[0], indexing="ij")
    rad = torch.sqrt(x * x + y * y + z * z)
    out = []
    for l, m in t.lm_list:
        v = _spline(tab, tab[2 + l], tab[11 + l], rad) / rad - _spline(tab, tab[1], tab[10], rad) / rad
        u = _spline(tab, tab[6 + l], tab[15 + l], rad) / rad
        sh = 0.282094791773878 if l == 0 else 0.488602511902920 * {-1: y, 0: z, 1: x}[m] / rad
        out.append(u * sh * v)
    return torch.stack(out) if out else torch.zeros((0,) + rad.shape, device=dev, dtype=torch.float64)


class _Windows:
    """H on the truncation windows of a batch of nodes."""

    def __init__(self, c, derivs=False):
        self.c, self.dev = c, _device()
        self.n = c.nw
        self.veff = torch.as_tensor(c.veff, device=self.dev)
        self.ext = self.veff.shape
        self.lap = [float(v) for v in c.coeff_lap]
        boxes, den, atom = [], [1.0], [0]
        for r in range(len(c.rep_type)):
            t = c.types[c.rep_type[r]]
            if t.nproj == 0:
                continue
            lo = [_round(c.rep_xyz[r, k] / c.delta) - t.nlocc - c.pnode_s[k] + c.nloc for k in range(3)]
            if any(lo[k] > self.ext[2 - k] - 1 or lo[k] + 2 * t.nlocc < 0 for k in range(3)):
                continue
            boxes.append((lo, 2 * t.nlocc, r, len(den)))
            den += [float(t.denom[l]) for l, _ in t.lm_list]
            atom += [int(c.rep_atom[r])] * t.nproj
        layers = []
        for b in boxes:  # balls of a layer do not overlap
            for lay in layers:
                if all(any(b[0][k] > o[0][k] + o[1] or o[0][k] > b[0][k] + b[1] for k in range(3)) for o in lay):
                    lay.append(b)
                    break
            else:
                layers.append([b])
        self.den = torch.tensor(den, device=self.dev, dtype=torch.float64)
        self.atom = torch.tensor(atom, device=self.dev)
        pm = max([t.nproj for t in c.types] + [1])
        self.layers = []
        for lay in layers:
            ids = torch.zeros(self.ext, dtype=torch.int64, device=self.dev)
            chi = torch.zeros((pm,) + tuple(self.ext), dtype=torch.float64, device=self.dev)
            dchi = torch.zeros((3, pm) + tuple(self.ext), dtype=torch.float64, device=self.dev) if derivs else None
            for lo, w, r, g in lay:
                cut = [(max(0, lo[k]), min(self.ext[2 - k] - 1, lo[k] + w)) for k in range(3)]
                at = tuple(slice(cut[k][0], cut[k][1] + 1) for k in (2, 1, 0))
                fr = (slice(None),) + tuple(slice(cut[k][0] - lo[k], cut[k][1] + 1 - lo[k]) for k in (2, 1, 0))
                u = _ball(c, r, self.dev)
                ids[at] = g
                chi[(slice(0, len(u)),) + at] = u[fr]
                for k in range(3) if derivs else ():
                    e = [1e-4 if j == k else 0.0 for j in range(3)]
                    du = (_ball(c, r, self.dev, e) - _ball(c, r, self.dev, [-v for v in e])) / 2e-4
                    dchi[(k, slice(0, len(u))) + at] = du[fr]
            self.layers.append((ids, chi, dchi))

    def batch(self, nodes):
        c, n, dev = self.c, self.n, self.dev
        nodes = torch.as_tensor(nodes, device=dev)
        o = torch.arange(n, device=dev)
        i, j, k = nodes % c.np_[0], (nodes // c.np_[0]) % c.np_[1], nodes // (c.np_[0] * c.np_[1])
        iz, iy, ix = k[:, None] + o, j[:, None] + o, i[:, None] + o
        at = (iz[:, :, None, None] * self.ext[1] + iy[:, None, :, None]) * self.ext[2] + ix[:, None, None, :]
        self.B = len(nodes)
        self.at = at
        self.v = self.veff.reshape(-1)[at]
        self.lay = []
        base = torch.arange(self.B, device=dev)[:, None, None, None] * len(self.den)
        for ids, chi, _ in self.layers:
            g = ids.reshape(-1)[at]
            self.lay.append((g, base + g, [x.reshape(-1)[at] for x in chi]))
        self.centre = (slice(None), c.nloc, c.nloc, c.nloc)

    def delta(self):
        v = torch.zeros((self.B, self.n, self.n, self.n), dtype=torch.float64, device=self.dev)
        v[self.centre] = 1.0
        return v

    def dots(self, v, fields=None):
        """chi^T v of every projector instance, [B, n_instances]."""
        out = torch.zeros(self.B * len(self.den) + 3, dtype=torch.float64, device=self.dev)
        for a, (g, bg, chi) in enumerate(self.lay):
            for q, x in enumerate(chi if fields is None else fields[a]):
                out.index_add_(0, (bg + q).reshape(-1), (x * v).reshape(-1))
        return out[:self.B * len(self.den)].reshape(self.B, -1)

    def apply(self, v):
        n = self.n
        p = torch.nn.functional.pad(v, (FD,) * 6)
        mid = slice(FD, FD + n)
        t = 3 * self.lap[0] * v
        for k in range(1, FD + 1):
            a, b = slice(FD - k, FD - k + n), slice(FD + k, FD + k + n)
            t += self.lap[k] * (p[:, mid, mid, a] + p[:, mid, mid, b] + p[:, mid, a, mid] + p[:, mid, b, mid]
                                + p[:, a, mid, mid] + p[:, b, mid, mid])
        h = -0.5 * t + self.v * v
        if self.lay:
            co = torch.cat([(self.dots(v) / self.den).reshape(-1), torch.zeros(3, dtype=torch.float64, device=self.dev)])
            for g, bg, chi in self.lay:
                for q, x in enumerate(chi):
                    h += co[bg + q] * x
        return h


def _extremes(a, b, m):
    """Smallest and largest eigenvalue of the m-row tridiagonals (diagonals
    a[:, :m], off-diagonals b[:, :m-1]) by 64-way bisection."""
    d, e = a[:, :m, None], b[:, :m, None]
    z = torch.zeros_like(e[:, :1])
    left = torch.cat([z, e[:, :m - 1]], 1).abs()
    right = torch.cat([e[:, :m - 1], z], 1).abs()
    lo = (d - left - right).amin((1, 2))
    hi = (d + left + right).amax((1, 2))
    lo, hi = torch.stack([lo, lo], 1), torch.stack([hi, hi], 1)
    f = torch.arange(1, 64, device=a.device, dtype=torch.float64) / 64
    want = torch.tensor([1, m], device=a.device)
    e2 = (e * e)[:, :, 0]
    for _ in range(10):
        x = lo[..., None] + (hi - lo)[..., None] * f
        q = d[:, 0, :, None] - x
        cnt = (q < 0).long()
        for i in range(1, m):
            q = d[:, i, :, None] - x - e2[:, i - 1, None, None] / torch.where(q == 0, torch.full_like(q, 1e-300), q)
            cnt += q < 0
        k = (cnt < want[:, None]).sum(-1)  # points below the wanted eigenvalue
        w = (hi - lo) / 64
        lo, hi = lo + w * k, lo + w * (k + 1)
    mid = (lo + hi) / 2
    return mid[:, 0], mid[:, 1]


def _lanczos(w, form, npl, tol):
    """Bounds after the reference's stop, and for the quadrature form the tridiagonal."""
    n, B = w.n, w.B
    if form == 2:
        v = w.delta()
    else:
        o = torch.arange(n, device=w.dev)
        s = 1.0 - 2.0 * ((o[:, None, None] + o[None, :, None] + o[None, None, :]) % 2).double()
        v = (1.0 + (0.5 if form == 1 else 0.0) * s).expand(B, n, n, n).clone()
        v /= v.norm() / math.sqrt(B)
    old, beta = torch.zeros_like(v), torch.zeros(B, dtype=torch.float64, device=w.dev)
    a = torch.zeros((B, 501), dtype=torch.float64, device=w.dev)
    b = torch.zeros_like(a)
    ends = prev = None
    lo, hi = torch.zeros(B, dtype=torch.float64, device=w.dev), torch.zeros(B, dtype=torch.float64, device=w.dev)
    rows = torch.zeros(B, dtype=torch.int64, device=w.dev)
    live = torch.ones(B, dtype=torch.bool, device=w.dev)
    bc = lambda x: x[:, None, None, None]
    kmin = npl // 2 + 1
    for m in range(500):
        y = w.apply(v) - bc(beta) * old
        a[:, m] = (y * v).sum((1, 2, 3))
        y -= bc(a[:, m]) * v
        if m + 2 >= kmin if form == 2 else m >= 1:
            ends = _extremes(a, b, m + 1)
            if form == 2 and prev is None:
                done = torch.zeros_like(live)
            else:
                p = prev if prev is not None else (torch.zeros_like(lo), torch.zeros_like(lo))
                done = ((ends[0] - p[0]).abs() <= tol) & ((ends[1] - p[1]).abs() <= tol)
            prev = ends
            fin = live & done
            lo, hi = torch.where(fin, ends[0], lo), torch.where(fin, ends[1], hi)
            rows = torch.where(fin, torch.full_like(rows, m + 1), rows)
            live = live & ~done
            if not bool(live.any()):
                break
        beta = (y * y).sum((1, 2, 3)).sqrt()
        b[:, m] = beta
        old, v = v, y / bc(beta)
    if bool(live.any()):
        lo, hi = torch.where(live, ends[0], lo), torch.where(live, ends[1], hi)
        rows = torch.where(live, torch.full_like(rows, 500), rows)
    return lo - tol, hi + tol, a, b, rows


def _exact_sq(case, c):
    w = _Windows(c)
    N, npl, h3 = c.n_nodes, c.npl, c.delta ** 3
    tol = max(c.lanczos_tol, 1e-3) if case["form"] else c.lanczos_tol
    chi, zee, mu = [], [], []
    size = max(1, min(N, int(9e6 / w.n ** 3)))
    for s in range(0, N, size):
        w.batch(np.arange(s, min(N, s + size)))
        lo, hi, a, b, rows = _lanczos(w, case["form"], npl, tol)
        x, z = (lo + hi) / 2, (hi - lo) / 2
        m = torch.zeros((w.B, npl + 1), dtype=torch.float64, device=w.dev)
        if case["form"] == 2:
            M = int(rows.max())
            keep = torch.arange(M, device=w.dev)[None] < rows[:, None]
            T = torch.diag_embed((a[:, :M] - x[:, None]) * keep)
            e = b[:, :M - 1] * keep[:, 1:]
            T = (T + torch.diag_embed(e, 1) + torch.diag_embed(e, -1)) / z[:, None, None]
            t0 = torch.zeros((w.B, M, 1), dtype=torch.float64, device=w.dev)
            t0[:, 0] = 1.0
            t1 = T @ t0
            m[:, 0], m[:, 1] = 1.0, t1[:, 0, 0]
            for j in range(2, npl + 1):
                t0, t1 = t1, 2 * (T @ t1) - t0
                m[:, j] = t1[:, 0, 0]
        else:
            bc = lambda q: q[:, None, None, None]
            t0 = w.delta()
            t1 = (w.apply(t0) - bc(x) * t0) / bc(z)
            m[:, 0], m[:, 1] = 1.0, t1[w.centre]
            half = npl // 2
            for j in range(2, half + 1):
                t0, t1 = t1, 2 * (w.apply(t1) - bc(x) * t1) / bc(z) - t0
                m[:, j] = t1[w.centre]
                m[:, 2 * j] = 2 * (t1 * t1).sum((1, 2, 3)) - 1
                m[:, 2 * j - 1] = 2 * (t1 * t0).sum((1, 2, 3)) - m[:, 1]
        chi.append(x)
        zee.append(z)
        mu.append(m / h3)
    chi, zee, mu = torch.cat(chi), torch.cat(zee), torch.cat(mu)
    K = npl + 1
    k = torch.arange(K, device=w.dev, dtype=torch.float64)
    xk = torch.cos(math.pi * (k + 0.5) / K)
    ct = torch.cos(math.pi * torch.outer(k, k + 0.5) / K) * (2.0 / K)
    ct[0] /= 2

    def occ(lam):
        return torch.sigmoid(-c.bet * zee[:, None] * (xk - (lam - chi[:, None]) / zee[:, None]))

    lo, hi = -100.0, 200.0
    for _ in range(100):
        lam = (lo + hi) / 2
        if float((2 * mu * (occ(lam) @ ct.T)).sum()) * h3 + c.ncharge > 0:
            hi = lam
        else:
            lo = lam
    f = occ(lam)
    ci = f @ ct.T
    r = (2 * mu * ci).sum(1)
    tiny = (f < 1e-14) | ((f - 1).abs() < 1e-14)
    ent = torch.where(tiny, torch.zeros_like(f), torch.xlogy(f, f) + torch.xlogy(1 - f, 1 - f))
    ebs = float((zee * (2 * mu * ((xk * f) @ ct.T)).sum(1) + chi * r).sum()) * h3
    eent = float((2 * mu * (ent @ ct.T)).sum()) * h3 / c.bet
    npy = lambda t: t.cpu().numpy()
    return _arrays(dict(rho=npy(r.abs()).reshape(c.np_[::-1]), rho_pj=npy(mu), Ci=npy(ci), chi=npy(chi),
                        zee=npy(zee), lambda_f=lam, Ebs=ebs, Eent=eent))


def _exact_forces(c, seed):
    w = _Windows(c)
    chi, zee, ci = (torch.as_tensor(x, device=w.dev) for x in _given_bounds(c, seed))
    out = torch.zeros((c.n_atm, 3), dtype=torch.float64, device=w.dev)
    size = max(1, min(c.n_nodes, int(9e6 / w.n ** 3)))
    bc = lambda q: q[:, None, None, None]
    h3 = c.delta ** 3
    n = w.n
    for s in range(0, c.n_nodes, size):
        e = slice(s, min(c.n_nodes, s + size))
        w.batch(np.arange(e.start, e.stop))
        x, z = bc(chi[e]), bc(zee[e])
        t0 = w.delta()
        t1 = (w.apply(t0) - x * t0) / z
        D = bc(ci[e, 0]) * t0 + bc(ci[e, 1]) * t1
        for j in range(2, c.npl + 1):
            t0, t1 = t1, 2 * (w.apply(t1) - x * t1) / z - t0
            D += bc(ci[e, j]) * t1
        p = torch.nn.functional.pad(D, (FD,) * 6)
        at0 = w.dots(w.delta())
        mid = slice(FD, FD + n)
        for k in range(3):
            g = torch.zeros_like(D)
            for q in range(1, FD + 1):
                a, b = slice(FD - q, FD - q + n), slice(FD + q, FD + q + n)
                ia = [mid] * 3
                ib = [mid] * 3
                ia[2 - k], ib[2 - k] = a, b
                g += float(c.coeff_grad[q]) * (p[(slice(None), *ib)] - p[(slice(None), *ia)])
            # D carries 1/h^3, the contraction h^3
            f = -4 * w.dots(g) * at0 / w.den
            out[:, k].index_add_(0, w.atom, f.sum(0))
    return out.cpu().numpy()


def _exact_vjp(c, seed):
    w = _Windows(c, derivs=True)
    chi, zee, ci = _given_bounds(c, seed)
    gm = torch.as_tensor(_weights(ci, seed), device=w.dev)
    chi, zee = torch.as_tensor(chi, device=w.dev), torch.as_tensor(zee, device=w.dev)
    h3, npl = c.delta ** 3, c.npl
    gv = torch.zeros(w.veff.numel(), dtype=torch.float64, device=w.dev)
    ga = torch.zeros((c.n_atm, 3), dtype=torch.float64, device=w.dev)
    size = max(1, min(c.n_nodes, int(4e9 / (8 * npl * w.n ** 3))))
    bc = lambda q: q[:, None, None, None]
    for s in range(0, c.n_nodes, size):
        e = slice(s, min(c.n_nodes, s + size))
        w.batch(np.arange(e.start, e.stop))
        x, z = bc(chi[e]), bc(zee[e])
        ec = w.delta()
        t = [ec, (w.apply(ec) - x * ec) / z]
        for j in range(2, npl):
            t.append(2 * (w.apply(t[-1]) - x * t[-1]) / z - t[-2])
        dl = [[[d.reshape(-1)[w.at] for d in dchi[k]] for _, _, dchi in w.layers] for k in range(3)]
        a1 = a2 = torch.zeros_like(ec)  # a_k+1, a_k+2
        g = torch.zeros_like(ec)
        for k in range(npl, 0, -1):
            a = bc(gm[e, k] / h3) * ec + 2 * (w.apply(a1) - x * a1) / z - a2
            a1, a2 = a, a1  # a1 = a_k
            fac = 1.0 if k == 1 else 2.0
            g += fac * a1 * t[k - 1]
            pa, pt = w.dots(a1), w.dots(t[k - 1])
            for d in range(3):
                q = (w.dots(a1, dl[d]) * pt + pa * w.dots(t[k - 1], dl[d])) / w.den * fac / zee[e][:, None]
                ga[:, d].index_add_(0, w.atom, q.sum(0))
        gv.index_add_(0, w.at.reshape(-1), (g / z).reshape(-1))
    return gv.reshape(w.ext).cpu().numpy(), ga.cpu().numpy()


def _exact_projectors(c):
    dev = _device()
    return np.concatenate([_ball(c, r, dev).cpu().numpy().reshape(-1) for r in range(len(c.rep_type))])


def _exact_local(case, seed):
    grid, loc, fields = _local_inputs(case, seed)
    dev = _device()
    T = lambda x: torch.as_tensor(x, device=dev)
    tabs = [T(t) for t in loc.tables]
    h, h3 = grid.delta, grid.delta ** 3
    sh = tuple(grid.np_[::-1])
    b, bt, vc, ra = (torch.zeros(sh, dtype=torch.float64, device=dev) for _ in range(4))
    phi, vcf, bf, btf = (T(f) for f in fields)
    lap, gr = [float(x) for x in grid.coeff_lap], [float(x) for x in grid.coeff_grad]
    scal = torch.zeros(5, dtype=torch.float64, device=dev)
    floc, fcorr = (torch.zeros((grid.n_atm, 3), dtype=torch.float64, device=dev) for _ in range(2))

    def inner(f, m):
        return f[m:-m, m:-m, m:-m]

    def shifted(f, ax, k, m):
        s = [slice(m, f.shape[i] - m) for i in range(3)]
        s[ax] = slice(m + k, f.shape[ax] - m + k)
        return f[tuple(s)]

    def nlap(f):
        t = 3 * lap[0] * inner(f, FD)
        for k in range(1, FD + 1):
            t = t + lap[k] * sum(shifted(f, ax, s * k, FD) for ax in range(3) for s in (-1, 1))
        return t * (-1 / (4 * math.pi))

    def grad(f, ax):
        return sum(gr[k] * (shifted(f, ax, k, FD) - shifted(f, ax, -k, FD)) for k in range(1, FD + 1))

    for r in range(loc.n_rep):
        t, bx = int(loc.rep_type[r]), [int(v) for v in loc.rep_box[r]]
        tab, Z, rc = tabs[t], float(loc.Z[t]), loc.rc_tilda
        ax = [torch.arange(bx[2 * k] - 2 * FD, bx[2 * k + 1] + 2 * FD + 1, device=dev, dtype=torch.float64) * h
              - float(loc.rep_xyz[r, k]) for k in range(3)]
        rad = torch.sqrt(ax[0][None, None, :] ** 2 + ax[1][None, :, None] ** 2 + ax[2][:, None, None] ** 2)
        V = _spline(tab, tab[1], tab[2], rad) / rad
        s = torch.minimum(rad, torch.full_like(rad, rc))
        poly = -Z * (9 * s ** 7 - 30 * rc * s ** 6 + 28 * rc ** 2 * s ** 5 - 14 * rc ** 5 * s ** 2 + 12 * rc ** 7) / (5 * rc ** 8)
        Vt = torch.where(rad < rc, poly, -Z / rad)
        B, Bt = nlap(V), nlap(Vt)  # box + FD
        at = tuple(slice(bx[2 * k] - grid.pnode_s[k], bx[2 * k + 1] - grid.pnode_s[k] + 1) for k in (2, 1, 0))
        V0, Vt0, B0, Bt0 = inner(V, 2 * FD), inner(Vt, 2 * FD), inner(B, FD), inner(Bt, FD)
        rho = _spline(tab, tab[3], tab[4], inner(rad, 2 * FD))
        b[at] += B0
        bt[at] += Bt0
        vc[at] += Vt0 - V0
        ra[at] += rho
        scal += torch.stack([0.5 * (B0 * V0).sum(), B0.sum(), rho.sum(), Bt0.sum(), 0.5 * (Bt0 * Vt0).sum()]) * h3
        ph = phi[tuple(slice(x.start + FD, x.stop + FD) for x in at)]
        bs, vg = bf[at] + btf[at], vcf[at]
        a = int(loc.rep_atom[r])
        Vi, Vti = inner(V, FD), inner(Vt, FD)
        for k in range(3):
            d = 2 - k
            Db, Dbt, DV, DVt = grad(B, d), grad(Bt, d), grad(Vi, d), grad(Vti, d)
            floc[a, k] += (Db * (ph - V0)).sum() * h3
            fcorr[a, k] += 0.5 * (Dbt * (vg - Vt0) + Db * (vg + V0) + (DVt - DV) * bs + B0 * DV - Bt0 * DVt).sum() * h3
    S = [float(x) for x in scal]
    v0 = float(vc[0, 0, 0]) if tuple(grid.pnode_s) == (0, 0, 0) else 0.0
    bt *= abs(S[1] / S[3])
    ecorr = float(0.5 * ((bt + b) * vc).sum()) * h3
    npy = lambda x: x.cpu().numpy()
    return _arrays(dict(b=npy(b), b_tilda=npy(bt), vc=npy(vc), rho_at=npy(ra), Eself=S[0], Ncharge=S[1],
                        Nelectron_at=S[2], Ncharge_tilda=S[3], Eself_tilda=S[4], Vcon=v0, Ecorr=ecorr + S[0] - S[4],
                        floc=npy(floc), fcorr=npy(fcorr)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "local":
        return _exact_local(case, seed)
    c = _case(case, seed)
    if kind == "projectors":
        return _exact_projectors(c)
    if kind == "sq":
        return _exact_sq(case, c)
    if kind == "forces":
        return _exact_forces(c, seed)
    return _exact_vjp(c, seed)
