"""The measured work of this framework: what its users have it compute, over the sizes they use.

Every case is one periodic box (or a list of boxes) taken through a public entry point:

* ``calculator``: ``FourierD3ASECalculator.calculate`` on host data, as an ASE script calls it;
* ``functional``: ``D3Model`` on device positions, as a molecular-dynamics program on the GPU calls it;
* ``module``: ``FourierD3.forward`` on a caller's edge list with gradients from autograd through the
  strain protocol, as a machine-learned force field that adds dispersion calls it;
* ``batch``: ``D3Batch`` with a captured graph, as a data set or a long simulation is evaluated;
* ``neighbours``: ``neighbour_list``, as a program that keeps its own edge list calls it.

Sizes, densities, elements and options are those of the repository's configurations, tests and
benchmark: SiO2 at 2.2 g/cm^3 from 648 to 139,968 atoms, HCNO at 1.3 g/cm^3 in triclinic cells,
ragged batches of Z = 1..54, spline orders 4-6, mesh spacings 1.0-1.2 A, SPME, PME, Ewald and the
k-space coordination number. Cells and elements belong to the case (they are what a plan is made
for); the positions come from the seed.

The ``mixed`` form computes its mesh in float32 and serves programs that work in float32 (the module
then takes and returns float32 itself); the functional and batch results of that form are therefore
handed on in float32. The ``fp64`` form is handed on as it is.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from fourierd3_b200 import D3Model, FourierD3, FourierD3ASECalculator, engine, structures
from fourierd3_b200.batch import D3Batch

DEV = "cuda"
A2B = 1 / 0.52917726
HA = 27.21138505
R_CUT = 6.0
DENSITY = {"sio2": 2.2, "hcno": 1.3, "z54": 2.0}
#: cells (lengths relative to the first, angles in degrees), by name
SHAPES = {"cubic": (1.0, 1.0, 90.0, 90.0, 90.0), "slab": (1.0, 0.5, 90.0, 90.0, 90.0),
          "triclinic": (1.0, 1.0, 84.0, 97.0, 92.0), "rod": (0.8, 1.7, 90.0, 103.0, 90.0)}


def _case(surface, chem, atoms, *, shape="cubic", precision="fp64", method="spme", order=5, spacing=1.2,
          cnfunc="smooth_cut", boxes=1, name=None):
    c = dict(surface=surface, chem=chem, atoms=atoms, shape=shape, precision=precision, method=method, order=order,
             spacing=spacing, cnfunc=cnfunc, boxes=boxes)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the smallest call: a molecular crystal's cell in a script's inner loop (latency and launches)
        _case("functional", "hcno", 14, shape="triclinic", order=4, name="molecule_14_fp64"),
        # the ordinary ASE call on a small box, from host arrays to host arrays
        _case("calculator", "sio2", 648, name="calculator_648_fp64"),
        # one ordinary box in a GPU program's loop, mixed precision
        _case("functional", "sio2", 5184, precision="mixed", name="sio2_5184_mixed"),
        # organic liquid in a triclinic cell: four elements, sixth order, finer mesh
        _case("functional", "hcno", 12000, shape="triclinic", precision="mixed", order=6, spacing=1.0,
              name="hcno_12000_mixed"),
        # the benchmark's box in its mixed form, replayed as a graph over a long simulation
        _case("batch", "sio2", 139968, precision="mixed", name="sio2_139968_mixed_graph"),
        # the same box in the plain form that a float64 study takes (the largest case)
        _case("functional", "sio2", 139968, name="sio2_139968_fp64"),
        # dispersion added to a float32 force field on its own edges (the molecular-dynamics box)
        _case("module", "sio2", 20736, shape="slab", precision="mixed", name="module_20736_mixed"),
        # the same with a float64 force field, Lagrange interpolation
        _case("module", "hcno", 2500, shape="triclinic", method="pme", order=6, name="module_pme_2500_fp64"),
        # a ragged batch of many elements: a data set is labelled
        _case("batch", "z54", 400, precision="mixed", boxes=12, name="ragged_12_mixed"),
        # direct k-space sum of a small box
        _case("functional", "hcno", 240, method="ewald", name="ewald_240_fp64"),
        # k-space coordination number, no neighbour search
        _case("functional", "hcno", 2592, shape="rod", cnfunc="d4", name="kspace_cn_2592_fp64"),
        # the edge list of a large box, for a force field that keeps its own
        _case("neighbours", "sio2", 41472, name="neighbours_41472"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes log-uniform (odd ones among them), shapes, forms and
    options at random; the atom count is cut where a box would cost more than the largest listed one of
its kind (Ewald sums, boxes of many elements, the rest)."""
    surface = rng.choice(["calculator", "functional", "functional", "functional", "module", "module", "batch",
                          "batch", "neighbours"])
    shape = rng.choice(list(SHAPES))
    precision = rng.choice(["fp64", "mixed"]) if surface != "calculator" else "fp64"
    order, spacing = rng.choice([4, 5, 6]), rng.choice([1.0, 1.1, 1.2])
    if surface == "batch" and rng.random() < 0.5:
        c = _case(surface, "z54", _log(rng, 60, 400), shape=shape, precision="mixed", order=order,
                  boxes=rng.randint(2, 10))
    elif surface == "neighbours":
        c = _case(surface, rng.choice(["sio2", "hcno"]), _log(rng, 600, 60000), shape=shape)
    else:
        chem = rng.choice(["sio2", "hcno"])
        method = rng.choice(["spme"] * 6 + ["pme"] * 2 + (["ewald"] if surface == "functional" else []))
        most = 500 if method == "ewald" else 139968 if chem == "sio2" and surface != "module" else 24000
        cnfunc = "d4" if method != "ewald" and surface == "functional" and rng.random() < 0.15 else "smooth_cut"
        c = _case(surface, chem, _log(rng, 10, most if surface != "calculator" else 6000), shape=shape,
                  precision=precision, method=method, order=order, spacing=spacing, cnfunc=cnfunc)
    alike = {(x["method"] == "ewald", x["chem"] == "z54"): _cost(x) for x in listed() if x["boxes"] > 1
             or x["method"] == "ewald" or x["atoms"] == 139968}
    while _cost(c) > alike[c["method"] == "ewald", c["chem"] == "z54"]:
        c["atoms"] = int(c["atoms"] / 1.5)
    return c


# ------------------------------------------------------------------ inputs
def _numbers(case, k):
    n, chem = _sizes(case)[k], case["chem"]
    rng = np.random.default_rng([k, n])
    if chem == "sio2":
        z = np.where(np.arange(n) < n // 3, 14, 8)
    elif chem == "hcno":
        z = np.repeat([1, 6, 7, 8], [n - (3 * n) // 10 - 2 * (n // 10), (3 * n) // 10, n // 10, n // 10])
    else:
        z = rng.integers(1, 55, n)
    return rng.permutation(z).astype(np.int64)


def _sizes(case):
    """Atom counts of the case's boxes: the largest first, then smaller and uneven ones."""
    return [max(8, int(case["atoms"] * (0.12 + 0.88 * ((k * 0.618) % 1.0 if k else 1.0)))) if k else case["atoms"]
            for k in range(case["boxes"])]


def _cell(case, k):
    b, c, al, be, ga = SHAPES[case["shape"]]
    unit = structures.cell_from_params(1.0, b, c, al, be, ga)
    z = _numbers(case, k)
    vol = np.linalg.det(structures.box_for_density(z, DENSITY[case["chem"]], (90.0, 90.0, 90.0)))
    return unit * (vol / np.linalg.det(unit)) ** (1.0 / 3.0)


def _positions(case, k, seed):
    """A disordered box: a random choice of the sites of a lattice with 1.25 sites per atom, each atom
    off its site by up to 0.15 of the site distance, in the lattice's order."""
    n, cell = _sizes(case)[k], _cell(case, k)
    rng = np.random.default_rng([seed % (1 << 31), k, n])
    if case["surface"] == "neighbours":   # one box moved through its cell: every seed has as many pairs
        at = _positions(dict(case, surface="functional"), k, 0) @ np.linalg.inv(cell) + rng.random(3)
        return (at - np.floor(at)) @ cell
    length = np.linalg.norm(cell, axis=1)
    m = np.maximum(1, np.floor(length * (1.25 * n / np.prod(length)) ** (1.0 / 3.0))).astype(int)
    while np.prod(m) < 1.1 * n:
        m[np.argmax(length / m)] += 1
    site = np.sort(rng.permutation(int(np.prod(m)))[:n])
    frac = (np.stack(np.unravel_index(site, m), 1) + rng.uniform(0.35, 0.65, (n, 3))) / m
    return frac @ cell


def _mesh(case, k):
    cell_b = _cell(case, k) * A2B
    if case["method"] == "ewald":
        return tuple(int(math.ceil(10.0 * v / (2 * math.pi))) for v in np.linalg.norm(cell_b, axis=1))
    v = 2.0 * np.linalg.norm(cell_b, axis=1) / (case["spacing"] * A2B) + 1.0
    return tuple(int(2 ** math.ceil(math.log2(x))) for x in v)


def _rank(case):
    return {"sio2": 4, "hcno": 5, "z54": 8}[case["chem"]]


def _cost(case):
    c = 0.0
    for k in range(case["boxes"]):
        s, m, n = len(np.unique(_numbers(case, k))), float(np.prod(_mesh(case, k))), _sizes(case)[k]
        if case["method"] == "ewald":
            c += 30.0 * n * m
        else:
            c += m * s * (_rank(case) + s / 2 + (4 if case["cnfunc"] == "d4" else 0)) + 300.0 * n
    return c * (2.0 if case["precision"] == "fp64" else 1.0)


def work(case):
    """Positions and elements read and energy, forces and stress written once; the operations of the
    transforms (5/2 M log2 M each way and channel), of the pair product at each k and of the stencils."""
    by = fl = 0.0
    b = 8 if case["precision"] == "fp64" else 4
    for k in range(case["boxes"]):
        n, m, s, r = _sizes(case)[k], float(np.prod(_mesh(case, k))), len(np.unique(_numbers(case, k))), _rank(case)
        pairs = n * 4.0 / 3.0 * math.pi * R_CUT ** 3 * n / abs(np.linalg.det(_cell(case, k)))
        if case["surface"] == "neighbours":
            by += 24.0 * n + 28.0 * pairs
            fl += 10.0 * pairs
            continue
        by += n * (24.0 + 4.0 + 3 * b) + 10 * b
        if case["surface"] == "module" and case["cnfunc"] != "d4":
            by += pairs * (16.0 + 3 * b)
        fl += 60.0 * pairs
        if case["method"] == "ewald":
            fl += n * m * (40.0 + 8.0 * r)
        else:
            fl += 5.0 * m * math.log2(max(m, 2)) * s * r + m / 2 * s * s * 4.0 * r + n * case["order"] ** 3 * 10.0 * r
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------ the calls
def _model_kw(case):
    return dict(method=case["method"], mesh_spacing=case["spacing"], interpolation_nodes=case["order"], r_cut=R_CUT)


def prepare(case, seed):
    pos, cell, z = _positions(case, 0, seed), _cell(case, 0), _numbers(case, 0)
    st = {"case": case, "cell": cell}
    kw = _model_kw(case)
    if case["surface"] == "calculator":
        st["calc"] = FourierD3ASECalculator(device=torch.device(DEV), dtype=torch.float64, cnfunc=case["cnfunc"], **kw)
        st["atoms"] = SimpleNamespace(numbers=z, positions=pos, cell=cell, pbc=(True, True, True))
        st["calc"]._build_model(st["atoms"])
    elif case["surface"] == "functional":
        st["model"] = D3Model(z, cell, precision=case["precision"], cnfunc=case["cnfunc"], device=torch.device(DEV),
                              **kw)
        st["pos"] = torch.tensor(pos, device=DEV)
    elif case["surface"] == "batch":
        boxes = [(_positions(case, k, seed), _cell(case, k), _numbers(case, k)) for k in range(case["boxes"])]
        st["model"] = D3Batch(boxes, precision=case["precision"], **kw)
        st["model"].capture()
        st["pos"] = torch.tensor(np.concatenate([p for p, _, _ in boxes]), device=DEV)
    elif case["surface"] == "module":
        dt = torch.float64 if case["precision"] == "fp64" else torch.float32
        st["model"] = FourierD3(z, cell, dtype=dt, device=torch.device(DEV), verbose=False, **kw)
        st["pos"] = torch.tensor(pos, dtype=dt, device=DEV)
        st["cell_t"] = torch.tensor(cell, dtype=dt, device=DEV)
        i, j, s = _pairs(torch.tensor(pos, device=DEV), torch.tensor(cell, device=DEV))
        order = torch.sort(i, stable=True).indices
        st["edges"], st["shifts"] = torch.stack((i, j))[:, order].contiguous(), s[order].to(dt)
    else:
        st["pos"] = torch.tensor(pos, device=DEV)
    return st


def run(st):
    case, surface = st["case"], st["case"]["surface"]
    if surface == "calculator":
        st["calc"].calculate(st["atoms"])
        r = st["calc"].results
        return r["energy"], r["forces"], r["stress"]
    if surface == "neighbours":
        return engine.neighbour_list(st["pos"], st["cell"], R_CUT)
    if surface == "module":
        model, cell = st["model"], st["cell_t"]
        strain = torch.zeros(3, 3, dtype=cell.dtype, device=DEV, requires_grad=True)
        scell = cell + cell @ strain.T
        pos = st["pos"].detach().requires_grad_(True)
        model._update_cell(scell)
        energy = model(pos + pos @ strain.T, st["edges"], st["shifts"] @ scell)
        gpos, gstrain = torch.autograd.grad(energy, (pos, strain))
        return energy.detach(), gpos, gstrain
    if surface == "functional":
        e, f, s = st["model"](st["pos"], st["cell"])
    else:
        e, f, s = st["model"](st["pos"])
    return (e, f, s) if case["precision"] == "fp64" else (e.float(), f.float(), s.float())


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _pairs(pos, cell):
    """(i, j, S) of every image pair closer than R_CUT, by bins of the fractional coordinates."""
    dev, n = pos.device, pos.shape[0]
    inv = torch.linalg.inv(cell)
    high = (1.0 / torch.linalg.norm(inv, dim=0)).tolist()
    nb = [max(1, int(h / R_CUT)) for h in high]
    reach = [math.ceil(R_CUT * b / h + 1e-9) for b, h in zip(nb, high)]
    frac = pos @ inv
    img = torch.floor(frac)
    nbt = torch.tensor(nb, device=dev)
    cell_of = torch.minimum(((frac - img) * nbt).long(), nbt - 1)
    key = (cell_of[:, 0] * nb[1] + cell_of[:, 1]) * nb[2] + cell_of[:, 2]
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=nb[0] * nb[1] * nb[2])
    start = torch.cumsum(count, 0) - count
    slot = torch.arange(int(count.max()), device=dev)
    out = []
    for a in range(-reach[0], reach[0] + 1):
        for b in range(-reach[1], reach[1] + 1):
            for c in range(-reach[2], reach[2] + 1):
                q = cell_of + torch.tensor([a, b, c], device=dev)
                wrap = torch.div(q, nbt, rounding_mode="floor")
                q = q - wrap * nbt
                k = (q[:, 0] * nb[1] + q[:, 1]) * nb[2] + q[:, 2]
                i, t = torch.nonzero(slot[None, :] < count[k][:, None], as_tuple=True)
                j = order[start[k[i]] + t]
                shift = wrap[i].to(pos.dtype) - img[j] + img[i]
                d = pos[j] - pos[i] + shift @ cell
                keep = ((d * d).sum(1) < R_CUT * R_CUT) & ~((i == j) & (shift == 0).all(1))
                out.append((i[keep], j[keep], shift[keep]))
    assert all(len(o[0]) <= n * 4096 for o in out)
    return tuple(torch.cat([o[q] for o in out]) for q in range(3))


def _spline(x, p, lagrange):
    if lagrange:
        t, w = x + 0.5 * (p - 1), []
        for k in range(p):
            f = torch.ones_like(x)
            for m in range(p):
                if m != k:
                    f = f * (t - m) / (k - m)
            w.append(f)
        return torch.stack(w, -1)
    a, v = 0.5 - x, [torch.ones_like(x)]
    for q in range(2, p + 1):
        v = [((a + j) * (v[j] if j < q - 1 else 0.0) + (q - a - j) * (v[j - 1] if j else 0.0)) / (q - 1)
             for j in range(q)]
    return torch.stack(v, -1)


def _green(k, qq, s6, s8, a1, a2):
    """Fourier transform of the damped -C6/r^6 - C8/r^8 pair term of each species pair, (nk, S, S)."""
    R = a1 * torch.sqrt(3.0 * qq) + a2
    small = k[:, None, None] * R < 1e-15
    ks = torch.where(small, torch.ones((), dtype=k.dtype, device=k.device), k[:, None, None])
    u = ks * R
    s, c = math.sin(math.pi / 8), math.cos(math.pi / 8)
    n6 = torch.exp(-u) - 2.0 * torch.exp(-0.5 * u) * torch.cos(math.pi / 3 + u * math.sqrt(3.0) / 2)
    n8 = torch.exp(-u * s) * torch.cos(math.pi / 4 + u * c) + torch.exp(-u * c) * torch.cos(3 * math.pi / 4 + u * s)
    g6 = torch.where(small, 2 * math.pi ** 2 / (3 * R ** 3), 2 * math.pi ** 2 / (3 * R ** 4) / ks * n6)
    g8 = torch.where(small, math.pi ** 2 * math.sqrt(2.0) * s / R ** 5, -math.pi ** 2 / R ** 6 / ks * n8)
    return s6 * g6 + 3.0 * s8 * qq * g8


def _energy(case, pos, cell, sp, setup, edges, shift):
    """The dispersion energy in Hartree of one box (Bohr), by the path's definition."""
    dev, dt = pos.device, torch.float64
    as_t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
    eigs, vq = as_t(setup.eigs), as_t(setup.eigvecs).view(setup.n_species, 7, -1)
    rcov, cnref, sq = as_t(setup.rcov), as_t(setup.cnref), as_t(setup.sqrtq)
    par = (1.0, 0.7875, 0.4289, 4.4407)
    S, n, rc = setup.n_species, pos.shape[0], R_CUT * A2B
    i, j = edges
    r = torch.linalg.norm(pos[j] - pos[i] + shift, dim=-1).clamp(min=1e-6)
    rcs = rcov[sp[i]] + rcov[sp[j]]
    r1 = 0.5 * rcs + 0.5 * rc
    co = torch.maximum(r, r1)
    kcn = 16.0 + (co - r1) ** 2 / ((rc - co) ** 2 + 1e-6)
    cn = torch.zeros(n, dtype=dt, device=dev).index_add(0, i, torch.sigmoid(kcn * (4.0 / 3.0 * rcs / r - 1.0)))
    ref = cnref[sp]
    w = torch.softmax((-4.0 * (cn[:, None] - ref) ** 2).masked_fill(ref == -1, -math.inf), 1)
    c6 = torch.einsum("nk,nkr->nr", w, vq[sp])
    qq = torch.outer(sq, sq)
    R = par[2] * torch.sqrt(3.0 * qq) + par[3]
    own = torch.diagonal(par[0] / R ** 6 + 3.0 * par[1] * qq / R ** 8)
    vol = torch.abs(torch.linalg.det(cell))
    e_self = 0.5 * (eigs * (c6 ** 2 * own[sp][:, None]).sum(0)).sum()
    rec = 2.0 * math.pi * torch.linalg.inv(cell).T
    ns = _mesh(case, case.get("box", 0))
    f = lambda m, half: (torch.fft.rfftfreq if half else torch.fft.fftfreq)(m, 1.0 / m, device=dev, dtype=dt)  # noqa: E731
    ewald = case["method"] == "ewald"
    grid = torch.stack(torch.meshgrid(f(ns[0], 0), f(ns[1], 0), f(ns[2], not ewald), indexing="ij"), -1).view(-1, 3)

    if ewald:
        def part(g, rec, pos, c6):
            k = g @ rec
            ph = k @ pos.T
            amp = torch.zeros(S, n, c6.shape[1], dtype=dt, device=dev)
            amp = amp.index_put((sp, torch.arange(n, device=dev)), c6 * torch.sqrt(torch.abs(eigs)))
            G = _green(torch.linalg.norm(k, dim=1), qq, *par)
            e = 0.0
            for t in (torch.cos(ph), torch.sin(ph)):
                s = torch.einsum("kn,anr->kar", t, amp)
                e = e + torch.einsum("kab,kar,kbr->", G, s, s)
            return e

        ek = sum(checkpoint(part, g, rec, pos, c6, use_reentrant=False) for g in grid.split(4096))
        return e_self - ek / (2.0 * vol)

    p = case["order"]
    nst = torch.tensor(ns, device=dev)
    u = nst * (pos @ torch.linalg.inv(cell))
    node = (torch.round(u) if p % 2 else torch.floor(u)).detach()
    ww = _spline(u - node - (0.0 if p % 2 else 0.5), p, case["method"] == "pme")
    at = (node.long()[:, :, None] + torch.arange(p, device=dev) + 1 - (p + 1) // 2) % nst[:, None]
    lin = ((at[:, 0, :, None, None] * ns[1] + at[:, 1, None, :, None]) * ns[2] + at[:, 2, None, None, :]).view(n, -1)
    wg = (ww[:, 0, :, None, None] * ww[:, 1, None, :, None] * ww[:, 2, None, None, :]).reshape(n, -1)
    M = ns[0] * ns[1] * ns[2]
    spec = []
    for q in range(c6.shape[1]):
        rho = torch.zeros(S * M, dtype=dt, device=dev)
        rho = rho.index_add(0, (lin + sp[:, None] * M).view(-1), (wg * c6[:, q:q + 1]).view(-1))
        spec.append(torch.fft.rfftn(rho.view(S, *ns), dim=(1, 2, 3)).view(S, -1))
    her = torch.full((ns[2] // 2 + 1,), 2.0, dtype=dt, device=dev)
    her[0] = her[-1] = 1.0
    her = her.repeat(ns[0] * ns[1])
    if case["method"] == "spme":   # the deconvolution window is a float32 table by definition
        a = [torch.sinc(f(m, h).float().cpu() / m) for m, h in zip(ns, (0, 0, 1))]
        win = torch.pow(a[0][:, None, None] * a[1][None, :, None] * a[2][None, None, :], 2 * p)
        her = her / torch.where(win < 1e-10, 1e-10, win).to(dev).to(dt).view(-1)

    def slab(lo, hi, rec, *spec):
        G = _green(torch.linalg.norm(grid[lo:hi] @ rec, dim=1), qq, *par) * her[lo:hi, None, None]
        e = 0.0
        for q, s in enumerate(spec):
            t = torch.view_as_real(s[:, lo:hi])
            e = e + eigs[q] * torch.einsum("kab,akc,bkc->", G, t, t)
        return e

    step = max(1, (1 << 27) // (S * S))
    ek = sum(checkpoint(slab, lo, min(lo + step, len(grid)), rec, *spec, use_reentrant=False)
             for lo in range(0, len(grid), step))
    return e_self - ek / (2.0 * vol)


def exact(case, seed):
    if case["surface"] == "neighbours" or case["cnfunc"] == "d4":
        return None
    es, fs, ss = [], [], []
    for k in range(case["boxes"]):
        pos = torch.tensor(_positions(case, k, seed), device=DEV)
        cell = torch.tensor(_cell(case, k), device=DEV)
        ei, ej, image = _pairs(pos, cell)
        if case["surface"] == "module" and case["precision"] == "mixed":
            pos, cell = pos.float().double(), cell.float().double()
        setup = engine.species_setup(_numbers(case, k), 1.0)   # the element tables and the rank-r C6 factors
        sp = torch.tensor(setup.species.astype(np.int64), device=DEV)
        strain = torch.zeros(3, 3, dtype=torch.float64, device=DEV, requires_grad=True)
        x = pos.clone().requires_grad_(True)
        scell = cell + cell @ strain.T
        e = _energy(dict(case, box=k), (x + x @ strain.T) * A2B, scell * A2B, sp, setup, (ei, ej),
                    (image @ scell) * A2B)
        gx, gs = torch.autograd.grad(e, (x, strain))
        vol = abs(float(torch.linalg.det(cell)))
        module = case["surface"] == "module"
        es.append(e.detach() * (1.0 if module else HA))
        fs.append(gx if module else -gx * HA)
        ss.append(gs if module else gs * HA / vol)
    if case["surface"] == "batch":
        return torch.stack(es), torch.cat(fs), torch.stack(ss)
    return (float(es[0]) if case["surface"] == "calculator" else es[0]), fs[0], ss[0]


