"""The work that users of this framework have it do, as timed cases.

Every case is one pass through public entry points of ``torchff_b200`` on synthetic TIP3P
water boxes (or, for ``pme``, the random charges of a PME benchmark). Kinds:

* ``md``: one molecular-dynamics force evaluation. The program keeps a ``FixedChargeSystem``
  and its buffers, captures ``evaluate_into`` once in a CUDA graph and replays it per step.
* ``eval``: the same evaluation called eagerly (``FixedChargeSystem.evaluate`` with the energy
  terms), as a script or a Monte-Carlo move does; rigid or flexible waters, orthorhombic or
  sheared boxes.
* ``train``: one frame of force matching: energy, forces with ``create_graph``, the loss on the
  forces and its double backward to per-atom charges, sigma and epsilon.
* ``ops``: the model composed from the drop-in operators, as code written for the operator API
  calls them: neighbour list, Lennard-Jones over type tables, real-space Ewald with exclusion
  correction, PME, backward to forces.
* ``pairs``: shifted Coulomb + Lennard-Jones over a neighbour list that the program holds for
  several steps, energy and gradients (forces alone, or parameter gradients too). The call's
  cutoff is 0.1 % longer than the list's, so that every held pair counts: the force of the
  shifted potential jumps at its cutoff, and which side of it a pair falls on would be a matter
  of rounding.
* ``pme``: reciprocal-space energy with gradients for coordinates and charges.
* ``batch``: many periodic systems of uneven size in one ``BatchEvaluator`` call on packed
  device buffers (replica ensembles, batched torch-sim states).
* ``server``: a burst of host requests through the continuous-batching ``Server``.

``exact`` evaluates the same expressions in float64 with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "torchff-lib_b200"))

import torchff_b200 as tff  # noqa: E402
from torchff_b200 import water as W  # noqa: E402
from torchff_b200.nonbonded import compute_nonbonded_energy_from_atom_pairs  # noqa: E402
from torchff_b200.serving import BatchEvaluator, Server, SystemSpec  # noqa: E402
from torchff_b200.system import FixedChargeNonbonded, FixedChargeSystem  # noqa: E402

KC = W.COULOMB_PREFACTOR
DENSITY = 33.4        # waters per nm^3
PAIR_FLOPS = 60.0     # per pair within the cutoff: LJ + erfc Coulomb, energy and forces
DTYPES = {"f32": torch.float32, "f64": torch.float64}
PAIRS_ROOM = 1.001     # call cutoff / list cutoff of a held list
PME_ALPHA = 0.2653    # 1/length unit of the random-charge PME benchmark, edge (10 N)^(1/3)


def listed():
    return [
        # the smallest box of the tests and configurations: launches and latency count
        {"name": "md_216_f32", "kind": "md", "waters": 216, "grid": 20, "dtype": "f32"},
        # the headline benchmark: 3000 waters, mixed precision
        {"name": "md_3000_f32", "kind": "md", "waters": 3000, "grid": 48, "dtype": "f32"},
        # the same box in double precision
        {"name": "md_3000_f64", "kind": "md", "waters": 3000, "grid": 48, "dtype": "f64"},
        # the large box of the configurations: 300,000 atoms
        {"name": "md_100k_f32", "kind": "md", "waters": 100000, "grid": 144, "dtype": "f32"},
        # eager calls on an odd-sized flexible system (bonds and angles in the evaluation)
        {"name": "eval_1231_flex_f32", "kind": "eval", "waters": 1231, "grid": 34, "dtype": "f32", "flexible": True,
         "sheared": False},
        # force matching on the 3000-water box
        {"name": "train_3000_f32", "kind": "train", "waters": 3000, "grid": 48, "dtype": "f32"},
        # operator API, mixed precision, cell list
        {"name": "ops_3000_f32", "kind": "ops", "waters": 3000, "grid": 48, "dtype": "f32", "algorithm": "cell_list"},
        # operator API, double precision, all-pairs list: the small validation box
        {"name": "ops_216_f64", "kind": "ops", "waters": 216, "grid": 20, "dtype": "f64", "algorithm": "nsquared"},
        # a held neighbour list of a large box (20 million pairs)
        {"name": "pairs_33k_f32", "kind": "pairs", "waters": 33000, "dtype": "f32", "params": False},
        # the reference's published PME benchmark: double precision, 30,000 random charges
        {"name": "pme_30000_f64", "kind": "pme", "charges": 30000, "grid": 48, "dtype": "f64"},
        # 60 systems of 64 to 4000 waters, device buffers
        {"name": "batch_60_f32", "kind": "batch", "systems": 60, "most": 4000, "dtype": "f32"},
        # a burst of 60 host requests of the same sizes
        {"name": "server_60_f32", "kind": "server", "systems": 60, "most": 4000, "dtype": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(n):
    return max(6, math.ceil(_edge(n) / 0.1))


def draw(rng):
    kind = rng.choice(["md", "md", "eval", "train", "ops", "pairs", "pme", "batch", "server"])
    dtype = "f64" if rng.random() < 0.35 else "f32"
    if kind == "md":
        n = _log(rng, 64, 40000 if dtype == "f32" else 10000)
        return {"kind": kind, "waters": n, "grid": _grid(n), "dtype": dtype}
    if kind == "eval":
        n = _log(rng, 64, 2000)
        return {"kind": kind, "waters": n, "grid": _grid(n), "dtype": dtype, "flexible": rng.random() < 0.5,
                "sheared": rng.random() < 0.3}
    if kind == "train":
        n = _log(rng, 64, 3000)
        return {"kind": kind, "waters": n, "grid": _grid(n), "dtype": dtype}
    if kind == "ops":
        n = _log(rng, 64, 6000)
        return {"kind": kind, "waters": n, "grid": _grid(n), "dtype": dtype,
                "algorithm": "cell_list" if n > 600 or rng.random() < 0.5 else "nsquared"}
    if kind == "pairs":
        return {"kind": kind, "waters": _log(rng, 216, 20000 if dtype == "f32" else 6000), "dtype": dtype,
                "params": rng.random() < 0.5}
    if kind == "pme":
        return {"kind": kind, "charges": _log(rng, 300, 100000), "grid": rng.randint(16, 49), "dtype": dtype}
    return {"kind": kind, "systems": rng.randint(4, 48), "most": _log(rng, 300, 4000), "dtype": "f32"}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _edge(n):
    return (n / DENSITY) ** (1.0 / 3.0)


def _cutoff(case):
    return 0.9 if case.get("waters", 0) < 1000 else 1.0


def _shear(case, edge):
    box = np.eye(3) * edge
    if case.get("sheared"):
        box[1, 0], box[2, 0], box[2, 1] = 0.12 * edge, -0.08 * edge, 0.1 * edge
    return box


def _water(case, seed):
    n = case["waters"]
    wb = W.make_water_box(n, _edge(n), math.ceil(n ** (1.0 / 3.0) - 1e-9), _cutoff(case), case.get("grid", 6), seed=seed)
    if case.get("sheared"):  # the lattice sites move with the box, the molecules stay rigid
        box = _shear(case, _edge(n))
        o = np.repeat(wb.coords[0::3], 3, axis=0)
        wb.coords, wb.box = wb.coords - o + o @ (box / _edge(n)), box
    if case.get("flexible"):
        wb.coords = wb.coords + np.random.default_rng(seed + 1).normal(0.0, 0.002, wb.coords.shape)
    return wb


def _train_inputs(case, seed):
    wb = _water(case, seed)
    q, s, e = W.force_matching_parameters(wb, seed)
    target = np.random.default_rng(seed + 2).normal(0.0, 300.0, wb.coords.shape)
    return wb, q, s, e, target


def _pme_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["charges"]
    edge = (10.0 * n) ** (1.0 / 3.0)
    q = rng.standard_normal(n)
    return rng.uniform(0.0, edge, (n, 3)), np.eye(3) * edge, q - q.mean()


def _serving(case, seed):
    # log-uniform sizes from 64 waters to `most`, in an order that mixes large and small ones
    ns = np.random.default_rng(7).permutation(np.exp(np.linspace(math.log(64), math.log(case["most"]), case["systems"])))
    return [W.serving_water_box(int(round(n)), seed=seed * 1009 + k) for k, n in enumerate(ns)]


def _capacity(natoms, cutoff):
    """Rows for a neighbour list at water density with 20 % room, as a program sizes it."""
    return int(natoms * 4.0 / 3.0 * math.pi * cutoff ** 3 * 3 * DENSITY / 2 * 1.2) + 64


def prepare(case, seed):
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    dev = torch.device("cuda")
    on = lambda a, t=dt, g=False: torch.tensor(np.ascontiguousarray(a), dtype=t, device=dev).requires_grad_(g)  # noqa: E731
    st = {"kind": kind}
    if kind in ("md", "eval"):
        wb = _water(case, seed)
        sy = FixedChargeSystem.from_water_box(wb, dtype=dt, device=dev, flexible=bool(case.get("flexible")))
        st.update(system=sy, x=on(wb.coords), box=on(wb.box))
        if kind == "md":
            st["out"] = {"energy": torch.zeros(1, dtype=torch.float64, device=dev), "forces": torch.zeros_like(st["x"]),
                         "terms": torch.zeros(4, dtype=torch.float64, device=dev)}
            o = st["out"]
            step = lambda: sy.evaluate_into(st["x"], st["box"], o["energy"], o["forces"], None, o["terms"])  # noqa: E731
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                step()
            torch.cuda.current_stream().wait_stream(side)
            st["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(st["graph"]):
                step()
            for t in o.values():
                t.zero_()
    elif kind == "train":
        wb, q, s, e, target = _train_inputs(case, seed)
        sy = FixedChargeSystem(q, s, e, wb.coulomb_exclusions, wb.cutoff, wb.alpha, wb.grid, dtype=dt, device=dev)
        st.update(model=FixedChargeNonbonded(sy), x=on(wb.coords, g=True), box=on(wb.box), target=on(target),
                  params=[on(a, g=True) for a in (q, s, e)])
    elif kind == "ops":
        wb = _water(case, seed)
        st.update(nbl=tff.NeighborList(wb.natoms, exclusions=torch.tensor(wb.nblist_exclusions),
                                       algorithm=case["algorithm"]).to(dev),
                  lj=tff.Vdw("LennardJones", use_customized_ops=True, use_type_pairs=True).to(dev),
                  coul=tff.MultipolarInteraction(0, wb.cutoff, wb.alpha, KC).to(dev),
                  pme=tff.PME(wb.alpha, wb.grid, 0, use_customized_ops=True).to(dev, dt),
                  x=on(wb.coords, g=True), box=on(wb.box), q=on(wb.charges), sig=on(wb.sigma_table),
                  eps=on(wb.epsilon_table), types=on(wb.atom_types, torch.int64),
                  excl=on(wb.coulomb_exclusions, torch.int64), cutoff=wb.cutoff,
                  cap=_capacity(wb.natoms, wb.cutoff))
    elif kind == "pairs":
        wb = _water(case, seed)
        x, box = on(wb.coords, g=True), on(wb.box)
        nbl = tff.NeighborList(wb.natoms, exclusions=torch.tensor(wb.nblist_exclusions),
                               algorithm="cell_list" if wb.natoms > 2000 else "nsquared").to(dev)
        p = bool(case["params"])
        st.update(x=x, box=box, cutoff=wb.cutoff, params=[on(a, g=p) for a in (wb.sigma, wb.epsilon, wb.charges)],
                  pairs=nbl(x.detach(), box, wb.cutoff, _capacity(wb.natoms, wb.cutoff)).clone())
    elif kind == "pme":
        x, box, q = _pme_inputs(case, seed)
        st.update(pme=tff.PME(PME_ALPHA, case["grid"], 0, use_customized_ops=True).to(dev, dt), x=on(x, g=True),
                  box=on(box), q=on(q, g=True))
    elif kind == "batch":
        boxes = _serving(case, seed)
        specs = [SystemSpec.from_water_box(b) for b in boxes]
        ev = BatchEvaluator(boxes[0].cutoff, boxes[0].alpha, dt, max_systems=len(specs),
                            max_atoms=sum(s.natoms for s in specs), max_grid_points=sum(s.pme_grid ** 3 for s in specs))
        st.update(ev=ev, packed=ev.pack(specs))
    else:
        boxes = _serving(case, seed)
        st.update(server=Server(boxes[0].cutoff, boxes[0].alpha, dt, lanes=4, max_systems_per_batch=64,
                                hbm_budget_bytes=3 << 30, grid_points_per_atom=12.0),
                  requests=[Server.prepare(SystemSpec.from_water_box(b)) for b in boxes])
    return st


# ---------------------------------------------------------------------------------------
# one pass. Of `md` and `eval` the energy comes back as its terms (real-space pairs, exclusion
# correction, reciprocal, self, bonds, angles): their sum cancels to a value near zero for some
# boxes, where a relative difference says nothing.
# ---------------------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "md":
        st["graph"].replay()
        return {"forces": st["out"]["forces"], "terms": st["out"]["terms"]}
    if kind == "eval":
        out = st["system"].evaluate(st["x"], st["box"], terms=True)
        return {"forces": out["forces"], "terms": out["terms"]}
    if kind == "train":
        for p in st["params"]:
            p.grad = None
        e = st["model"](st["x"], st["box"], *st["params"])
        (gx,) = torch.autograd.grad(e, st["x"], create_graph=True)
        loss = torch.mean((-gx - st["target"]) ** 2)
        loss.backward(inputs=st["params"])
        q, s, eps = st["params"]
        return {"loss": loss.detach(), "forces": -gx.detach(), "charges": q.grad, "sigma": s.grad, "epsilon": eps.grad}
    if kind == "ops":
        x, box = st["x"], st["box"]
        x.grad = None
        pairs, npairs = st["nbl"](x.detach(), box, st["cutoff"], st["cap"], padding=True)
        lj = st["lj"](x, pairs, box, st["sig"], st["eps"], st["cutoff"], atom_types=st["types"])
        coul = st["coul"](x, box, pairs, st["q"], pairs_excl=st["excl"])
        rec = st["pme"](x, box, st["q"]) * KC
        (lj + coul + rec).backward()
        return {"lj": lj.detach(), "coulomb": coul.detach(), "pme": rec.detach(), "gradient": x.grad, "npairs": npairs}
    if kind == "pairs":
        st["x"].grad = None
        for p in st["params"]:
            p.grad = None
        sig, eps, q = st["params"]
        e = compute_nonbonded_energy_from_atom_pairs(st["x"], st["pairs"], st["box"], sig, eps, q, KC,
                                                     PAIRS_ROOM * st["cutoff"], True)
        e.backward()
        return {"energy": e.detach(), "gradient": st["x"].grad, "sigma": sig.grad, "epsilon": eps.grad, "charges": q.grad}
    if kind == "pme":
        st["x"].grad = st["q"].grad = None
        e = st["pme"](st["x"], st["box"], st["q"])
        e.backward()
        return {"energy": e.detach(), "gradient": st["x"].grad, "charges": st["q"].grad}
    if kind == "batch":
        st["ev"].evaluate_packed(st["packed"])
        return {"energies": st["packed"]["energies"], "forces": st["packed"]["forces"]}
    reqs = [st["server"].submit(r) for r in st["requests"]]
    got = [r.wait() for r in reqs]
    for r in reqs:
        r.release()
    return {"energies": np.array([g[0] for g in got]), "forces": [g[1] for g in got]}


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _model_work(natoms, cutoff, grid, size, passes=1.0):
    pairs = natoms * 4.0 / 3.0 * math.pi * cutoff ** 3 * 3 * DENSITY / 2
    fft = 2 * 2.5 * grid ** 3 * math.log2(grid ** 3)
    return {"bytes": natoms * (9.0 * size + 8.0) * passes,  # coordinates, q, sigma, eps, exclusions in; forces out
            "flops": (PAIR_FLOPS * pairs + fft + 12.0 * grid ** 3 + natoms * 216 * 10.0) * passes}


def work(case):
    kind, size = case["kind"], 4 if case["dtype"] == "f32" else 8
    if kind in ("md", "eval", "ops"):
        return _model_work(3 * case["waters"], _cutoff(case), case["grid"], size)
    if kind == "train":  # the evaluation with parameter gradients, then a Hessian-vector product
        return _model_work(3 * case["waters"], _cutoff(case), case["grid"], size, 2.5)
    if kind == "pairs":
        n, rc = 3 * case["waters"], _cutoff(case)
        pairs = n * 4.0 / 3.0 * math.pi * rc ** 3 * 3 * DENSITY / 2
        return {"bytes": pairs * 16.0 + n * (12.0 if case["params"] else 9.0) * size, "flops": 35.0 * pairs}
    if kind == "pme":
        n, k = case["charges"], case["grid"]
        return {"bytes": n * 8.0 * size, "flops": 5.0 * k ** 3 * math.log2(k ** 3) + 12.0 * k ** 3 + n * 216 * 10.0}
    mean = (case["most"] - 64) / math.log(case["most"] / 64.0)  # waters per system
    one = _model_work(3 * mean, 0.9, math.ceil(_edge(mean) / 0.1), 8 if kind == "server" else size)
    return {k: v * case["systems"] for k, v in one.items()}


def tolerance(case):
    """About four times the error against float64 over the range: forces in mixed precision are
    up to 5e-6 off (erfc to 1.5e-7, FP32 coordinates of a 14 nm box), Hessian-vector products
    7e-6, the total energy of a held pair list 1e-5 (it cancels); FP64 sums differ by 1e-14 to
    1e-13 with their order."""
    if case["dtype"] == "f64":
        return {"rel": 1e-11}
    if case["kind"] == "pme":
        return {"rel": 5e-6}
    return {"rel": 5e-5 if case["kind"] == "pairs" else 3e-5}


# ---------------------------------------------------------------------------------------
# the same in float64 with plain torch
# ---------------------------------------------------------------------------------------
def _rounded(a, dtype):
    return torch.tensor(np.asarray(a), dtype=dtype).to("cuda", torch.float64)


def _image(d, box):
    s = d @ torch.linalg.inv(box)
    return (s - torch.floor(s + 0.5)) @ box


def _pair_list(x, box, rc):
    """(i, j) of every pair of different molecules (3 consecutive atoms) within rc."""
    n, edge = x.shape[0], float(box[0, 0])
    cells = int(edge / rc)
    ortho = bool(torch.count_nonzero(box - torch.diag(torch.diagonal(box))) == 0)
    found = []

    def keep(i, j):
        other = i // 3 != j // 3
        found.append((i[other], j[other]))

    if cells < 4 or not ortho:
        for lo in range(0, n, 1024):
            i = torch.arange(lo, min(lo + 1024, n), device=x.device)
            d = _image(x[i][:, None] - x[None], box)
            a, b = torch.nonzero((d * d).sum(-1) <= rc * rc, as_tuple=True)
            keep(i[a][i[a] > b], b[i[a] > b])
    else:
        c = torch.clamp((x / edge - torch.floor(x / edge)) * cells, max=cells - 1).long()
        cell = (c[:, 0] * cells + c[:, 1]) * cells + c[:, 2]
        order = torch.argsort(cell)
        count = torch.bincount(cell, minlength=cells ** 3)
        first = torch.cumsum(count, 0) - count
        most = int(count.max())
        slot = torch.arange(most, device=x.device)
        table = torch.where(slot < count[:, None], order[torch.clamp(first[:, None] + slot, max=n - 1)], -1)
        grid = table.view(cells, cells, cells, most)
        half = [(a, b, c) for a in (0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) >= (0, 0, 0)]
        for k in range(14):  # the cell itself and one of each two opposite neighbours
            other = torch.roll(grid, [-o for o in half[k]], dims=(0, 1, 2)).reshape(-1, most)
            for lo in range(0, cells ** 3, 512):
                i, j = table[lo:lo + 512, :, None], other[lo:lo + 512, None, :]
                ok = (i >= 0) & (j >= 0)
                ok = ok & (i > j) if k == 0 else ok
                i, j = i.expand_as(ok)[ok], j.expand_as(ok)[ok]
                d = _image(x[i] - x[j], box)
                near = (d * d).sum(-1) <= rc * rc
                keep(i[near], j[near])
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _splines(w):
    """(..., 6): M6(w + k), k = 0..5."""
    m = [w, 1.0 - w]
    for n in range(3, 7):
        prev, new = torch.zeros_like(w), []
        for k in range(n):
            cur = m[k] if k < n - 1 else torch.zeros_like(w)
            new.append(((w + k) * cur + (n - w - k) * prev) / (n - 1))
            prev = cur
        m = new
    return torch.stack(m, -1)


def _reciprocal(x, box, q, alpha, K):
    """Smooth PME of order 6, reciprocal part, in units without the Coulomb constant."""
    inv = torch.linalg.inv(box)
    u = K * (x @ inv)
    m0 = torch.ceil(u.detach())
    th = _splines(m0 - u)
    g = ((m0.long()[..., None] - 3 + torch.arange(6, device=x.device)) % K)
    at = ((g[:, 0, :, None, None] * K + g[:, 1, None, :, None]) * K + g[:, 2, None, None, :]).reshape(-1)
    wt = q[:, None, None, None] * th[:, 0, :, None, None] * th[:, 1, None, :, None] * th[:, 2, None, None, :]
    grid = torch.zeros(K ** 3, dtype=x.dtype, device=x.device).index_add(0, at, wt.reshape(-1)).view(K, K, K)
    s = torch.fft.rfftn(grid)
    m6 = _splines(torch.zeros((), dtype=x.dtype, device=x.device))
    k = torch.arange(K, device=x.device, dtype=x.dtype)
    mod = sum(m6[m + 3] * torch.cos(2.0 * math.pi * m * k / K) for m in range(-3, 3))
    f = torch.where(2 * k < K, k, k - K)
    kz = K // 2 + 1
    mv = torch.stack(torch.meshgrid(f, f, f[:kz], indexing="ij"), -1)
    k2 = ((2.0 * math.pi * mv @ inv.T) ** 2).sum(-1)
    k2[0, 0, 0] = 1.0
    theta = mod[:, None, None] * mod[None, :, None] * mod[None, None, :kz]
    c = 4.0 * math.pi / torch.abs(torch.linalg.det(box)) * torch.exp(-k2 / (4.0 * alpha ** 2)) / (k2 * theta ** 2)
    c[0, 0, 0] = 0.0
    twice = torch.full((kz,), 2.0, dtype=x.dtype, device=x.device)
    twice[0] = 1.0
    if K % 2 == 0:
        twice[-1] = 1.0
    return 0.5 * (twice * c * (s.real ** 2 + s.imag ** 2)).sum()


def _lj(r2, sig, eps):
    sr6 = (sig * sig / r2) ** 3
    return (4.0 * eps * sr6 * (sr6 - 1.0)).sum()


def _terms(x, box, q, sig, root, rc, alpha, K):
    """Lennard-Jones, real-space Coulomb, exclusion correction, reciprocal and self energy of
    rigid-water exclusions; root = sqrt(epsilon). One entry each, differentiable twice."""
    i, j = _pair_list(x.detach(), box, rc)
    d = _image(x[i] - x[j], box)
    r2 = (d * d).sum(-1)
    r = torch.sqrt(r2)
    lj = _lj(r2, 0.5 * (sig[i] + sig[j]), root[i] * root[j])
    real = (KC * q[i] * q[j] * torch.erfc(alpha * r) / r).sum()
    o = torch.arange(0, x.shape[0], 3, device=x.device)
    a, b = torch.cat([o, o, o + 1]), torch.cat([o + 1, o + 2, o + 2])
    re = torch.sqrt((_image(x[a] - x[b], box) ** 2).sum(-1))
    excl = -(KC * q[a] * q[b] * torch.erf(alpha * re) / re).sum()
    rec = KC * _reciprocal(x, box, q, alpha, K)
    return lj, real, excl, rec, -KC * alpha / math.sqrt(math.pi) * (q * q).sum()


def _bonded(x, n):
    bt = W.water_bonded_terms(n)
    t = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    bd, an = t(bt.bonds), t(bt.angles)
    r = torch.sqrt(((x[bd[:, 0]] - x[bd[:, 1]]) ** 2).sum(-1))
    u, v = x[an[:, 0]] - x[an[:, 1]], x[an[:, 2]] - x[an[:, 1]]
    th = torch.atan2(torch.linalg.norm(torch.linalg.cross(u, v), dim=-1), (u * v).sum(-1))
    return 0.5 * (t(bt.kb) * (r - t(bt.b0)) ** 2).sum(), 0.5 * (t(bt.kth) * (th - t(bt.th0)) ** 2).sum()


def _forces(wb, dt, flexible=False):
    x = _rounded(wb.coords, dt).requires_grad_(True)
    box = _rounded(wb.box, dt)
    q, sig = _rounded(wb.charges, dt), _rounded(wb.sigma, dt)
    lj, real, excl, rec, self_ = _terms(x, box, q, sig, torch.sqrt(_rounded(wb.epsilon, dt)), wb.cutoff, wb.alpha, wb.grid)
    terms = [lj + real, excl, rec, self_] + (list(_bonded(x, wb.n_waters)) if flexible else [])
    total = sum(terms)
    (g,) = torch.autograd.grad(total, x)
    return {"lj": lj.detach(), "energy": total.detach(), "terms": torch.stack([t.detach() for t in terms]), "gradient": g}


def exact(case, seed):
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    if kind in ("md", "eval"):
        f = _forces(_water(case, seed), dt, bool(case.get("flexible")))
        return {"forces": -f["gradient"], "terms": f["terms"]}
    if kind == "ops":
        f = _forces(_water(case, seed), dt)
        t = f["terms"]
        return {"lj": f["lj"], "coulomb": t[0] - f["lj"] + t[1], "pme": t[2] + t[3], "gradient": f["gradient"],
                "npairs": None}
    if kind == "train":
        wb, q, s, e, target = _train_inputs(case, seed)
        x = _rounded(wb.coords, dt).requires_grad_(True)
        q, s = (_rounded(a, dt).requires_grad_(True) for a in (q, s))
        root = torch.sqrt(_rounded(e, dt)).requires_grad_(True)
        total = sum(_terms(x, _rounded(wb.box, dt), q, s, root, wb.cutoff, wb.alpha, wb.grid))
        (gx,) = torch.autograd.grad(total, x, create_graph=True)
        loss = torch.mean((-gx - _rounded(target, dt)) ** 2)
        dq, ds, dr = torch.autograd.grad(loss, [q, s, root])
        de = torch.where(root > 0, dr / (2.0 * torch.clamp(root, min=1e-300)), torch.zeros_like(dr)).detach()
        return {"loss": loss.detach(), "forces": -gx.detach(), "charges": dq, "sigma": ds, "epsilon": de}
    if kind == "pairs":
        wb = _water(case, seed)
        x, box = _rounded(wb.coords, dt).requires_grad_(True), _rounded(wb.box, dt)
        q, s = (_rounded(a, dt).requires_grad_(True) for a in (wb.charges, wb.sigma))
        root = torch.sqrt(_rounded(wb.epsilon, dt)).requires_grad_(True)
        energy, grads = 0.0, None
        i_all, j_all = _pair_list(x.detach(), box, wb.cutoff)
        for i, j in zip(i_all.split(1 << 22), j_all.split(1 << 22)):
            d = _image(x[i] - x[j], box)
            r2 = (d * d).sum(-1)
            e = _lj(r2, 0.5 * (s[i] + s[j]), root[i] * root[j]) + (
                KC * q[i] * q[j] * (torch.rsqrt(r2) - 1.0 / (PAIRS_ROOM * wb.cutoff))).sum()
            g = torch.autograd.grad(e, [x, s, root, q])
            energy, grads = energy + e.detach(), g if grads is None else [a + b for a, b in zip(grads, g)]
        gx, gs, gr, gq = grads
        ge = torch.where(root > 0, gr / (2.0 * torch.clamp(root, min=1e-300)), torch.zeros_like(gr)).detach()
        if not case["params"]:
            gs = ge = gq = None
        # in 32 bits the total (of both signs, hundreds of times smaller than its parts) is off by
        # what the rounding of millions of terms happens to leave: the gradients say how exact they are
        e = energy.reshape(1) if case["dtype"] == "f64" else None
        return {"energy": e, "gradient": gx, "sigma": gs, "epsilon": ge, "charges": gq}
    if kind == "pme":
        x, box, q = _pme_inputs(case, seed)
        x, q, box = _rounded(x, dt).requires_grad_(True), _rounded(q, dt).requires_grad_(True), _rounded(box, dt)
        e = _reciprocal(x, box, q, PME_ALPHA, case["grid"]) - PME_ALPHA / math.sqrt(math.pi) * (q * q).sum()
        gx, gq = torch.autograd.grad(e, [x, q])
        return {"energy": e.detach(), "gradient": gx, "charges": gq}
    fs = [_forces(b, dt) for b in _serving(case, seed)]
    energies = torch.stack([f["energy"] for f in fs])
    if kind == "batch":
        return {"energies": energies, "forces": torch.cat([-f["gradient"] for f in fs])}
    return {"energies": energies.cpu().numpy(), "forces": [(-f["gradient"]).cpu().numpy() for f in fs]}
