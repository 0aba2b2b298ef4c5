"""The timed cases of this package: what its users have it do, over the real range of sizes.

Every case goes through the public entry points, as a solver, a fit or a
device-side driver calls them:

* ``force``  a solver's step on host arrays: ``NeighbourList.check_and_rebuild``
             and the force function, numpy in and numpy out;
* ``eval``   ``potential.evaluate`` on a device batch with a prebuilt list
             (the energy / force / virial call of every device-side loop);
* ``set``    captured ``BatchedEvaluator`` runs over a set of small uneven
             cells (phonon, elastic and training sets);
* ``list``   ``DeviceNeighbourList.build``;
* ``md``     ``md.NVE.run``: a block of ten velocity-Verlet steps;
* ``fit``    ``PotentialFit.loss_and_grad``: forward and backward over a
             training set.

Structures are the seeded synthetic ones of the benchmark (fcc and diamond
supercells with Gaussian displacements), with vacancies and strain where a
case asks for them.  Results of the mixed-precision path are kept in float32,
the precision of its bond terms.

``exact`` restates each energy function in float64 torch and takes forces,
virials and fit gradients from autograd; it uses none of the package's code,
only its published parameter tables.
"""
import math

import numpy as np
import torch

from akitsushima_b200.published_parameters import (SW_GESN_TOMITA_2018, SW_SI_1985, TERSOFF_1989, TERSOFF_SI_1988,
                                                   ZHOU_2004)

DIAMOND = [[0, 0, 0], [0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0], [0.25, 0.25, 0.25], [0.25, 0.75, 0.75],
           [0.75, 0.25, 0.75], [0.75, 0.75, 0.25]]
FCC = [[0, 0, 0], [0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0]]

# name: (basis, lattice constant, displacement sigma, species, smallest cells
# per axis, r_cut, neighbours inside the cutoff); the cells are the
# benchmark's, the smallest ones those the minimum image admits
MODELS = {
    "ni": (FCC, 3.52, 0.08, ["Ni"], 4, 5.75, 76),
    "cuni": (FCC, 3.58, 0.08, ["Cu", "Ni"], 4, 5.81, 73),
    "cunial": (FCC, 3.70, 0.08, ["Cu", "Ni", "Al"], 4, 6.69, 86),
    "cuni_setfl": (FCC, 3.58, 0.08, ["Cu", "Ni"], 4, 5.81, 73),
    "sw_si": (DIAMOND, 5.431, 0.1, ["Si"], 2, 3.77, 5),
    "sw_gesn": (DIAMOND, 5.762, 0.1, ["Ge", "Sn"], 2, 4.46, 16),
    "tersoff_si": (DIAMOND, 5.431, 0.05, ["Si"], 2, 3.0, 4),
    "tersoff_sic": (DIAMOND, 4.36, 0.1, ["Si", "C"], 2, 3.0, 7),
}
SKIN = 0.3


def _case(name, kind, model, precision, cells, **more):
    c = {"kind": kind, "model": model, "precision": precision, "nx": cells[0], "ny": cells[1], "nz": cells[2],
         "strain": 0.0, "vacancies": 0, "structures": 1}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # the smallest call in earnest: a 64-atom silicon cell stepped by a host solver
        _case("force_tersoff_si64", "force", "tersoff_si", "fp64", (2, 2, 2)),
        # an ordinary metal cell from the same host loop, default precision
        _case("force_eam_ni4000", "force", "ni", "fp64", (10, 10, 10)),
        # the headline: one evaluation of 256,000 Cu-Ni atoms, mixed precision
        _case("eam_cuni_256k_mixed", "eval", "cuni", "mixed", (40, 40, 40)),
        # the default precision at a middle size, with vacancies (ragged rows, odd atom count)
        _case("eam_cuni_32k_fp64", "eval", "cuni", "fp64", (20, 20, 20), vacancies=37),
        # the same alloy read from tables (setfl splines), as most published EAM potentials come
        _case("eam_setfl_cuni_256k_mixed", "eval", "cuni_setfl", "mixed", (40, 40, 40)),
        # a multi-species Stillinger-Weber alloy of 64,000 atoms
        _case("sw_gesn_64k_mixed", "eval", "sw_gesn", "mixed", (20, 20, 20)),
        # multi-species Tersoff in a strained (triclinic) cell, default precision
        _case("tersoff_sic_32k_fp64", "eval", "tersoff_sic", "fp64", (16, 16, 16), strain=0.02),
        # a displacement / strain set: 512 uneven silicon cells through two potentials, one graph each
        _case("set_si512_mixed", "set", "tersoff_si+sw_si", "mixed", (4, 4, 4), strain=0.03, structures=512),
        # the list of the headline structure, as a moving structure needs it again and again
        _case("list_cuni_256k", "list", "cuni", "fp64", (40, 40, 40)),
        # ten NVE steps of 4096 silicon atoms, default precision
        _case("md_tersoff_si4096_fp64", "md", "tersoff_si", "fp64", (8, 8, 8)),
        # one step of a fit: loss and gradient over 256 SiC cells, Tersoff-1989 variables
        _case("fit_sic256", "fit", "tersoff_sic", "fp64", (2, 2, 2), strain=0.02, structures=256),
        # and over 256 Ni3Al cells, Zhou EAM variables
        _case("fit_ni3al256", "fit", "ni3al", "fp64", (4, 4, 4), strain=0.02, structures=256),
    ]


def _cells(rng, lo, hi):
    """Cells per axis: a size spread over its logarithm, the axes up to a third apart."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return tuple(max(lo, min(hi, int(n * rng.uniform(0.75, 1.3)))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["force", "eval", "eval", "eval", "set", "list", "md", "fit"])
    precision = rng.choice(["fp64", "mixed"])
    strain = rng.choice([0.0, 0.0, round(rng.uniform(0.005, 0.03), 4)])
    if kind == "fit":
        model = rng.choice(["tersoff_sic", "ni3al"])
        n = int(math.exp(rng.uniform(math.log(16), math.log(257))))
        lo = 2 if model == "tersoff_sic" else 4
        return _case(None, kind, model, "fp64", (lo,) * 3, strain=round(rng.uniform(0.005, 0.025), 4), structures=n)
    if kind == "set":
        model = rng.choice(["tersoff_si+sw_si", "tersoff_si", "sw_si"])
        return _case(None, kind, model, precision, (rng.randint(2, 4),) * 3, strain=round(rng.uniform(0.01, 0.03), 4),
                     structures=int(math.exp(rng.uniform(math.log(16), math.log(513)))))
    if kind == "md":
        model = rng.choice(["sw_si", "tersoff_si", "sw_gesn", "cuni"])
        hi = 20 if MODELS[model][0] is DIAMOND else 16
        return _case(None, kind, model, precision, _cells(rng, MODELS[model][4], hi), vacancies=rng.choice([0, 1, 5]))
    model = rng.choice(list(MODELS))
    eam = MODELS[model][0] is FCC
    if kind == "force":
        return _case(None, kind, model, "fp64", _cells(rng, MODELS[model][4], 12 if eam else 10),
                     strain=strain, vacancies=rng.choice([0, 1, 3]))
    if kind == "list":
        return _case(None, kind, model, "fp64", _cells(rng, MODELS[model][4], 38 if eam else 24), strain=strain,
                     vacancies=rng.choice([0, 1, 3]))
    return _case(None, kind, model, precision, _cells(rng, MODELS[model][4], 38 if eam else 22), strain=strain,
                 vacancies=rng.choice([0, 1, 11]))


# ---- inputs ------------------------------------------------------------------

def _strain(rng, amp):
    e = rng.uniform(-amp, amp, (3, 3))
    return np.eye(3) + 0.5 * (e + e.T)


def _structure(rng, basis, a, sigma, species, cells, strain, vacancies, random_species=True):
    """(lattice, positions, species ids): a displaced, strained supercell."""
    g = np.stack(np.meshgrid(*[np.arange(n) for n in cells], indexing="ij"), -1).reshape(-1, 3)
    frac = (np.asarray(basis, float)[None] + g[:, None]).reshape(-1, 3)
    lat = np.diag(np.asarray(cells, float) * a)
    pos = frac * a
    nb = len(basis)
    if len(species) == 1:
        ids = np.zeros(len(pos), np.int32)
    elif species == ["Si", "C"]:       # zincblende
        ids = np.tile(np.repeat(np.arange(2), nb // 2), len(g)).astype(np.int32)
    elif species == ["Al", "Ni"]:      # L1_2 Ni3Al
        ids = np.tile(np.array([0, 1, 1, 1]), len(g)).astype(np.int32)
    elif species == ["Ge", "Sn"]:
        ids = rng.choice(2, len(pos), p=[0.75, 0.25]).astype(np.int32)
    else:
        ids = rng.integers(0, len(species), len(pos)).astype(np.int32)
    if strain:
        m = _strain(rng, strain)
        lat, pos = lat @ m, pos @ m
    pos = pos + rng.normal(0.0, sigma, pos.shape)
    if vacancies:
        keep = np.ones(len(pos), bool)
        keep[rng.choice(len(pos), vacancies, replace=False)] = False
        pos, ids = pos[keep], ids[keep]
    return lat, np.ascontiguousarray(pos), np.ascontiguousarray(ids)


def _one(case, seed):
    basis, a, sigma, species = MODELS[case["model"]][:4]
    # a list's length depends on the positions: its seeds are one structure,
    # moved through the cell and numbered from another atom
    moved = case["kind"] == "list"
    rng = np.random.default_rng([1 if moved else seed, 11])
    lat, pos, ids = _structure(rng, basis, a, sigma, species, (case["nx"], case["ny"], case["nz"]), case["strain"],
                               case["vacancies"])
    if moved:
        rng = np.random.default_rng([seed, 17])
        k = int(rng.integers(len(pos)))
        pos, ids = np.roll(pos, k, axis=0) + rng.uniform(0.0, 1.0, 3) @ lat, np.roll(ids, k)
    return lat, pos, ids, species


def _many(case, seed):
    """The structures of a set or fit case: uneven cells around (nx, ny, nz),
    of the same sizes for every seed."""
    rng = np.random.default_rng([seed, 12])
    sizes = np.random.default_rng(18)
    out = []
    for _ in range(case["structures"]):
        if case["kind"] == "set":      # 1 .. n cells per axis
            cells = tuple(int(c) for c in sizes.integers(1, case["nx"] + 1, 3))
            out.append(_structure(rng, DIAMOND, 5.431, 0.1, ["Si"], cells, case["strain"], 0))
            continue
        n = int(sizes.integers(case["nx"], case["nx"] + 2))
        args = (DIAMOND, 4.36, 0.1, ["Si", "C"]) if case["model"] == "tersoff_sic" else (FCC, 3.57, 0.08, ["Al", "Ni"])
        out.append(_structure(rng, *args, (n, n, n), case["strain"], 0))
    return out


def _fit_refs(structures, seed, fit_ni3al):
    """Reference energies per atom, forces and stresses of the training set,
    of the size a rattled cell's have."""
    rng = np.random.default_rng([seed, 13])
    e0, df, ds = (-4.5, 0.8, 0.02) if fit_ni3al else (-6.2, 1.5, 0.05)
    return [(e0 + 0.1 * rng.normal(), rng.normal(0.0, df, p.shape), (lambda s: 0.5 * (s + s.T))(rng.normal(0.0, ds, (3, 3))))
            for _, p, _ in structures]


T1989_KEYS = ("A", "B", "lambda", "mu", "c", "d", "h")
T1989_LOG = ("A", "B", "lambda", "mu", "c", "d", "chi")
ZHOU_FIT_KEYS = ("A", "B", "alpha", "beta", "Fn2", "Fn3", "F2", "F3", "eta")
ZHOU_FIT_LOG = ("A", "B", "alpha", "beta")
FIT_WEIGHTS = {"energy": 1.0, "forces": 1.0, "stress": 0.1}


def _fit_x(model, seed):
    """The optimiser's variables: near the published values."""
    if model == "ni3al":
        x = [math.log(ZHOU_2004[s][k]) if k in ZHOU_FIT_LOG else ZHOU_2004[s][k] for s in ("Al", "Ni")
             for k in ZHOU_FIT_KEYS]
    else:
        x = [math.log(TERSOFF_1989["elements"][s][k]) if k in T1989_LOG else TERSOFF_1989["elements"][s][k]
             for s in ("Si", "C") for k in T1989_KEYS] + [math.log(TERSOFF_1989["chi"]["C-Si"])]
    x = np.array(x)
    return x + 0.01 * np.random.default_rng([seed, 14]).normal(size=x.shape)


def _velocities(case, seed, n):
    """About 300 K."""
    return np.random.default_rng([seed, 15]).normal(0.0, 3.0e-3, (n, 3))


# ---- the calls ---------------------------------------------------------------

def _potential(model, precision):
    import akitsushima_b200 as ak
    from akitsushima_b200 import eam
    if model in ("ni", "cuni", "cunial", "cuni_setfl"):
        species = MODELS[model][3]
        pot = ak.zhou_eam({s: ZHOU_2004[s] for s in species}, species, precision=precision)
        return eam.tabulate(pot, precision=precision) if model == "cuni_setfl" else pot
    if model == "sw_si":
        return ak.StillingerWeberPotential(SW_SI_1985, species=["Si"], precision=precision)
    if model == "sw_gesn":
        return ak.StillingerWeberPotential(SW_GESN_TOMITA_2018, species=["Ge", "Sn"], precision=precision)
    if model == "tersoff_si":
        return ak.TersoffPotential(TERSOFF_SI_1988, species=["Si"], precision=precision)
    el = {s: dict(TERSOFF_1989["elements"][s]) for s in ("Si", "C")}
    return ak.TersoffPotential(ak.tersoff1989_to_triplets(el, TERSOFF_1989["chi"], ["Si", "C"]), species=["Si", "C"],
                               precision=precision)


def prepare(case, seed):
    import akitsushima_b200 as ak
    kind = case["kind"]
    s = {"kind": kind, "precision": case["precision"]}
    if kind == "fit":
        from akitsushima_b200 import fit
        ni3al = case["model"] == "ni3al"
        species = ["Al", "Ni"] if ni3al else ["Si", "C"]
        structs = _many(case, seed)
        refs = _fit_refs(structs, seed, ni3al)
        train = [{"lattice": L, "positions": P, "atom_types": t, "natoms": len(P), "ref_energy": e, "ref_forces": f,
                  "ref_stress": st} for (L, P, t), (e, f, st) in zip(structs, refs)]
        if ni3al:
            ps = fit.ZhouEAMParameterSet({k: dict(ZHOU_2004[k]) for k in species}, species)
        else:
            ps = fit.Tersoff1989ParameterSet({k: dict(TERSOFF_1989["elements"][k]) for k in species},
                                             TERSOFF_1989["chi"], species)
        s["fit"] = fit.PotentialFit(ps, train, FIT_WEIGHTS)
        s["x"] = _fit_x(case["model"], seed)
        return s
    if kind == "set":
        structs = _many(case, seed)
        s["evaluators"] = []
        for model in case["model"].split("+"):
            ev = ak.BatchedEvaluator(_potential(model, case["precision"]), structs, skin=SKIN)
            s["evaluators"].append(ev.capture())
        return s
    lat, pos, ids, species = _one(case, seed)
    if kind == "force":
        pot = _potential(case["model"], case["precision"])
        s["fn"] = ak.make_force_fn(pot)
        s["types"] = [species[k] for k in ids]
        s["lat"], s["pos"] = lat, pos
        s["list"] = ak.NeighbourList(pot.r_cut, skin_width=SKIN)
        s["list"].build(lat, pos + np.random.default_rng([seed, 16]).normal(0.0, 0.01, pos.shape))
        return s
    if kind == "md":
        from akitsushima_b200 import md
        pot = _potential(case["model"], case["precision"])
        s["nve"] = md.NVE(pot, lat, pos, [species[k] for k in ids], velocities=_velocities(case, seed, len(pos)),
                          dt=1.0, skin=SKIN, steps_per_graph=10)
        s["nve"].capture()
        return s
    s["batch"] = ak.Batch.single(lat, pos, ids)
    if kind == "list":
        r_cut = MODELS[case["model"]][5]
        s["list"] = ak.DeviceNeighbourList(r_cut + SKIN).build(s["batch"])
        return s
    s["pot"] = _potential(case["model"], case["precision"])
    s["list"] = ak.DeviceNeighbourList(s["pot"].r_cut + SKIN).build(s["batch"])
    return s


def _keep(s, *tensors):
    """float32 for what the mixed path computes in float32."""
    return [t.float() for t in tensors] if s["precision"] == "mixed" else list(tensors)


def run(s):
    kind = s["kind"]
    if kind == "force":
        s["list"].check_and_rebuild(s["lat"], s["pos"])
        return s["fn"](s["lat"], s["pos"], s["types"], s["list"])
    if kind == "eval":
        r = s["pot"].evaluate(s["batch"], s["list"])
        return _keep(s, r.energy, r.forces, r.virial)
    if kind == "set":
        outs = [ev.run() for ev in s["evaluators"]]
        return [_keep(s, r.energy, r.forces, r.virial) for r in outs]
    if kind == "list":
        d = s["list"].build(s["batch"])
        return d.row_off[:d.n_atoms + 1], d.nbr[:d.n_slots], d.rev[:d.n_slots], d.upper[:d.n_atoms]
    if kind == "md":
        nve = s["nve"].run(10)
        return _keep(s, nve.batch.pos, nve.vel, nve.out.forces, nve.out.energy)
    return s["fit"].loss_and_grad(s["x"])


# ---- the work a case cannot do without ------------------------------------------

# floating-point operations (add, multiply 1; divide, root 4; exp, log, pow,
# sin 8) per neighbour inside the cutoff, per ordered angle and per atom
_PAIR = {"ni": 240, "cuni": 290, "cunial": 290, "cuni_setfl": 150, "sw_si": 160, "sw_gesn": 160, "tersoff_si": 200,
         "tersoff_sic": 200}
_ANGLE = {"sw_si": 45, "sw_gesn": 55, "tersoff_si": 110, "tersoff_sic": 110}


def _eval_work(model, n):
    basis, a, _, _, _, rc, k = MODELS[model]
    slots = n * len(basis) / a ** 3 * 4.0 / 3.0 * math.pi * (rc + SKIN) ** 3
    per = 0.5 * k * _PAIR[model] if basis is FCC else k * 0.5 * _PAIR[model] + k * (k - 1) * _ANGLE[model]
    # positions, species, forces and one offset an atom; one neighbour index a slot
    return {"bytes": n * (24 + 4 + 24 + 4) + 4 * slots, "flops": n * per}


def work(case):
    kind = case["kind"]
    if kind == "fit":
        per = (case["nx"] ** 3 + (case["nx"] + 1) ** 3) / 2.0
        if case["model"] == "ni3al":
            n = case["structures"] * 4 * per
            w = _eval_work("cunial", n)
        else:
            n = case["structures"] * 8 * per
            w = _eval_work("tersoff_sic", n)
        # forward, then the adjoint: the terms and their parameter derivatives along a tangent
        return {"bytes": 2 * w["bytes"] + 24 * n, "flops": 5 * w["flops"]}
    if kind == "set":
        mean = ((1 + case["nx"]) / 2.0) ** 3
        n = case["structures"] * 8 * mean
        ws = [_eval_work(m, n) for m in case["model"].split("+")]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"] * len(MODELS[case["model"]][0]) - case["vacancies"]
    w = _eval_work(case["model"], n)
    if kind == "list":
        slots = (w["bytes"] - 56 * n) / 4
        # positions in; offsets, neighbours, reverse slots and upper offsets out; one distance test a listed pair
        return {"bytes": n * (24 + 8) + 8 * slots, "flops": 10 * slots}
    if kind == "md":
        # per step: the force call, and positions, velocities and masses through the kicks
        return {"bytes": 10 * (w["bytes"] + n * (2 * 48 + 8)), "flops": 10 * (w["flops"] + 60 * n)}
    return w


# ---- the same values in float64 torch --------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _f(a):
    return torch.as_tensor(np.asarray(a, float), dtype=torch.float64, device=_dev())


def _pairs(lat, pos, rc):
    """Every directed pair (i, j, image of j) within rc: i, j, image - wrap shift (P, 3) Cartesian."""
    dev = _dev()
    L, r = _f(lat), _f(pos)
    inv = torch.linalg.inv(L)
    base = torch.floor(r @ inv)
    w = r - base @ L
    n = len(w)
    widths = 1.0 / torch.linalg.norm(inv, dim=0).cpu().numpy()
    ii, jj, sh = [], [], []
    if n <= 4096:
        m = [int(rc / d + 1.0) for d in widths]
        for a in range(-m[0], m[0] + 1):
            for b in range(-m[1], m[1] + 1):
                for c in range(-m[2], m[2] + 1):
                    v = torch.tensor([a, b, c], dtype=torch.float64, device=dev)
                    if n <= 512:
                        d = (w + v @ L)[None] - w[:, None]
                        hit = (d * d).sum(-1) < rc * rc
                    else:
                        hit = torch.cdist(w, w + v @ L, compute_mode="donot_use_mm_for_euclid_dist") < rc
                    if a == b == c == 0:
                        hit.fill_diagonal_(False)
                    i, j = hit.nonzero(as_tuple=True)
                    ii.append(i)
                    jj.append(j)
                    sh.append(v.expand(len(i), 3))
    else:
        nc = np.maximum(3, np.floor(widths / rc).astype(int))
        g = torch.as_tensor(nc, device=dev)
        ci = torch.minimum(((w @ inv) * g).long().clamp_(min=0), g - 1)
        cell = (ci[:, 0] * g[1] + ci[:, 1]) * g[2] + ci[:, 2]
        order = torch.argsort(cell)
        cnt = torch.bincount(cell, minlength=int(np.prod(nc)))
        start = torch.cumsum(cnt, 0) - cnt
        cols = torch.arange(int(cnt.max()), device=dev)
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                for c in (-1, 0, 1):
                    t = ci + torch.tensor([a, b, c], device=dev)
                    v = torch.div(t, g, rounding_mode="floor")
                    t = t - v * g
                    k = (t[:, 0] * g[1] + t[:, 1]) * g[2] + t[:, 2]
                    q = start[k][:, None] + cols[None]
                    ok = cols[None] < cnt[k][:, None]
                    j = order[q.clamp(max=n - 1)]
                    v = v.double()
                    d = w[j] + (v @ L)[:, None] - w[:, None]
                    hit = ok & ((d * d).sum(-1) < rc * rc)
                    if a == b == c == 0:
                        hit &= j != torch.arange(n, device=dev)[:, None]
                    i, q = hit.nonzero(as_tuple=True)
                    ii.append(i)
                    jj.append(j[i, q])
                    sh.append(v[i])
    i, j, s = torch.cat(ii), torch.cat(jj), torch.cat(sh)
    o = torch.argsort(i, stable=True)
    i, j, s = i[o], j[o], s[o]
    return i, j, (s - base[j] + base[i]) @ L


class _System:
    """Concatenated structures and their directed pairs within rc."""

    def __init__(self, structs, rc):
        i, j, sh, off = [], [], [], 0
        for lat, pos, _ in structs:
            a, b, s = _pairs(lat, pos, rc)
            i.append(a + off)
            j.append(b + off)
            sh.append(s)
            off += len(pos)
        self.i, self.j, self.shift = torch.cat(i), torch.cat(j), torch.cat(sh)
        self.pos = _f(np.concatenate([p for _, p, _ in structs]))
        self.types = torch.as_tensor(np.concatenate([t for _, _, t in structs]).astype(np.int64), device=_dev())
        self.n = [len(p) for _, p, _ in structs]
        self.struct = torch.repeat_interleave(torch.arange(len(structs), device=_dev()),
                                              torch.tensor(self.n, device=_dev()))
        self.n_atoms, self.n_struct = off, len(structs)

    def triplets(self):
        """Ordered pairs (e, f) of directed pairs with one centre, e != f."""
        cnt = torch.bincount(self.i, minlength=self.n_atoms)
        start = torch.cumsum(cnt, 0) - cnt
        rep = cnt[self.i]
        e = torch.repeat_interleave(torch.arange(len(self.i), device=_dev()), rep)
        first = torch.cumsum(rep, 0) - rep
        f = start[self.i[e]] + torch.arange(len(e), device=_dev()) - first[e]
        keep = e != f
        return e[keep], f[keep]

    def efs(self, atom_energy, create_graph=False, pos=None):
        """(E (S,), F (N, 3), W (S, 9)) of sum of atom_energy(system, d)."""
        with torch.enable_grad():
            r = (self.pos if pos is None else pos).detach().requires_grad_(True)
            eps = torch.zeros((self.n_struct, 3, 3), dtype=torch.float64, device=_dev(), requires_grad=True)
            d = r[self.j] + self.shift - r[self.i]
            d = d + (eps[self.struct[self.i]] @ d[:, :, None])[:, :, 0]
            u = atom_energy(self, d)
            E = torch.zeros(self.n_struct, dtype=torch.float64, device=_dev()).index_add(0, self.struct, u)
            gr, ge = torch.autograd.grad(E.sum(), (r, eps), create_graph=create_graph)
        return E, -gr, -ge.reshape(-1, 9)


def _per_atom(S, i, v):
    return torch.zeros(S.n_atoms, dtype=torch.float64, device=_dev()).index_add(0, i, v)


ZK = ("r_e", "f_e", "rho_e", "rho_s", "alpha", "beta", "A", "B", "kappa", "lambda", "Fn0", "Fn1", "Fn2", "Fn3", "F0",
      "F1", "F2", "F3", "eta", "F_e")


def _zhou_continuous(p):
    """Fn0, Fn1, F0 and F_e from the continuity of F and F' at 0.85 and 1.15 rho_e."""
    q = {k: _f(v) if not torch.is_tensor(v) else v for k, v in p.items()}
    y, x = 0.15, -0.15
    t0 = 1.15 * q["rho_e"] / q["rho_s"]
    lt = torch.log(t0)
    q["F_e"] = ((q["F1"] + 2 * q["F2"] * y + 3 * q["F3"] * y * y) / q["rho_e"]) / (
        -q["eta"] ** 2 * lt * t0 ** (q["eta"] - 1.0) / q["rho_s"])
    q["F0"] = q["F_e"] * (1 - q["eta"] * lt) * t0 ** q["eta"] - (q["F1"] * y + q["F2"] * y * y + q["F3"] * y ** 3)
    q["Fn0"] = q["F0"] + q["F1"] * x + q["F2"] * x * x + q["F3"] * x ** 3
    q["Fn1"] = 0.85 * (q["F1"] + 2 * q["F2"] * x + 3 * q["F3"] * x * x)
    return q


def _zhou_fu(p, r):
    """Unswitched density f and pair phi_aa of one element."""
    x = r / p["r_e"]
    g = torch.exp(-p["beta"] * (x - 1)) / (1 + (x - p["lambda"]) ** 20)
    return p["f_e"] * g, p["A"] * torch.exp(-p["alpha"] * (x - 1)) / (1 + (x - p["kappa"]) ** 20) - p["B"] * g


def _zhou_cut(els, tol=1e-6):
    """The distance past which both functions of every element have decayed below tol."""
    rc = 0.0
    for p in els:
        r = torch.linspace(float(p["r_e"]), 5.0 * float(p["r_e"]), 40001, dtype=torch.float64)
        q = {k: float(v) for k, v in p.items()}
        f, u = _zhou_fu(q, r)
        bad = (~((u.abs() < tol * max(q["A"], q["B"])) & (f < tol * q["f_e"]))).nonzero()
        rc = max(rc, float(r[int(bad[-1]) + 1]) if len(bad) else float(r[0]))
    return rc


def _switch(r, rc, width=0.5):
    s = ((r - (rc - width)) / width).clamp(0.0, 1.0)
    return 1.0 - s ** 3 * (10.0 - 15.0 * s + 6.0 * s * s)


def _zhou_F(p, rho):
    rn = 0.85 * p["rho_e"]
    z, y = rho / rn - 1.0, rho / p["rho_e"] - 1.0
    lo = p["Fn0"] + z * (p["Fn1"] + z * (p["Fn2"] + z * p["Fn3"]))
    mid = p["F0"] + y * (p["F1"] + y * (p["F2"] + y * p["F3"]))
    top = 1.15 * p["rho_e"]
    t = torch.where(rho >= top, rho, top * torch.ones_like(rho)) / p["rho_s"]
    hi = p["F_e"] * (1.0 - p["eta"] * torch.log(t)) * t ** p["eta"]
    return torch.where(rho < rn, lo, torch.where(rho >= top, hi, mid))


def _zhou_energy(els, rc):
    def u(S, d):
        r = (d * d).sum(-1).sqrt()
        sw = _switch(r, rc)
        fu = [_zhou_fu(p, r) for p in els]
        ti, tj = S.types[S.i], S.types[S.j]
        rho = torch.zeros_like(r)
        phi = torch.zeros_like(r)
        for b in range(len(els)):
            rho = torch.where(tj == b, fu[b][0], rho)
        for a in range(len(els)):
            for b in range(a, len(els)):
                if a == b:
                    v, m = fu[a][1], (ti == a) & (tj == a)
                else:
                    q = fu[b][0] / fu[a][0]
                    v, m = 0.5 * (q * fu[a][1] + fu[b][1] / q), ((ti == a) & (tj == b)) | ((ti == b) & (tj == a))
                phi = torch.where(m, v, phi)
        bar = _per_atom(S, S.i, rho * sw)
        F = torch.zeros_like(bar)
        for a, p in enumerate(els):
            F = torch.where(S.types == a, _zhou_F(p, bar), F)
        return F + 0.5 * _per_atom(S, S.i, phi * sw)
    return u


def _spline(x, y):
    """Cubic spline on uniform knots, not-a-knot ends: coefficients (4, n - 1), highest power first."""
    n, h = len(x), x[1] - x[0]
    A = np.zeros((n, n))
    b = np.zeros(n)
    k = np.arange(1, n - 1)
    A[k, k - 1], A[k, k], A[k, k + 1] = 1.0, 4.0, 1.0
    b[1:-1] = 6.0 * (y[2:] - 2 * y[1:-1] + y[:-2]) / h ** 2
    A[0, :3], A[-1, -3:] = (1.0, -2.0, 1.0), (1.0, -2.0, 1.0)
    m = np.linalg.solve(A, b)
    return np.stack([(m[1:] - m[:-1]) / (6 * h), m[:-1] / 2, (y[1:] - y[:-1]) / h - h * (2 * m[:-1] + m[1:]) / 6, y[:-1]])


def _setfl_energy(els, rc):
    """The Zhou alloy written to 2000-point tables and read back as splines."""
    n = 2000
    r_g = np.linspace(0.0, rc, n)
    r_p = torch.as_tensor(np.where(r_g > 0.0, r_g, r_g[1]))
    q = [{k: float(v) for k, v in p.items()} for p in els]
    sw = _switch(r_p, rc)
    fu = [_zhou_fu(p, r_p) for p in q]
    rho_t = [(f * sw).numpy() for f, _ in fu]
    rho_g = np.linspace(0.0, 50.0 * max(t.max() for t in rho_t), n)
    F_t = [_zhou_F({k: torch.tensor(v, dtype=torch.float64) for k, v in p.items()}, torch.as_tensor(rho_g)).numpy() for p in q]
    cross = 0.5 * (fu[1][0] / fu[0][0] * fu[0][1] + fu[0][0] / fu[1][0] * fu[1][1])
    phi_t = [[fu[0][1], cross], [cross, fu[1][1]]]
    R = [(_f(r_g), _f(_spline(r_g, t))) for t in rho_t]
    F = [(_f(rho_g), _f(_spline(rho_g, t))) for t in F_t]
    P = [[(_f(r_g), _f(_spline(r_g, r_g * (v * sw).numpy()))) for v in row] for row in phi_t]

    def at(table, r):
        x, c = table
        k = ((r.detach() - x[0]) / (x[1] - x[0])).long().clamp(0, len(x) - 2)
        d = r - x[k]
        return ((c[0][k] * d + c[1][k]) * d + c[2][k]) * d + c[3][k]

    def u(S, d):
        r = (d * d).sum(-1).sqrt()
        ti, tj = S.types[S.i], S.types[S.j]
        bar = _per_atom(S, S.i, torch.where(tj == 0, at(R[0], r), at(R[1], r)))
        bar = torch.where(bar > 0, bar, torch.zeros_like(bar))
        like = torch.where(ti == 0, at(P[0][0], r), at(P[1][1], r))
        phi = torch.where(ti != tj, at(P[0][1], r), like) / r
        return torch.where(S.types == 0, at(F[0], bar), at(F[1], bar)) + 0.5 * _per_atom(S, S.i, phi)
    return u


def _sw_energy(records, species):
    ns = len(species)
    two = _f([[[records[(a, b, b)][k] for k in ("epsilon", "sigma", "a", "A", "B", "p", "q", "gamma")] for b in species]
              for a in species])
    tri = _f([[[[0.5 * records[(a, b, c)]["epsilon"] * records[(a, b, c)]["lambda"], records[(a, b, c)]["costheta0"]]
                for c in species] for b in species] for a in species])
    assert two.shape[0] == ns

    def u(S, d):
        r = (d * d).sum(-1).sqrt()
        p = two[S.types[S.i], S.types[S.j]]
        x = r / p[:, 1]
        inside = x < p[:, 2]
        xa = torch.where(inside, x - p[:, 2], -torch.ones_like(x))
        zero = torch.zeros_like(x)
        v2 = torch.where(inside, p[:, 0] * p[:, 3] * (p[:, 4] * x ** -p[:, 5] - x ** -p[:, 6]) * torch.exp(1 / xa), zero)
        leg = torch.where(inside, torch.exp(p[:, 7] / xa), zero)
        e, f = S.triplets()
        cos = (d[e] * d[f]).sum(-1) / (r[e] * r[f])
        c = tri[S.types[S.i[e]], S.types[S.j[e]], S.types[S.j[f]]]
        v3 = c[:, 0] * leg[e] * leg[f] * (cos - c[:, 1]) ** 2
        return 0.5 * _per_atom(S, S.i, v2) + _per_atom(S, S.i[e], v3)
    return u


def _tersoff_energy(pair, angle):
    """pair (ns, ns, 8): A B lambda1 lambda2 R D beta n; angle (ns, 3): c d h of the centre; lambda3 = 0."""
    def u(S, d):
        r = (d * d).sum(-1).sqrt()
        p = pair[S.types[S.i], S.types[S.j]]
        A, B, l1, l2, R, D, beta, n = p.unbind(-1)
        x = ((r - R) / D).clamp(-1.0, 1.0)
        fc = torch.where(r > R + D, torch.zeros_like(r), 0.5 - 0.5 * torch.sin(0.5 * math.pi * x))
        e, f = S.triplets()
        c, dd, h = angle[S.types[S.i[e]]].unbind(-1)
        cos = (d[e] * d[f]).sum(-1) / (r[e] * r[f])
        hc = (h - cos) ** 2
        g = 1.0 + c * c * hc / (dd * dd * (dd * dd + hc))
        zeta = torch.zeros_like(r).index_add(0, e, fc[f] * g)
        live = zeta > 0
        z = torch.where(live, zeta, torch.ones_like(zeta))
        b = torch.where(live, (1.0 + (beta * z) ** n) ** (-0.5 / n), torch.ones_like(z))
        v = fc * (A * torch.exp(-l1 * r) - b * B * torch.exp(-l2 * r))
        return 0.5 * _per_atom(S, S.i, v)
    return u


def _t1989(el, chi):
    """Tersoff (1989) mixing of element parameters (tensors) for two elements."""
    def mean(k):
        v = torch.stack([e[k] for e in el])
        return 0.5 * (v[:, None] + v[None])

    def root(k):
        v = torch.stack([e[k] for e in el])
        return torch.sqrt(v[:, None] * v[None])
    one = torch.ones((2, 2), dtype=torch.float64, device=_dev())
    x = torch.eye(2, dtype=torch.float64, device=_dev())
    x = x + chi * (one - x)
    R, Sx = root("R"), root("S")
    cen = [torch.stack([e[k] for e in el])[:, None] * one for k in ("beta", "n")]
    pair = torch.stack([root("A"), x * root("B"), mean("lambda"), mean("mu"), 0.5 * (R + Sx), 0.5 * (Sx - R)] + cen, -1)
    return pair, torch.stack([torch.stack([e[k] for k in ("c", "d", "h")]) for e in el])


def _reference(model):
    """(energy function, cutoff) of a model in float64 torch."""
    if model in ("ni", "cuni", "cunial", "cuni_setfl"):
        els = [_zhou_continuous(ZHOU_2004[s]) for s in MODELS[model][3]]
        rc = _zhou_cut(els)
        return (_setfl_energy if model == "cuni_setfl" else _zhou_energy)(els, rc), rc
    if model == "sw_si":
        return _sw_energy({("Si",) * 3: SW_SI_1985}, ["Si"]), SW_SI_1985["a"] * SW_SI_1985["sigma"]
    if model == "sw_gesn":
        rec = {(r["i"], r["j"], r["k"]): r for r in SW_GESN_TOMITA_2018}
        return _sw_energy(rec, ["Ge", "Sn"]), max(r["a"] * r["sigma"] for r in SW_GESN_TOMITA_2018 if r["j"] == r["k"])
    if model == "tersoff_si":
        p = TERSOFF_SI_1988
        pair = _f([[[p[k] for k in ("A", "B", "lambda1", "lambda2", "R", "D", "beta", "n")]]])
        return _tersoff_energy(pair, _f([[p["c"], p["d"], p["h"]]])), p["R"] + p["D"]
    el = [{k: _f(v) for k, v in TERSOFF_1989["elements"][s].items()} for s in ("Si", "C")]
    return _tersoff_energy(*_t1989(el, _f(TERSOFF_1989["chi"]["C-Si"]))), TERSOFF_1989["elements"]["Si"]["S"]


def _exact_fit(case, seed):
    structs = _many(case, seed)
    ni3al = case["model"] == "ni3al"
    refs = _fit_refs(structs, seed, ni3al)
    x = _f(_fit_x(case["model"], seed)).requires_grad_(True)
    if ni3al:
        els = []
        for a, s in enumerate(("Al", "Ni")):
            p = {k: _f(v) for k, v in ZHOU_2004[s].items()}
            for k, v in zip(ZHOU_FIT_KEYS, x[9 * a:9 * a + 9]):
                p[k] = torch.exp(v) if k in ZHOU_FIT_LOG else v
            els.append(_zhou_continuous(p))
        rc = _zhou_cut([_zhou_continuous(ZHOU_2004[s]) for s in ("Al", "Ni")])
        u = _zhou_energy(els, rc)
    else:
        el = []
        for a, s in enumerate(("Si", "C")):
            p = {k: _f(v) for k, v in TERSOFF_1989["elements"][s].items()}
            for k, v in zip(T1989_KEYS, x[7 * a:7 * a + 7]):
                p[k] = torch.exp(v) if k in T1989_LOG else v
            el.append(p)
        rc = TERSOFF_1989["elements"]["Si"]["S"]
        u = _tersoff_energy(*_t1989(el, torch.exp(x[14])))
    S = _System(structs, rc)
    E, F, W = S.efs(u, create_graph=True)
    n = _f(S.n)
    vol = _f([abs(np.linalg.det(L)) for L, _, _ in structs])
    e_sq = (E - n * _f([e for e, _, _ in refs])) ** 2
    dF = F - _f(np.concatenate([f for _, f, _ in refs]))
    f_sq = torch.zeros_like(E).index_add(0, S.struct, (dF * dF).sum(1)) / (3.0 * n)
    ds = W / vol[:, None] - _f(np.stack([s.reshape(9) for _, _, s in refs]))
    s_sq = vol ** 2 * (ds * ds).mean(1)
    loss = (FIT_WEIGHTS["energy"] * e_sq + FIT_WEIGHTS["forces"] * f_sq + FIT_WEIGHTS["stress"] * s_sq).sum()
    g, = torch.autograd.grad(loss, x)
    return float(loss.detach()), g.cpu().numpy()


AMU = {"Si": 28.086, "Ge": 72.630, "Sn": 118.71, "Cu": 63.546, "Ni": 58.693}
EV_ANG_TO_AMU_ANG_FS2 = (1.60217663e-19 / 1.0e-10) / (1.66053906660e-27) * 1.0e-20


def _exact_md(case, seed):
    lat, pos, ids, species = _one(case, seed)
    u, rc = _reference(case["model"])
    L = _f(lat)
    inv = torch.linalg.inv(L)
    r, v = _f(pos), _f(_velocities(case, seed, len(pos)))
    h = 0.5 * EV_ANG_TO_AMU_ANG_FS2 / _f([AMU[species[k]] for k in ids])[:, None]

    def force(r):
        S = _System([(lat, r.cpu().numpy(), ids)], rc)
        E, F, _ = S.efs(u)
        return E.detach(), F
    E, F = force(r)
    for _ in range(10):
        v = v + h * F
        s = (r + v) @ inv
        r = (s - torch.floor(s)) @ L
        E, F = force(r)
        v = v + h * F
    return [r, v, F, E]


def exact(case, seed):
    kind = case["kind"]
    if kind == "list":
        return None                      # whole numbers: nothing is rounded
    big = work(case)["flops"] > 2e8 and not torch.cuda.is_available()
    if big:
        return None                      # minutes on a CPU
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "md":
        return _exact_md(case, seed)
    if kind == "set":
        structs = _many(case, seed)
        out = []
        for model in case["model"].split("+"):
            u, rc = _reference(model)
            S = _System([_replicated(s, _reps(s[0], rc + SKIN)) for s in structs], rc)
            E, F, W = S.efs(u)
            out.append([E.detach(), F, W])
        return out
    lat, pos, ids, _ = _one(case, seed)
    u, rc = _reference(case["model"])
    E, F, W = _System([(lat, pos, ids)], rc).efs(u)
    if kind == "force":
        return float(E[0].detach()), F.cpu().numpy(), (W[0].reshape(3, 3) / abs(np.linalg.det(lat))).cpu().numpy()
    return [E.detach(), F, W]


def _reps(lat, r_list):
    """Copies per axis that give the smallest supercell the minimum image admits."""
    widths = 1.0 / np.linalg.norm(np.linalg.inv(lat), axis=0)
    reps = []
    for w in widths:
        k = 1
        while w * k / 2.0 <= r_list:
            k += 1
        reps.append(k)
    return reps


def _replicated(s, reps):
    lat, pos, ids = s
    shifts = np.array([[a, b, c] for a in range(reps[0]) for b in range(reps[1]) for c in range(reps[2])], float)
    return lat * np.array(reps, float)[:, None], (pos[None] + (shifts @ lat)[:, None]).reshape(-1, 3), np.tile(ids, len(shifts))
