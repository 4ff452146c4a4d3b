"""Timed cases: what users of this library have it compute, through its public entry points.

Six kinds of case:

  train      the training driver's loop over one buffer of frames (alphanesgpu_b200/train.py): host arrays in,
             loss_and_grad_host_begin / adam_update_dev / loss_and_grad_host_end with two steps in flight
  train_dev  one training step of a program that keeps its frames on the GPU: loss_and_grad[_virial] + Adam
  infer      energies and forces (and virials) of a batch of frames on the GPU: StafModel.energy_force[_virial]
  domain     one rank's share of a slab-decomposed box: owned + ghost atoms, StafModel.energy_force_domain
  libstaf    the C API that a molecular-dynamics code links: staf_compute on host double arrays, with the library's
             own neighbour list or (list = True) with the caller's list over owned + ghost atoms
  operators  the operator surface (alphanesgpu_b200/ops.py) as a framework's graph calls it: descriptors, then for
             every central species fingerprints, forces and all their gradients

Frames are synthetic liquid water: rigid molecules in random orientations on a jittered lattice with a few random
vacancies, orthorhombic boxes.  Models are the 2-species, 5-channels-per-class, 64-32-1 one of the benchmark, or
("wide") the 20 + 40 channel, 140-140-1 one of tests/golden.
"""
import ctypes as C
import math
import random
import shutil
import tempfile

import numpy as np
import torch

from alphanesgpu_b200 import _lib, ops, params
from alphanesgpu_b200.model import StafModel
from alphanesgpu_b200.params import ModelShape
from alphanesgpu_b200.train import init_params

CFG = dict(Rc=4.5, Rs=2.25, Ra=4.5, nr=60, na=1770)
DENSITY = 0.094            # atoms per cubic Angstrom: about 38 neighbours, as in tests/golden/ref_frame0
SKIN = 1.0                 # halo of a slab beyond the cutoff, as the slab driver is used
LR = 1e-5                  # a late step of the drivers' decaying learning rate
CHANNELS = {"small": dict(map_rad_afs={0: [5, 5], 1: [5, 5]}, map_ang_afs={0: [5, 5, 5], 1: [5, 5, 5]}),
            "wide": dict(map_rad_afs={0: [10, 10], 1: [10, 10]}, map_ang_afs={0: [13, 13, 14], 1: [13, 13, 14]})}
WIDTHS = {"small": [64, 32, 1], "wide": [140, 140, 1]}


def listed():
    def case(name, kind, mol, frames=1, steps=1, dtype="f32", model="small", virial=False, list=False):
        return dict(name=name, kind=kind, mol=mol, frames=frames, steps=steps, dtype=dtype, model=model,
                    virial=virial, list=list)
    return [
        # the smallest call there is: one 96-atom frame, where launches and the host path count
        case("infer-96", "infer", 32),
        # a handful of ragged frames with virials in double precision, as a constant-pressure run or a check wants
        case("infer-virial-3x579-f64", "infer", 193, frames=3, dtype="f64", virial=True),
        # a quarter of the 24,576-atom box on one rank of four
        case("domain-6144", "domain", 2048),
        # molecular dynamics of the 24,576-atom box through the C API
        case("libstaf-24576", "libstaf", 8192),
        # the same C API as a code with its own neighbour lists and ghost atoms calls it, the larger model
        case("libstaf-list-2997-wide", "libstaf", 999, model="wide", list=True),
        # training on small frames: two 96-atom frames per step (the test suite's data set)
        case("train-2x96", "train", 32, frames=2, steps=8),
        # the benchmark's step: four 768-atom frames
        case("train-4x768", "train", 256, frames=4, steps=8),
        # the data-parallel configuration: 64 frames in batches of eight
        case("train-8x768", "train", 256, frames=8, steps=8),
        # the benchmark's step in double precision
        case("train-4x768-f64", "train", 256, frames=4, steps=8, dtype="f64"),
        # the benchmark's step with the larger model
        case("train-4x768-wide", "train", 256, frames=4, steps=8, model="wide"),
        # energy + force + virial training with frames resident on the GPU, ragged sizes
        case("train-dev-virial-3x579", "train_dev", 193, frames=3, virial=True),
        # every operator, forward and backward, on one 768-atom frame
        case("operators-768", "operators", 256),
    ]


def draw(rng: random.Random):
    """One more case.  Sizes are spread over their logarithm; at most 6,144 atoms a training step (3,072 in double
    precision or with the larger model), 24,576 in an inference call (6,144 with those), 1,536 in the operators."""
    kind = rng.choice(["train", "train", "train_dev", "infer", "domain", "libstaf", "operators"])
    dtype = rng.choice(["f32", "f32", "f64"])
    model = rng.choice(["small", "small", "wide"]) if dtype == "f32" else "small"
    heavy = dtype == "f64" or model == "wide"
    most = {"train": 2048, "train_dev": 2048, "operators": 512}.get(kind, 2048 if heavy else 8192)
    if kind in ("train", "train_dev") and heavy:
        most //= 2
    batched = kind in ("train", "train_dev", "infer")
    least = 256 if kind == "domain" else 32  # a slab is at least two halos wide
    mol = int(round(math.exp(rng.uniform(math.log(least), math.log(min(1024, most) if batched else most)))))
    frames = int(round(math.exp(rng.uniform(0.0, math.log(max(1, min(16, most // mol))))))) if batched else 1
    return dict(kind=kind, mol=mol, frames=frames, steps=rng.randint(4, 8) if kind == "train" else 1, dtype=dtype,
                model=model, virial=kind in ("infer", "train_dev", "domain") and rng.random() < 0.4,
                list=kind == "libstaf" and mol <= 2048 and rng.random() < 0.5)


# ---------------------------------------------------------------- frames
def lattice(mol, edges=None):
    """Sites per edge and edges of a box for `mol` molecules: few vacancies, spacings alike, no edge below two
    cutoffs (then a cube)."""
    vol, best = 3 * mol / DENSITY, None
    cube = np.full(3, vol ** (1.0 / 3.0))
    h = (cube if edges is None else np.asarray(edges, np.float64)) / (vol / mol) ** (1.0 / 3.0)
    for a in range(max(1, int(0.6 * h[0])), int(1.5 * h[0]) + 2):
        for b in range(max(1, int(0.6 * h[1])), int(1.5 * h[1]) + 2):
            n = np.array([a, b, -(-mol // (a * b))])
            if edges is not None:
                L = np.asarray(edges, np.float64)
            else:
                L = n * (vol / n.prod()) ** (1.0 / 3.0)
                L = cube if L.min() < 9.3 or L.max() > 2.2 * L.min() else L
            cost = 2.0 * (n.prod() / mol - 1.0) + (L / n).max() / (L / n).min() - 1.0
            if best is None or cost < best[0]:
                best = (cost, n, L)
    return best[1:]


def water(rng, mol, edges=None):
    """One frame: positions [3*mol, 3] (oxygens, then hydrogens), box6."""
    n, L = lattice(mol, edges)
    L = L * (1.0 + rng.uniform(-0.005, 0.005, 3))
    site = np.sort(rng.permutation(int(n.prod()))[:mol])
    O = (np.stack(np.unravel_index(site, n), axis=1) + 0.5) * (L / n) + rng.normal(0.0, 0.1, (mol, 3))
    u = rng.normal(size=(mol, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = np.cross(u, rng.normal(size=(mol, 3)))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    half = np.deg2rad(104.52 / 2)
    H = O[:, None] + 0.9572 * (np.cos(half) * u[:, None] + np.sin(half) * np.stack([v, -v], axis=1))
    return np.concatenate([O, H.reshape(-1, 3)]), np.array([L[0], 0.0, 0.0, L[1], 0.0, L[2]])


def frames_of(rng, case, count):
    fr = [water(rng, case["mol"]) for _ in range(count)]
    return np.stack([f[0].reshape(-1) for f in fr]), np.stack([f[1] for f in fr])


def shape_of(case, tipos):
    ch = CHANNELS[case["model"]]
    return ModelShape(nt=2, tipos=list(tipos), Fr=[sum(ch["map_rad_afs"][t]) for t in (0, 1)],
                      Fa=[sum(ch["map_ang_afs"][t]) for t in (0, 1)], widths=list(WIDTHS[case["model"]]))


def dtypes(case):
    return (np.float32, torch.float32) if case["dtype"] == "f32" else (np.float64, torch.float64)


def ghosts_of(x, nominal, L, rc):
    """Periodic images (positions, owners) of the wrapped atoms x around the box, nearest first: as many as a shell a
    little wider than rc holds, whatever the atoms."""
    n = int(len(x) * (np.prod(nominal + 2.0 * (rc + 0.6)) / np.prod(nominal) - 1.0))
    far, gx, owner = 2.0 * rc, [], []
    for shift in np.ndindex(3, 3, 3):
        if shift == (1, 1, 1):
            continue
        img = x + (np.array(shift) - 1) * L
        keep = np.all((img > -far) & (img < L + far), axis=1)
        gx.append(img[keep])
        owner.append(np.nonzero(keep)[0])
    gx, owner = np.concatenate(gx), np.concatenate(owner)
    out = np.maximum(-gx, gx - L).max(axis=1)  # how far outside the box
    first = np.argsort(out, kind="stable")[:n]
    assert out[first[-1]] > rc
    return gx[first], owner[first]


def neighbour_rows(xall, n, rc, width):
    """Cutoff-filtered, distance-sorted rows of the first n atoms over all atoms."""
    xa = torch.as_tensor(xall, device="cuda")
    how, rows = [], []
    for lo in range(0, n, 256):
        d = torch.cdist(xa[lo:min(n, lo + 256)], xa, compute_mode="donot_use_mm_for_euclid_dist")
        k = torch.arange(d.shape[0], device="cuda")
        d[k, lo + k] = 1e30
        near, idx = torch.topk(d, width, dim=1, largest=False, sorted=True)
        inside = near < rc
        how.append(inside.sum(1).to(torch.int32))
        rows.append(torch.where(inside, idx, torch.zeros_like(idx)).to(torch.int32))
    return torch.cat(how).cpu().numpy(), torch.cat(rows).cpu().numpy()


class StafOptions(C.Structure):
    _fields_ = [("mlp_backend", C.c_int), ("device_id", C.c_int), ("precision", C.c_int), ("reserved", C.c_int)]


class Potential:
    """A potential loaded through the C API from an exported model directory."""

    def __init__(self, shape, theta, emb, double):
        self.lib = _lib.lib()
        self.lib.staf_load.restype = C.c_void_p
        self.lib.staf_load.argtypes = [C.c_char_p, C.c_void_p]
        self.lib.staf_compute.argtypes = ([C.c_void_p, C.c_int, C.c_int] + [C.c_void_p] * 5 + [C.c_int] +
                                          [C.c_void_p] * 3)
        self.lib.staf_free.argtypes = [C.c_void_p]
        folder = tempfile.mkdtemp(prefix="staf_model_")
        params.save_model_dir(folder, CFG, shape, theta, emb, precision=1 if double else 0)
        opt = StafOptions(0, torch.cuda.current_device(), 1 if double else 0, 0)
        self.h = self.lib.staf_load(folder.encode(), C.byref(opt))
        shutil.rmtree(folder, ignore_errors=True)
        if not self.h:
            raise RuntimeError("staf_load failed")

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.staf_free(self.h)
            self.h = None


class State:
    pass


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    npd, td = dtypes(case)
    mol, nf = case["mol"], case["frames"]
    s = State()
    s.case = case
    dev = torch.device("cuda", torch.cuda.current_device())
    to = lambda a: torch.as_tensor(np.ascontiguousarray(a, npd)).to(dev)
    tipos = [mol, 2 * mol]
    theta, emb = init_params(shape_of(case, tipos), CHANNELS[case["model"]], int(rng.integers(1 << 31)))
    kind = case["kind"]
    if kind in ("train", "train_dev", "infer"):
        n = nf * case["steps"]
        pos, box = frames_of(rng, case, n)
        el, fl, vl = rng.normal(size=n), rng.normal(size=pos.shape), rng.normal(0.0, 2.0, (n, 9))
        s.model = StafModel(shape_of(case, tipos), CFG, theta, emb, nf, dtype=td, device=dev)
        if kind == "train":
            s.host = [np.ascontiguousarray(a, npd) for a in (pos, box, el, fl)]
            s.stream = torch.cuda.Stream(device=dev)  # the driver's own stream
        else:
            s.data = [to(a) for a in (pos, box, el, fl, vl)]
    elif kind == "domain":
        # the global box is four slabs long; this rank owns the one that starts at z = 0
        edge = max((3 * mol / DENSITY) ** (1.0 / 3.0), 2.0 * (CFG["Rc"] + SKIN))
        side = math.sqrt(3 * mol / DENSITY / edge)
        x, box = water(rng, 4 * mol, edges=(side, side, 4 * edge))
        types = np.repeat(np.array([0, 1], np.int32), [4 * mol, 8 * mol])
        z = x[:, 2] - np.floor(x[:, 2] / box[5]) * box[5]
        up = np.argsort(z, kind="stable")
        n, ng = 3 * mol, int(3 * mol * (CFG["Rc"] + SKIN) / edge)  # owned atoms, ghosts beyond each face
        own = np.sort(up[:n])
        ids = np.concatenate([own, up[n:n + ng], up[-ng:]])
        counts = [int((types[own] == t).sum()) for t in (0, 1)]
        s.model = StafModel(shape_of(case, counts), CFG, theta, emb, 1, dtype=td, device=dev, n_max=len(ids))
        s.data = [to(x[ids]), to(box), torch.as_tensor(types[ids]).to(dev)]
    elif kind == "libstaf":
        x, box = water(rng, mol)
        types = np.repeat(np.array([0, 1], np.int32), tipos)
        order = rng.permutation(len(types))  # an MD code's atoms come in any order
        x, types = x[order], types[order]
        s.how = s.rows = None
        s.nghost = 0
        if case["list"]:
            L = box[[0, 3, 5]]
            x = x - np.floor(x / L) * L
            gx, owner = ghosts_of(x, lattice(mol)[1], L, CFG["Rc"])
            s.nghost = len(owner)
            x, types = np.concatenate([x, gx]), np.concatenate([types, types[owner]])
            s.how, s.rows = neighbour_rows(x, 3 * mol, CFG["Rc"], 64)
        s.x, s.box, s.types = np.ascontiguousarray(x.reshape(-1)), box, np.ascontiguousarray(types)
        s.pot = Potential(shape_of(case, tipos), theta, emb, case["dtype"] == "f64")
    else:
        pos, box = frames_of(rng, case, nf)
        shape = shape_of(case, tipos)
        N = shape.N
        ops.construct_descriptors_light(CFG["Rc"], CFG["nr"], CFG["na"], N, None, CFG["Rs"], CFG["Ra"], nf, dtype=td)
        s.data = [to(pos), to(box)]
        s.type_map = torch.as_tensor(shape.type_map).to(dev)
        s.tipos = torch.as_tensor(np.asarray(tipos, np.int32)).to(dev)
        s.species = []
        for t in (0, 1):
            o, Fr, Fa = shape.offsets(t), shape.Fr[t], shape.Fa[t]
            cut = lambda a, lo, r, c: to(a[lo:lo + r * c].reshape(r, c))
            s.species.append(dict(
                rows=slice(shape.shift(t), shape.shift(t) + tipos[t]),
                this=torch.tensor([t], dtype=torch.int32, device=dev),
                a2=cut(theta, o["a2"], 2, Fr), a3=cut(theta, o["a3"], 3, 3 * Fa),
                e2=cut(emb, o["emb"], 2, Fr), e3=cut(emb, o["emb"] + 2 * Fr, 3, Fa),
                # what the network behind the operators hands back: d(e)/d(AF) and dL/d(AF)
                nd2=to(rng.normal(size=(nf, tipos[t], Fr))), nd3=to(rng.normal(size=(nf, tipos[t], Fa))),
                g2=to(rng.normal(size=(nf, tipos[t], Fr))), g3=to(rng.normal(size=(nf, tipos[t], Fa)))))
        s.fbar = to(rng.normal(size=(nf, 3 * N)))
    return s


def run(s):
    kind, case = s.case["kind"], s.case
    if kind == "train":
        m, (pos, box, el, fl), nf, losses = s.model, s.host, case["frames"], []
        with torch.cuda.stream(s.stream):
            for k in range(case["steps"]):
                b = slice(k * nf, (k + 1) * nf)
                m.loss_and_grad_host_begin(pos[b], box[b], el[b], fl[b], k & 1)
                m.adam_update_dev(LR)
                if k:
                    losses.append(m.loss_and_grad_host_end((k - 1) & 1))
            losses.append(m.loss_and_grad_host_end((case["steps"] - 1) & 1))
        return dict(losses=np.stack(losses), grad=m.grad, theta=m.theta, adam_m=m.adam_m, adam_v=m.adam_v)
    if kind == "train_dev":
        m, (pos, box, el, fl, vl) = s.model, s.data
        if case["virial"]:
            m.loss_and_grad_virial(pos, box, el, fl, vl, pv=0.5)
        else:
            m.loss_and_grad(pos, box, el, fl)
        m.adam_update_dev(LR)
        return dict(losses=m.losses5 if case["virial"] else m.losses, grad=m.grad, theta=m.theta, adam_m=m.adam_m,
                    adam_v=m.adam_v)
    if kind == "infer":
        pos, box = s.data[:2]
        return s.model.energy_force_virial(pos, box) if case["virial"] else s.model.energy_force(pos, box)
    if kind == "domain":
        # as the slab driver calls it: the status word is looked at when the halo changes, not on every call
        return s.model.energy_force_domain(*s.data, virial=case["virial"], check_status=False)
    if kind == "libstaf":
        n = 3 * case["mol"]
        f, vir, e = np.zeros(len(s.x)), np.zeros(6), C.c_double()
        a = lambda v: None if v is None else v.ctypes.data
        rc = s.pot.lib.staf_compute(s.pot.h, n, s.nghost, a(s.x), a(s.box), a(s.types), a(s.how), a(s.rows),
                                    64 if case["list"] else 0, C.addressof(e), a(f), a(vir))
        if rc != 0:
            raise RuntimeError("staf_compute: %d" % rc)
        return dict(energy=e.value, force=f, virial=vir)
    d = ops.compute_descriptors_light(*s.data)
    out = list(d)
    for p in s.species:
        rad, ang, des3, im2, im3, d2, d3, d3s, nt = (x[:, p["rows"]] for x in d)
        a2, e2, a3, e3, tm, tp, at = p["a2"], p["e2"], p["a3"], p["e3"], s.type_map, s.tipos, p["this"]
        out.append(ops.compute_sort_proj(rad, im2, a2, e2, tm))
        out.append(ops.compute_sort_proj3body(ang, des3, im3, im2, a3, e3, tm, nt))
        out.append(ops.compute_force_radial(p["nd2"], d2, im2, rad, a2, e2, tm, tp, at))
        out.append(ops.compute_force_tripl(p["nd3"], des3, ang, d3s, d3, im2, im3, a3, e3, tm, tp, at, nt))
        out += ops.compute_two_body_par_grad(p["g2"], rad, im2, a2, e2, tm)
        out += ops.compute_sort_proj3body_grad(p["g3"], ang, des3, im3, im2, a3, e3, tm, nt)
        out += ops.compute_force_radial_grad(s.fbar, p["nd2"], d2, im2, rad, a2, e2, tm, tp, at)
        out += ops.compute_force_tripl_grad(s.fbar, p["nd3"], des3, ang, d3s, d3, im2, im3, a3, e3, tm, tp, at, nt)
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: inputs and outputs once.  Operations: multiply-adds (2) and exponentials (1) of the triplet sums (a mean
    of 720 triplets per atom at this density) and of the network."""
    es = 4 if case["dtype"] == "f32" else 8
    atoms = 3 * case["mol"] * case["frames"]
    shape = shape_of(case, [1, 1])
    act = shape.Fa[0] / shape.C
    trip, near = 720.0 * atoms, 38.0 * atoms
    net = sum(a * b for a, b in zip([shape.Fr[0] + shape.Fa[0]] + shape.widths[:-1], shape.widths))
    nparam, kind = shape.n_params, case["kind"]
    if kind in ("train", "train_dev"):
        flops = trip * (95 + 95 * act) + 16.0 * net * atoms
        one = es * (atoms * 6 + case["frames"] * 16) + 7 * es * nparam
        return {"bytes": one * case["steps"], "flops": flops * case["steps"]}
    if kind == "operators":
        isz = 4
        na, nr = CFG["na"], CFG["nr"]
        tensors = atoms * (es * (na + 6 * na + 8 * nr) + isz * (2 * na + nr + 2))
        reads = trip * (es * 7 + 2 * isz) + near * (es * 8 + isz)  # the filled slots, once for all operators
        chan = atoms * (shape.Fr[0] + shape.Fa[0]) * es * 4
        return {"bytes": tensors + reads + chan + atoms * 9 * es, "flops": trip * (95 + 95 * act)}
    flops = trip * (51 + 51 * act) + 4.0 * net * atoms
    moved = atoms * (24 + 24 + 4) if kind == "libstaf" else atoms * 6 * es
    if case["list"]:
        moved += atoms * (64 * 4 + 4)
    return {"bytes": moved + es * nparam, "flops": flops}


def tolerance(case):
    """32-bit sums over tens of neighbours and thousands of atoms, added in no fixed order; Adam moves a parameter
    whose gradient is rounding noise by up to the learning rate, which "max" leaves room for."""
    return {"rel": 2e-5, "max": 1e-3} if case["dtype"] == "f32" else {"rel": 1e-11, "max": 1e-8}
