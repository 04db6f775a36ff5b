"""The calls that a user's program makes into this framework, as cases that can be timed.

A program optimises a design (``Context.begin`` and ``Context.step``, the loop of TOP3D_XL), or it
uses the solver's parts on its own: the stiffness operator on device vectors, the preconditioner after
new moduli, a linear solve, the PDE filter, element compliances.  The listed cases take these over the
sizes of this repository's workloads and tests (cuboids of 16x32x16 to 128x256x128 elements, generated
irregular domains), GLOBAL and LOCAL, FP64 and mixed precision, and odd sizes; ``draw`` takes them over
the ranges in between.

A design run starts from the uniform density as every run does: its first iterations are the
ones whose outputs do not depend on the last bits of the arithmetic (a PCG stopped at 1e-3 on a developed
design amplifies rounding by up to 1e8).
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from top3d_xl_b200 import Context
from top3d_xl_b200.workloads import irregular_domain, write_topvoxel

SIMP, EMIN, POISSON = 3.0, 1e-6, 0.3  # the reference's settings, the defaults of Context
CORNERS = [(1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 0), (1, 0, 1), (1, 1, 1), (0, 1, 1), (0, 0, 1)]  # (y, x, z) of a hex's nodes


def listed():
    def design(name, size, cons, **more):
        case = {"name": name, "kind": "design", "ny": size[0], "nx": size[1], "nz": size[2], "domain": "cuboid", "cons": cons,
                "precision": "fp64", "V0": 0.12 if cons == "GLOBAL" else 0.5, "rMin": math.sqrt(3),
                "rHat": 0.0 if cons == "GLOBAL" else 6.0, "loops": 1 if cons == "GLOBAL" else 3}
        return dict(case, **more)

    def part(name, kind, size, **more):
        return dict({"name": name, "kind": kind, "ny": size[0], "nx": size[1], "nz": size[2], "domain": "cuboid"}, **more)

    return [
        # the smallest job of a served stream: launches and latency
        design("design_small", (16, 32, 16), "GLOBAL"),
        # the reference's demo cuboid, TOP3D_XL(true(50,100,50),'GLOBAL',0.12,50,sqrt(3))
        design("design_demo", (50, 100, 50), "GLOBAL"),
        # half a million elements
        design("design_large", (64, 128, 64), "GLOBAL"),
        # the benchmark's cuboid, 4.2 million elements, as porous infill
        design("infill_large", (128, 256, 128), "LOCAL", loops=2),
        # porous infill of a part with bores through it
        design("infill_part", (72, 144, 72), "LOCAL", domain="bored"),
        # the demo's infill in mixed precision, as the job server runs it
        design("infill_mixed", (50, 100, 50), "LOCAL", precision="mixed", loops=1),
        # one linear elasticity analysis of a graded cuboid
        part("solve", "solve", (32, 64, 32)),
        # new moduli, the multigrid operators and the coarse factor for them, and one preconditioner call
        part("precondition", "precondition", (64, 128, 64)),
        # the operator inside a caller's own iteration on device vectors: a large grid, and a small odd one
        part("operator", "operator", (64, 128, 64)),
        part("operator_small", "operator", (13, 27, 11), domain="holes"),
        # the density filter with a wide radius on an irregular part (ellipsoids and rods: two thirds of the box
        # are void), and the element energies of a displacement field
        part("filter", "filter", (96, 192, 96), domain="part", rMin=6.0),
        part("energy", "energy", (75, 150, 75)),
    ]


def draw(rng):
    def extent(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["design"] * 5 + ["solve", "precondition", "operator", "operator", "filter", "energy"])
    cons = rng.choice(["GLOBAL", "LOCAL"])
    small, large = {"design": (14, 64 if cons == "GLOBAL" else 110), "solve": (14, 48), "precondition": (14, 72), "operator": (8, 66),
                    "filter": (14, 72), "energy": (14, 90)}[kind]
    ny = extent(small, large)
    nx, nz = max(6, int(ny * rng.uniform(1.2, 2.05))), max(6, int(ny * rng.uniform(0.7, 1.05)))
    case = {"kind": kind, "ny": ny, "nx": nx, "nz": nz, "domain": "cuboid"}
    if kind == "operator":
        case["domain"] = rng.choice(["cuboid", "holes"])
    if kind in ("precondition", "filter") and ny >= 30:
        case["domain"] = rng.choice(["cuboid", "part"])
    if kind == "filter":
        case["rMin"] = rng.choice([math.sqrt(3), 2.5, 6.0])
    if kind == "design":
        case.update(cons=cons, precision="fp64", loops=1, rMin=rng.choice([math.sqrt(3), 2.5]), rHat=0.0)
        case["V0"] = rng.uniform(0.08, 0.2) if cons == "GLOBAL" else rng.uniform(0.45, 0.6)
        if cons == "LOCAL":
            case.update(rHat=6.0, loops=rng.choice([1, 2, 3]))
            if ny >= 48 and rng.random() < 0.5:
                case.update(precision="mixed", loops=1)
            elif ny >= 20:
                case["domain"] = rng.choice(["cuboid", "bored"])
    return case


# --- inputs ------------------------------------------------------------------------------------------


def _domain(case, rng):
    """The voxel mask, the fixed nodes and the loads (node, fx, fy, fz), with node ids as in a .TopVoxel file."""
    ny, nx, nz = case["ny"], case["nx"], case["nz"]
    if case["domain"] == "part":
        s = ny / 192.0  # the generator's full-size box is 192 wide
        vox, fixed, loads = irregular_domain(seed=8, box=(ny, nx, nz), semi=(20 * s, 90 * s),
                                             radius=(max(2, 10 * s), 30 * s), half_length=(50 * s, 150 * s))
        at = [row[0] for row in loads]
        f = rng.standard_normal((len(at), 3))  # the generator's unit forces in random directions
        return vox, np.asarray(fixed), np.asarray(at), f / np.linalg.norm(f, axis=1, keepdims=True)
    vox = np.ones((ny, nx, nz), bool)
    if case["domain"] == "holes":
        vox = np.random.default_rng(5).random((ny, nx, nz)) < 0.75
        vox[:, 0, :] = vox[:, -1, :] = True
    if case["domain"] == "bored":
        y, x = np.meshgrid(np.arange(ny) + 0.5, np.arange(nx) + 0.5, indexing="ij")
        for at in (0.28, 0.7):
            vox[np.hypot(y - ny / 2, x - at * nx) < min(0.32 * ny, 0.15 * nx)] = False
    y, z = np.meshgrid(np.arange(ny + 1), np.arange(nz + 1), indexing="ij")
    fixed = (1 + y + (ny + 1) * (nx + 1) * z).ravel()
    y, z = np.meshgrid(np.arange(ny + 1), np.arange(1 + nz // 6), indexing="ij")
    at = (1 + y + (ny + 1) * (nx + (nx + 1) * z)).ravel()
    # forces about the direction -z, as the built-in cuboid's
    f = np.array([0.0, 0.0, -1.0]) + 0.3 * rng.standard_normal((len(at), 3))
    return vox, np.asarray(fixed), np.asarray(at), f / len(at)


def _moduli(rng, n, lowest):
    x = rng.uniform(lowest, 1.0, n)
    return EMIN + x ** SIMP * (1.0 - EMIN)


def prepare(case, seed):
    rng = np.random.default_rng([seed, case["ny"], case["nx"], case["nz"]])
    vox, fixed, at, force = _domain(case, rng)
    ctx = Context(case.get("precision", "fp64"))
    state = {"case": case, "ctx": ctx, "vox": vox, "fixed": fixed, "at": at, "force": force}
    kind = case["kind"]
    if case["domain"] == "part":
        with tempfile.TemporaryDirectory() as folder:
            path = os.path.join(folder, "part.TopVoxel")
            write_topvoxel(path, vox, fixed.tolist(), [(n, *f) for n, f in zip(at.tolist(), force.tolist())])
            ctx.load_topvoxel(path)
    else:
        ctx.load_voxels(vox)
    if kind in ("design", "solve"):
        fixing = np.ones((len(fixed), 4))
        fixing[:, 0] = fixed
        ctx.set_bc(fixing, np.column_stack([at, force, np.ones(len(at))]))
    if kind == "design":
        # page-locked, as a program that fetches every design does
        state["density"] = torch.empty(ctx.numElements, dtype=torch.float64, pin_memory=True).numpy()
    elif kind == "solve":
        state["E"] = _moduli(rng, ctx.numElements, 0.3)
        ctx.set_moduli(state["E"])
        ctx.assemble()
    elif kind == "precondition":
        state["E"] = _moduli(rng, ctx.numElements, 0.05)
        state["r"] = rng.standard_normal(ctx.numDOFs)
    elif kind == "operator":
        state["E"] = _moduli(rng, ctx.numElements, 0.05)
        ctx.set_moduli(state["E"])
        state["u"] = torch.from_numpy(rng.standard_normal(ctx.numDOFs)).cuda()
        state["y"] = torch.empty_like(state["u"])
    elif kind == "filter":
        state["src"] = rng.uniform(0.0, 1.0, ctx.numElements)
    elif kind == "energy":
        state["U"] = rng.standard_normal((ctx.numDOFs, 1))
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "design":
        solid = ctx.begin(case["cons"], case["V0"], 50, case["rMin"], case["rHat"])
        rows = [ctx.step() for _ in range(case["loops"])]
        return {"solid": solid, "compliance": np.array([r["c"] for r in rows]), "volume": np.array([r["vol"] for r in rows]),
                "sharpness": np.array([r["sharp"] for r in rows]), "iterations": np.array([r["its"] for r in rows]),
                "density": ctx.density(state["density"])}
    if kind == "solve":
        u, its = ctx.pcg()
        return {"u": u, "iterations": its}
    if kind == "precondition":
        ctx.set_moduli(state["E"])
        ctx.assemble()
        return ctx.vcycle(state["r"])
    if kind == "operator":
        u, y = state["u"], state["y"]
        ctx._check(ctx.lib.topx_ku_noalloc(ctx._h, ctypes.c_void_p(u.data_ptr()), ctypes.c_void_p(y.data_ptr()), u.numel()))
        return y
    if kind == "filter":
        out, its = ctx.filter(case["rMin"], state["src"])
        return {"filtered": out, "iterations": its}
    return ctx.unit_compliance(state["U"])


# --- what a pass cannot do without -----------------------------------------------------------------------


def work(case):
    """Bytes that have to move between the caller's arrays, HBM and the chip, and floating-point operations.

    A PCG iteration (node fields of 3 doubles): the operator reads r (or z) and p and the moduli, writes p and K p, and updates u; the
    residual update reads r and K p and writes r; the preconditioner reads r again for the coarse levels: 11 fields of 24 bytes and 8 bytes
    of moduli.  An operator application takes 600 multiply-adds per node as the element matrix stands; its reflections split it into
    3x3 blocks, which with their transforms need about 170 operations per node: those are counted.
    """
    ny, nx, nz = case["ny"], case["nx"], case["nz"]
    fill = {"cuboid": 1.0, "holes": 0.75, "bored": 0.74, "part": 0.33}[case["domain"]]
    elems, nodes = fill * ny * nx * nz, min(1.0, 1.1 * fill) * (ny + 1) * (nx + 1) * (nz + 1)
    kind = case["kind"]
    it_bytes, it_flops = 11 * 24 * nodes + 8 * elems, 230 * nodes
    filter_bytes, filter_flops = 8 * 8 * nodes + elems, 60 * nodes
    if kind == "design":
        solves = 1 + case["loops"]  # of the solid domain, and one for each design: 25 iterations each
        filters = case["loops"] * (1 if case["cons"] == "GLOBAL" else 5)  # of 6 to 15 iterations
        its = 6 if case["cons"] == "GLOBAL" else 10
        update = 50 * 16 if case["cons"] == "GLOBAL" else 60 * 80  # bisection or interior-point passes over element arrays
        chip = min(1.0, elems * 16 / 1e8)  # arrays that stay on the chip are read once
        return {"bytes": solves * 25 * it_bytes + filters * its * filter_bytes + case["loops"] * update * elems * chip + 8 * elems,
                "flops": solves * 25 * it_flops + filters * its * filter_flops + case["loops"] * elems * 350}
    if kind == "solve":
        return {"bytes": 30 * it_bytes + 48 * nodes, "flops": 30 * it_flops}
    if kind == "precondition":
        return {"bytes": 8 * elems + 48 * nodes + 576 * 8 * elems / 64 * 2.3 + 24 * nodes, "flops": elems * 2 * 576 + 200 * nodes}
    if kind == "operator":
        return {"bytes": 48 * nodes + 8 * elems, "flops": 170 * nodes}
    if kind == "filter":
        return {"bytes": 15 * filter_bytes + 16 * elems, "flops": 15 * filter_flops}
    return {"bytes": 24 * nodes + 8 * elems, "flops": 324 * 2 * elems}


# --- the same in 64 bits with torch --------------------------------------------------------------------------


def _hexahedron():
    """Ke of the unit cube (nu = 0.3, E = 1) and the gradient and mass parts of the filter's matrix, 2x2x2 Gauss points."""
    sign = np.array([(2 * x - 1, 1 - 2 * y, 2 * z - 1) for y, x, z in CORNERS], float)  # the row index y runs against the y axis
    points = np.array([(a, b, c) for c in (-1, 1) for b in (-1, 1) for a in (-1, 1)]) / math.sqrt(3)
    lam, mu = POISSON / ((1 + POISSON) * (1 - 2 * POISSON)), 0.5 / (1 + POISSON)
    D = np.diag([2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam
    Ke, grad, mass = np.zeros((24, 24)), np.zeros((8, 8)), np.zeros((8, 8))
    for p in points:
        t = 1 + sign * p
        N = t.prod(1) / 8
        d = np.stack([sign[:, i] * t[:, (i + 1) % 3] * t[:, (i + 2) % 3] / 8 for i in range(3)])  # natural coordinates
        g = 2 * d  # the cell's edge is 1
        B = np.zeros((6, 24))
        for i in range(3):
            B[i, i::3] = g[i]
        B[3, 0::3], B[3, 1::3] = g[1], g[0]
        B[4, 1::3], B[4, 2::3] = g[2], g[1]
        B[5, 2::3], B[5, 0::3] = g[0], g[2]
        Ke += B.T @ D @ B / 8
        grad += d.T @ d
        mass += np.outer(N, N) / 8
    return Ke, grad, mass


class _Grid:
    """Element sums on the dense grid of the case's box (y fastest); compact vectors hold the solid part in grid order."""

    def __init__(self, vox):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.ny, self.nx, self.nz = vox.shape
        self.solid = torch.from_numpy(np.ascontiguousarray(vox.transpose(2, 1, 0))).to(dev)
        self.present = self.scatter(self.solid.double().unsqueeze(-1).expand(*self.solid.shape, 8)) > 0

    def gather(self, u):
        return torch.stack([u[z:z + self.nz, x:x + self.nx, y:y + self.ny] for y, x, z in CORNERS], 3)

    def scatter(self, f):
        out = torch.zeros((self.nz + 1, self.nx + 1, self.ny + 1) + tuple(f.shape[4:]), dtype=torch.float64, device=f.device)
        for a, (y, x, z) in enumerate(CORNERS):
            out[z:z + self.nz, x:x + self.nx, y:y + self.ny] += f[:, :, :, a]
        return out

    def elements(self, v):
        out = torch.zeros(self.solid.shape, dtype=torch.float64, device=self.solid.device)
        out[self.solid] = torch.from_numpy(np.asarray(v)).to(out.device)
        return out


def _cg(apply, b, diag, tol, most):
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz, stop = z.clone(), (r * z).sum(), tol * float(b.norm())
    for it in range(most):
        q = apply(p)
        step = rz / (p * q).sum()
        x += step * p
        r -= step * q
        if it % 20 == 0 and float(r.norm()) < stop:
            break
        z = r / diag
        new = (r * z).sum()
        p = z + new / rz * p
        rz = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("design", "precondition"):
        return None  # whole runs, and the multigrid cycle, which is this method's own
    if kind == "solve" and case["ny"] * case["nx"] * case["nz"] > 80000:
        return None
    state = prepare(case, seed)
    grid = _Grid(state["vox"])
    dev = grid.solid.device
    Ke, grad, mass = _hexahedron()
    K = torch.from_numpy(Ke).to(dev)
    nodes = grid.present.sum().item()

    def field(v):
        out = torch.zeros(grid.present.shape + (3,), dtype=torch.float64, device=dev)
        out[grid.present] = torch.as_tensor(v).to(dev).reshape(nodes, 3)
        return out

    if kind == "energy":
        ue = grid.gather(field(state["U"][:, 0])).flatten(3)
        return ((ue @ K) * ue).sum(-1)[grid.solid].cpu().numpy()
    if kind == "filter":
        R = case["rMin"] / 2 / math.sqrt(3)
        A = torch.from_numpy(R * R * grad + mass).to(dev)
        b = grid.scatter((grid.elements(state["src"]) / 8).unsqueeze(-1).expand(*grid.solid.shape, 8))
        one = grid.solid.double().unsqueeze(-1)
        diag = grid.scatter(one * A.diagonal())
        y = _cg(lambda v: grid.scatter(one * (grid.gather(v) @ A)), b, diag, 1e-14, 2000)
        return {"filtered": grid.gather(y).mean(-1)[grid.solid].cpu().numpy(), "iterations": None}
    E = grid.elements(state["E"]).unsqueeze(-1)
    fixed = torch.zeros(grid.present.numel(), dtype=torch.bool, device=dev)
    fixed[torch.from_numpy(state["fixed"] - 1).to(dev)] = True
    free = (~fixed).reshape(grid.present.shape).unsqueeze(-1) & grid.present.unsqueeze(-1)

    def stiffness(u):
        ue = grid.gather(u * free)
        f = (E * (ue.flatten(3) @ K)).unflatten(3, (8, 3))
        return torch.where(free, grid.scatter(f), u)

    if kind == "operator":
        return stiffness(field(state["u"]))[grid.present].reshape(-1)
    f = torch.zeros((grid.present.numel(), 3), dtype=torch.float64, device=dev)
    f[torch.from_numpy(state["at"] - 1).to(dev)] = torch.from_numpy(state["force"]).to(dev)
    diag = torch.where(free, grid.scatter((E * K.diagonal()).unflatten(3, (8, 3))), torch.ones_like(E[:1, :1, :1, :1]))
    u = _cg(stiffness, f.reshape(grid.present.shape + (3,)), diag, 1e-13, 6000)
    return {"u": u[grid.present].reshape(-1).cpu().numpy(), "iterations": None}
