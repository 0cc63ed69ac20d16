"""Measured cases of the Newton-step solve and the steps in front of it, through the package's public entry points.

Every case is something a Newton loop or a differentiable simulation has this package do, on the boxes of tetrahedra
that the workloads of `agipc_learning_b200.synth` are made of (Freudenthal boxes, point-triangle contacts, affine
bodies above a slab), with device-resident arrays as the reference hands them over:

  step       contacts, matrix, preconditioner build and solve of one Newton system (`MasPcg.set_contacts`,
             `set_matrix`, `build`, `solve`) on a kept graph and handle
  refresh    new values on a kept structure, then the solve (`refresh_values`, `solve`)
  adjoint    the differentiable solve, forward and backward (`newton_solve`, `newton_solve_modulus`)
  elements   per-tet gradient and projected Hessian triplets (`maspcg_fem_snk1_gradient_hessian`)
  merge      raw element and contact triplets to the unique upper blocks (`MasPcg.convert_bcoo`)
  partition  contact triplets grouped by kind (`MasPcg.partition_contact_triplets`)
  coarse     the AGIPC coarse system: P^T A P, P^T b and P x_c (`maspcg_galerkin_*`)
  operators  one FP64 product and one preconditioner apply, as a caller's own Krylov loop issues them
"""
import ctypes
import functools
import math

import numpy as np
import torch

from agipc_learning_b200 import autograd, synth
from agipc_learning_b200 import _native as native
from agipc_learning_b200.solver import MasPcg

H = 0.01          # vertex spacing of the boxes
DT = 1 / 60
NU = 0.45
RHO = 1000.0
DHAT = 1e-3
UPPER = [(a, b) for a in range(4) for b in range(a, 4)]


# ------------------------------------------------------------------ listed --

def _case(name, kind, nx, ny, nz, **more):
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "pairs": 0, "E": 1e6, "kappa": 1e7}
    c.update(more)
    return c


def listed():
    return [
        # the headline workload: 64^3 vertices with 50,000 contacts, mixed precision to the FP64-verified 1e-4
        _case("step_64_mixed", "step", 64, 64, 64, pairs=50000, precision="mixed", inverse="bf16", gate="euclid",
              preconditioner="mas32", tol=1e-4),
        # the app's default: CEMAS16 in the reference precision with the reference's own stopping rule
        _case("step_48_cemas16", "step", 48, 48, 48, pairs=28000, precision="reference", inverse="fp32", gate="rz",
              preconditioner="cemas16", tol=1e-4),
        # the library's default configuration (MAS32, reference precision, rz gate) on a box of odd edges
        _case("step_odd_mas32", "step", 61, 37, 45, pairs=15000, precision="reference", inverse="fp32", gate="rz",
              preconditioner="mas32", tol=1e-4),
        # the smallest workload: 20^3 without contacts, where latency and launches count
        _case("step_20_small", "step", 20, 20, 20, E=1e5, precision="mixed", inverse="bf16", gate="euclid",
              preconditioner="mas32", tol=1e-4),
        # affine bodies coupled to a stiff slab
        _case("step_hybrid", "step", 50, 50, 8, pairs=7500, E=1e8, kappa=1e8, bodies=500, precision="reference",
              inverse="fp32", gate="euclid", preconditioner="mas32", tol=1e-4),
        # a second Newton step on the same contact set: FP16 inverses, accurate sums with reliable replacement
        _case("refresh_40_accurate", "refresh", 40, 40, 40, pairs=9000, precision="mixed", inverse="fp16",
              gate="euclid", preconditioner="mas32", tol=1e-4, matrix="f32_accurate", replacement="reliable"),
        # system identification: 32^3 with a modulus per tet, forward and backward through the raw element triplets
        _case("adjoint_modulus_32", "adjoint", 32, 32, 32, E=1e5, precision="mixed", inverse="bf16", gate="euclid",
              preconditioner="mas32", tol=1e-10, modulus=True),
        # the same solve differentiated in its merged blocks, a small ragged box in the reference precision
        _case("adjoint_blocks_odd", "adjoint", 23, 17, 13, pairs=600, kappa=1e6, precision="reference",
              inverse="fp32", gate="euclid", preconditioner="mas32", tol=1e-8, modulus=False),
        # the element kernel on the headline mesh: 1,500,282 tets
        _case("elements_64", "elements", 64, 64, 64),
        # its triplets and the contacts', merged
        _case("merge_48", "merge", 48, 48, 48, pairs=28000),
        # the AGIPC coarse system for 2x2x2 aggregates
        _case("coarse_40", "coarse", 40, 40, 40, pairs=9000),
        # a caller's own loop on a small system
        _case("operators_16", "operators", 16, 16, 16, pairs=400, precision="reference", inverse="fp32", gate="rz",
              preconditioner="mas32", tol=1e-4),
    ]


def draw(rng):
    """Another case of the same kinds: box edges over the logarithm of the volume, odd ones among them."""
    kind = rng.choice(["step"] * 5 + ["refresh", "adjoint", "adjoint", "elements", "merge", "partition", "coarse",
                                      "operators"])
    most = {"step": 120000, "refresh": 64000, "adjoint": 32768, "elements": 250000, "merge": 110000,
            "partition": 110000, "coarse": 64000, "operators": 120000}[kind]
    volume = math.exp(rng.uniform(math.log(1500), math.log(most)))
    nx = max(5, int(round(volume ** (1 / 3) * rng.uniform(0.7, 1.4))))
    ny = max(5, int(round(math.sqrt(volume / nx) * rng.uniform(0.8, 1.25))))
    nz = max(4, int(volume / (nx * ny)))
    surface = 2 * (nx * ny + ny * nz + nx * nz)
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "pairs": int(surface * rng.choice([0, 0.3, 1.0, 2.0])),
         "E": 10 ** rng.uniform(5, 6.5), "kappa": 1e7}
    if kind in ("merge", "partition"):
        c["pairs"] = max(c["pairs"], 50)
    if kind in ("elements", "merge", "partition", "coarse"):
        return c
    mode = rng.choice(["mixed_bf16", "mixed_fp16", "reference", "reference", "cemas16"])
    if kind == "adjoint":
        mode = "reference" if c["pairs"] else rng.choice(["mixed_bf16", "reference"])
    c.update(precision="reference", inverse="fp32", gate="rz", preconditioner="mas32", tol=1e-4)
    if mode.startswith("mixed"):
        c.update(precision="mixed", inverse=mode[6:], gate="euclid")
    if mode == "cemas16":
        c.update(preconditioner="cemas16")
    if kind == "adjoint":
        if c["pairs"]:  # stiff contacts take hundreds of iterations per decade: smaller boxes
            c.update(nx=min(nx, 20), ny=min(ny, 20), nz=min(nz, 20), kappa=1e5)
            c["pairs"] = min(c["pairs"], 4 * c["nx"] * c["ny"])
        c.update(gate="euclid", tol=1e-8 if c["pairs"] else 1e-10, modulus=rng.random() < 0.5)
    if kind == "refresh" and c["precision"] == "mixed":
        c.update(matrix=rng.choice(["f32", "f32_accurate", "f32_compensated"]),
                 replacement=rng.choice(["periodic", "reliable"]))
        if c["matrix"] != "f32_accurate":
            c["replacement"] = "periodic"
    if kind == "step" and mode == "reference" and rng.random() < 0.25:
        c.update(nx=max(12, nx), ny=max(12, ny), nz=min(max(4, nz), 8), E=1e8, kappa=1e8,
                 bodies=rng.randint(20, 500), pairs=rng.randint(300, 7500))
        c["nx"], c["ny"] = min(c["nx"], 60), min(c["ny"], 60)
    return c


# ------------------------------------------------------------------ inputs --

class _Box:
    """What does not change with the seed: mesh, neighbour lists, partition, surface, and how the element triplets
    merge.  sorted_ids numbers the vertices in Morton order, as the app's METIS-sorted meshes number a part's."""

    def __init__(self, nx, ny, nz, sorted_ids):
        X, tets = synth.box_mesh(nx, ny, nz, H)
        self.bank = 16 if sorted_ids else 32
        if sorted_ids:
            pmr, _ = synth.morton_partition(X)
            order = pmr[pmr >= 0].astype(np.int64)
            new = np.empty(len(X), np.int64)
            new[order] = np.arange(len(X))
            X, tets = X[order], new[tets].astype(np.int32)
            nv = len(X)
            self.pmr = np.full((nv + 15) // 16 * 16, -1, np.int32)
            self.pmr[:nv] = np.arange(nv, dtype=np.int32)
            self.rmp = np.arange(nv, dtype=np.int32)
        else:
            self.pmr, self.rmp = synth.morton_partition(X)
        self.nv, self.nt = len(X), len(tets)
        self.start, self.num, self.lst = synth.vertex_neighbors(self.nv, tets)
        grid = np.rint(X / H).astype(np.int64)
        self.edges = np.array([nx, ny, nz])
        self.at = np.empty(self.nv, np.int64)  # vertex of each grid point
        self.at[(grid[:, 2] * ny + grid[:, 1]) * nx + grid[:, 0]] = np.arange(self.nv)
        faces = np.concatenate([tets[:, f] for f in ([1, 2, 3], [0, 3, 2], [0, 1, 3], [0, 2, 1])])
        on, axis = [], []
        for ax in range(3):
            for side in (0, self.edges[ax] - 1):
                k = np.flatnonzero((grid[faces, ax] == side).all(axis=1))
                on.append(faces[k])
                axis.append(np.full(len(k), ax))
        self.tris, self.tri_axis = np.concatenate(on).astype(np.int64), np.concatenate(axis)
        self.grid = grid
        self.X = torch.from_numpy(X).cuda()
        self.tets = torch.from_numpy(tets).cuda()
        t = self.tets.long()
        a, b = torch.tensor([p[0] for p in UPPER]).cuda(), torch.tensor([p[1] for p in UPPER]).cuda()
        r, c = t[:, a], t[:, b]
        self.swap = r > c
        self.raw_rows, self.raw_cols = torch.minimum(r, c).reshape(-1), torch.maximum(r, c).reshape(-1)
        v = torch.arange(self.nv).cuda()
        key = torch.cat([self.raw_rows * self.nv + self.raw_cols, v * self.nv + v])
        key, self.merge_perm = torch.sort(key, stable=True)
        self.keys, self.merge_len = torch.unique_consecutive(key, return_counts=True)


@functools.lru_cache(maxsize=3)
def _box(nx, ny, nz, sorted_ids):
    return _Box(nx, ny, nz, sorted_ids)


def _box_of(case):
    return _box(case["nx"], case["ny"], case["nz"], case.get("preconditioner") == "cemas16")


def _segments(values, perm, lengths):
    """Sums of equal keys in sorted order, one after another (no atomics, so inputs repeat to the bit)."""
    return torch.segment_reduce(values[perm], "sum", lengths=lengths, axis=0)


def _positions(box, gen, noise=0.1):
    return box.X + noise * H * (2 * torch.rand(box.X.shape, generator=gen, dtype=torch.float64, device="cuda") - 1)


def _lame(E):
    return E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))


def _element_values(box, x, E):
    """dt^2 V (lambda g_a g_b^T + mu g_b g_a^T + mu (g_a.g_b) I) for the 10 upper blocks of each tet, column-major."""
    t = box.tets.long()
    Ds = torch.stack([x[t[:, k]] - x[t[:, 0]] for k in (1, 2, 3)], dim=2)
    vol = torch.linalg.det(Ds).abs() / 6
    inv = torch.linalg.inv(Ds)
    g = torch.cat([-inv.sum(dim=1, keepdim=True), inv], dim=1)
    lam, mu = _lame(E)
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    out = torch.empty((box.nt, 10, 9), dtype=torch.float64, device="cuda")
    for q, (a, b) in enumerate(UPPER):
        ga, gb = g[:, a], g[:, b]
        k = lam[:, None, None] * ga[:, :, None] * gb[:, None, :] + mu[:, None, None] * gb[:, :, None] * ga[:, None, :]
        k += (mu * (ga * gb).sum(1))[:, None, None] * eye
        k *= (DT * DT * vol)[:, None, None]
        k = torch.where(box.swap[:, q, None, None], k.transpose(1, 2), k)
        out[:, q] = k.transpose(1, 2).reshape(-1, 9)
    return out.reshape(-1, 9)


def _mass_values(box):
    m = torch.zeros(box.nv, dtype=torch.float64)
    share = RHO * H ** 3 / 6 / 4
    m += torch.bincount(box.tets.reshape(-1).long().cpu(), minlength=box.nv).double() * share
    return m.cuda()[:, None] * torch.eye(3, dtype=torch.float64, device="cuda").reshape(1, 9)


def _contacts(box, rng, count, kappa):
    """Point-triangle pairs of surface vertices with triangles within two cells of the same face: the pairs in IPC's
    sign encoding and the 10 upper triplets of each projected barrier Hessian, kappa dt^2 b'' t t^T (x) n n^T.  The
    pairs belong to the case (so outputs of another seed have the same shapes), their distances and weights to `rng`."""
    want = int(count)
    pairs_rng = np.random.default_rng(want)
    pick = pairs_rng.integers(0, len(box.tris), 2 * want + 64)
    tri, ax = box.tris[pick], box.tri_axis[pick]
    off = pairs_rng.integers(-2, 3, (len(pick), 3))
    off[np.arange(len(pick)), ax] = 0
    p = np.clip(box.grid[tri[:, 0]] + off, 0, box.edges - 1)
    v = box.at[(p[:, 2] * box.edges[1] + p[:, 1]) * box.edges[0] + p[:, 0]]
    keep = np.flatnonzero((v[:, None] != tri).all(axis=1))[:want]
    tri, ax, v = tri[keep], ax[keep], v[keep]
    n = len(v)
    d = DHAT * (0.1 + 0.9 * rng.random(n))
    w = rng.dirichlet([1.0, 1.0, 1.0], n)
    t4 = np.concatenate([np.ones((n, 1)), -w], axis=1)
    b2 = -2 * np.log(d / DHAT) - 4 * (d - DHAT) / d + ((d - DHAT) / d) ** 2
    nn = np.zeros((n, 3))
    nn[np.arange(n), ax] = 1.0
    blk = (kappa * DT * DT * b2)[:, None, None] * nn[:, :, None] * nn[:, None, :]
    ids = np.concatenate([v[:, None], tri], axis=1)
    rows, cols, vals = [], [], []
    for a, b in UPPER:
        rows.append(np.minimum(ids[:, a], ids[:, b]))
        cols.append(np.maximum(ids[:, a], ids[:, b]))
        vals.append(((t4[:, a] * t4[:, b])[:, None, None] * blk).reshape(n, 9))
    pairs = np.concatenate([-v[:, None] - 1, tri], axis=1).astype(np.int32)
    st = lambda l: torch.from_numpy(np.stack(l, axis=1).reshape((10 * n,) + l[0].shape[1:])).cuda()  # noqa: E731
    return pairs, st(rows), st(cols), st(vals)


def _raw(case, seed):
    """The unmerged triplets of the system: elements, masses, contacts."""
    box = _box_of(case)
    gen = torch.Generator("cuda").manual_seed(seed)
    E = torch.full((box.nt,), float(case["E"]), dtype=torch.float64, device="cuda")
    if case.get("modulus") is not None:  # log-uniform in a decade to either side
        E = E * 10 ** (2 * torch.rand(box.nt, generator=gen, dtype=torch.float64, device="cuda") - 1)
    x = _positions(box, gen)
    vals = torch.cat([_element_values(box, x, E), _mass_values(box)])
    pairs, cr, cc, cv = _contacts(box, np.random.default_rng(seed), case["pairs"], case["kappa"])
    return box, E, vals, pairs, cr, cc, cv


def _merged(box, vals, cr, cc, cv):
    """Unique upper blocks in ascending (row, column) order."""
    base = _segments(vals, box.merge_perm, box.merge_len)
    key, perm = torch.sort(torch.cat([box.keys, cr * box.nv + cc]), stable=True)
    key, lengths = torch.unique_consecutive(key, return_counts=True)
    return ((key // box.nv).int(), (key % box.nv).int(), _segments(torch.cat([base, cv]), perm, lengths))


def _rhs(n, seed):
    gen = torch.Generator("cuda").manual_seed(seed + 7)
    return torch.randn(n, generator=gen, dtype=torch.float32, device="cuda").double()


def _system(case, seed):
    """A Newton system with its caller-side MAS inputs, values and right-hand side on the device."""
    if case.get("bodies"):
        s = synth.hybrid_system(case["bodies"], (case["nx"], case["ny"], case["nz"]), E=case["E"],
                                kappa=case["kappa"], pairs=case["pairs"], seed=int(seed))
        d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        return {"nb": s.nb, "off": s.fem_offset, "bodies": s.abd_bodies, "rows": d(s.rows), "cols": d(s.cols),
                "vals": d(s.vals), "b": d(s.b), "pairs": torch.from_numpy(np.ascontiguousarray(s.pairs)).cuda(),
                "graph": (s.fem_count, s.node_offset, s.neighbor_start, s.neighbor_num, s.neighbor_list,
                          s.part_map_real, s.real_map_part)}
    box, E, vals, pairs, cr, cc, cv = _raw(case, seed)
    rows, cols, v = _merged(box, vals, cr, cc, cv)
    return {"nb": box.nv, "off": 0, "bodies": 0, "rows": rows, "cols": cols, "vals": v,
            "b": _rhs(3 * box.nv, seed), "pairs": torch.from_numpy(pairs).cuda(),
            "graph": (box.nv, 0, box.start, box.num, box.lst, box.pmr, box.rmp)}


def _handle(case):
    return MasPcg(tolerance=case["tol"], gate=case["gate"], precision=case["precision"], inverse=case["inverse"],
                  preconditioner=case["preconditioner"], matrix=case.get("matrix", "f32"),
                  replacement=case.get("replacement", "periodic"), max_iter_ratio=3.0)


def _on_torch_stream(m):
    """A torch stream of its own that the handle runs on too, so torch's work and the library's are ordered."""
    stream = torch.cuda.Stream()
    m.set_stream(stream.cuda_stream)
    return stream


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _rest(box, gen):
    """Per-tet rest data as the element kernel takes them (fem.rest_data on the device), a modulus per tet."""
    t = box.tets.long()
    Dm = torch.stack([box.X[t[:, k]] - box.X[t[:, 0]] for k in (1, 2, 3)], dim=2)
    E = 10 ** (4 + 2 * torch.rand(box.nt, generator=gen, dtype=torch.float64, device="cuda"))
    lam, mu = _lame(E)
    return (torch.linalg.inv(Dm).reshape(-1, 9).contiguous(), torch.linalg.det(Dm).abs() / 6, 4 * mu / 3,
            lam + 5 * mu / 6)


def _aggregates(box):
    """2x2x2 vertex cubes, alternately affine (four blocks) and translational (one)."""
    g = box.grid // 2
    e = (box.edges + 1) // 2
    owner = ((g[:, 2] * e[1] + g[:, 1]) * e[0] + g[:, 0]).astype(np.int32)
    _, owner = np.unique(owner, return_inverse=True)
    count = int(owner.max()) + 1
    masks = np.where(np.arange(count) % 2 == 0, 15, 1).astype(np.int32)
    width = np.where(masks == 15, 4, 1)
    bases = np.concatenate([[0], np.cumsum(width)[:-1]]).astype(np.int32)
    return owner.astype(np.int32), bases, masks, int(width.sum())


# ----------------------------------------------------------------- prepare --

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "refresh", "operators"):
        s = _system(case, seed)
        m = _handle(case)
        m.set_graph(*s["graph"])
        s.update(kind=kind, m=m, x=torch.zeros_like(s["b"]), z=torch.zeros_like(s["b"]))
        if kind != "step":
            m.set_contacts(s["pairs"])
            m.set_matrix(s["vals"], s["rows"], s["cols"], s["nb"], s["off"], s["bodies"])
            m.build()
        if kind == "refresh":  # the values of the next Newton step
            gen = torch.Generator("cuda").manual_seed(seed + 99)
            scale = 1 + 0.1 * torch.rand((), generator=gen, dtype=torch.float64, device="cuda")
            s["vals"] = s["vals"] * scale
        return s
    if kind == "adjoint":
        box, E, vals, pairs, cr, cc, cv = _raw(case, seed)
        m = _handle(case)
        m.set_graph(box.nv, 0, box.start, box.num, box.lst, box.pmr, box.rmp)
        m.set_contacts(pairs)
        if case["modulus"]:
            v = torch.arange(box.nv).cuda()
            rows = torch.cat([box.raw_rows, v, cr]).int()
            cols = torch.cat([box.raw_cols, v, cc]).int()
            vals = torch.cat([vals, cv])
        else:
            rows, cols, vals = _merged(box, vals, cr, cc, cv)
        b = _rhs(3 * box.nv, seed)
        return {"kind": kind, "m": m, "E": E, "vals": vals, "rows": rows, "cols": cols, "b": b, "nb": box.nv,
                "target": 0.1 * _rhs(3 * box.nv, seed + 1), "modulus": case["modulus"]}
    box = _box_of(case)
    m = MasPcg()
    if kind == "elements":
        gen = torch.Generator("cuda").manual_seed(seed)
        x = _positions(box, gen, 0.2).reshape(-1)
        rest = _rest(box, gen)
        n = 10 * box.nt
        return {"kind": kind, "m": m, "stream": _on_torch_stream(m), "tets": box.tets, "x": x, "rest": rest,
                "nt": box.nt, "nv": box.nv, "grad": torch.zeros(3 * box.nv, dtype=torch.float64, device="cuda"),
                "rows": torch.zeros(n, dtype=torch.int32, device="cuda"),
                "cols": torch.zeros(n, dtype=torch.int32, device="cuda"),
                "vals": torch.zeros((n, 9), dtype=torch.float64, device="cuda")}
    _, E, vals, pairs, cr, cc, cv = _raw(case, seed)
    if kind == "merge":
        v = torch.arange(box.nv).cuda()
        return {"kind": kind, "m": m, "rows": torch.cat([box.raw_rows, v, cr]).int(),
                "cols": torch.cat([box.raw_cols, v, cc]).int(), "vals": torch.cat([vals, cv])}
    if kind == "partition":
        gen = torch.Generator("cuda").manual_seed(seed + 3)
        types = torch.randint(0, 4, (len(cr),), generator=gen, device="cuda")
        return {"kind": kind, "m": m, "rows": cr.int(), "cols": cc.int(), "vals": cv, "types": types}
    rows, cols, v = _merged(box, vals, cr, cc, cv)
    owner, bases, masks, blocks = _aggregates(box)
    keep = [torch.from_numpy(a).cuda() for a in (owner, bases, masks)] + [box.X.contiguous()]
    g = native.GalerkinMap(*[_ptr(t) for t in keep], 0, box.nv, len(bases), blocks)
    cap = 16 * len(rows)
    return {"kind": kind, "m": m, "stream": _on_torch_stream(m), "map": g, "keep": keep, "rows": rows, "cols": cols,
            "vals": v, "b": _rhs(3 * box.nv, seed), "xc": _rhs(3 * blocks, seed + 5), "cap": cap,
            "crows": torch.zeros(cap, dtype=torch.int32, device="cuda"),
            "ccols": torch.zeros(cap, dtype=torch.int32, device="cuda"),
            "cvals": torch.zeros((cap, 9), dtype=torch.float64, device="cuda"),
            "bc": torch.zeros(3 * blocks, dtype=torch.float64, device="cuda"),
            "xf": torch.zeros(3 * box.nv, dtype=torch.float64, device="cuda")}


# --------------------------------------------------------------------- run --

def run(s):
    kind, m = s["kind"], s["m"]
    if kind == "step":
        m.set_contacts(s["pairs"])
        m.set_matrix(s["vals"], s["rows"], s["cols"], s["nb"], s["off"], s["bodies"])
        m.build()
        m.solve(s["b"], s["x"])
        return {"x": s["x"]}
    if kind == "refresh":
        m.refresh_values(s["vals"])
        m.solve(s["b"], s["x"])
        return {"x": s["x"]}
    if kind == "operators":
        return {"y": m.spmv(s["b"], y=s["x"]), "z": m.apply_preconditioner(s["b"], s["z"])}
    if kind == "adjoint":
        b = s["b"].detach().requires_grad_(True)
        if s["modulus"]:
            p = s["E"].detach().requires_grad_(True)
            x = autograd.newton_solve_modulus(p, b, s["vals"], m, s["rows"], s["cols"], s["nb"])
        else:
            p = s["vals"].detach().requires_grad_(True)
            x = autograd.newton_solve(p, b, m, s["rows"], s["cols"], s["nb"])
        ((x - s["target"]) ** 2).sum().backward()
        return {"x": x.detach(), "grad": p.grad, "grad_b": b.grad}
    if kind == "elements":
        with torch.cuda.stream(s["stream"]):
            s["grad"].zero_()
            native.check(m.lib.maspcg_fem_snk1_gradient_hessian(
                m.h, s["nt"], _ptr(s["tets"]), s["nv"], _ptr(s["x"]), *[_ptr(t) for t in s["rest"]], DT, 0,
                _ptr(s["grad"]), _ptr(s["rows"]), _ptr(s["cols"]), _ptr(s["vals"])), m.h)
        return {"grad": s["grad"], "rows": s["rows"], "cols": s["cols"], "vals": s["vals"]}
    if kind == "merge":
        r, c, v = m.convert_bcoo(s["rows"], s["cols"], s["vals"])
        return {"rows": r, "cols": c, "vals": v}
    if kind == "partition":
        r, c, v, k = m.partition_contact_triplets(s["rows"], s["cols"], s["vals"], s["types"])
        return {"rows": r, "cols": c, "vals": v, "counts": k}
    n = ctypes.c_int()
    with torch.cuda.stream(s["stream"]):
        native.check(m.lib.maspcg_galerkin_coarse_matrix(
            m.h, ctypes.byref(s["map"]), _ptr(s["vals"]), _ptr(s["rows"]), _ptr(s["cols"]), len(s["rows"]),
            _ptr(s["cvals"]), _ptr(s["crows"]), _ptr(s["ccols"]), s["cap"], ctypes.byref(n)), m.h)
        native.check(m.lib.maspcg_galerkin_restrict(m.h, ctypes.byref(s["map"]), _ptr(s["b"]), _ptr(s["bc"])), m.h)
        native.check(m.lib.maspcg_galerkin_prolong(m.h, ctypes.byref(s["map"]), _ptr(s["xc"]), _ptr(s["xf"])), m.h)
    k = n.value
    return {"rows": s["crows"][:k], "cols": s["ccols"][:k], "vals": s["cvals"][:k], "bc": s["bc"], "xf": s["xf"]}


# ------------------------------------------------- work, tolerance, exact --

def work(case):
    """Inputs read once and outputs written once.  The iterations of a solve come on top: their number depends on the
    values, and every one of them reads the matrix and the preconditioner again where these do not fit on the chip."""
    nv = case["nx"] * case["ny"] * case["nz"]
    nt = 6 * (case["nx"] - 1) * (case["ny"] - 1) * (case["nz"] - 1)
    blocks = 8 * nv + 10 * case["pairs"]          # merged upper blocks, about
    raw = 10 * nt + nv + 10 * case["pairs"]
    kind = case["kind"]
    if kind in ("step", "refresh", "operators"):
        return {"bytes": 80 * blocks + 2 * 24 * nv + 24 * nv, "flops": 2 * 9 * 2 * blocks}
    if kind == "adjoint":
        b = raw if case["modulus"] else blocks
        return {"bytes": 80 * b + (16 * nt if case["modulus"] else 72 * b) + 4 * 24 * nv, "flops": 4 * 9 * 2 * b}
    if kind == "elements":
        return {"bytes": nt * (16 + 72 + 24 + 800) + 2 * 24 * nv, "flops": 2000 * nt}
    if kind == "merge":
        return {"bytes": 80 * (raw + blocks), "flops": 9 * raw}
    if kind == "partition":
        return {"bytes": 10 * case["pairs"] * (80 + 80 + 8), "flops": 0}
    return {"bytes": 80 * blocks + 80 * blocks + 4 * 24 * nv, "flops": 18 * 7 * blocks}


def tolerance(case):
    """About four times what a change of rounding was seen to move the outputs by (other inverse storage, other sums, a
    right-hand side perturbed by 1e-7)."""
    kind = case["kind"]
    if kind == "elements":
        return {"rel": 2e-14, "max": 1e-11}
    if kind in ("merge", "partition", "coarse"):
        return {"rel": 1e-14}       # FP64 sums in another order; whole numbers the same
    if kind == "operators":
        return {"rel": 1e-5}        # the apply runs on FP32 inverses and vectors
    if kind == "adjoint":
        return {"rel": 200 * case["tol"]}
    # a stopped iterate: the r.z gate of the reference stops far from the solution, where one iteration more or less
    # moves x by 3e-3; at the FP64-verified gate it moves it by about the tolerance
    return {"rel": 1.5e-2, "max": 0.3} if case["gate"] == "rz" else {"rel": 5e-4, "max": 2e-2}


def _full(rows, cols, vals, nb):
    """y = A x of upper blocks (repeats add) as a torch CSR matrix in 64 bits."""
    r, c = rows.long(), cols.long()
    v = vals.reshape(-1, 3, 3).transpose(1, 2)  # [block, i, j]
    off = r != c
    R = torch.cat([r, c[off]])
    C = torch.cat([c, r[off]])
    V = torch.cat([v, v[off].transpose(1, 2)])
    key, perm = torch.sort(R * nb + C, stable=True)
    key, lengths = torch.unique_consecutive(key, return_counts=True)
    V = _segments(V.reshape(-1, 9), perm, lengths).reshape(-1, 3, 3)
    R, C = key // nb, key % nb
    per_row = torch.bincount(R, minlength=nb)
    first = torch.cumsum(per_row, 0) - per_row
    rank = torch.arange(len(key), device="cuda") - first[R]
    i = torch.arange(3, device="cuda")
    crow = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), torch.cumsum((3 * per_row).repeat_interleave(3), 0)])
    at = crow[(3 * R)[:, None] + i][:, :, None] + (3 * rank)[:, None, None] + i[None, None, :]
    col = torch.empty(9 * len(key), dtype=torch.long, device="cuda")
    val = torch.empty(9 * len(key), dtype=torch.float64, device="cuda")
    col[at] = (3 * C)[:, None, None] + i[None, None, :].expand(1, 3, 3)
    val[at] = V
    diag = torch.zeros((nb, 3, 3), dtype=torch.float64, device="cuda")
    d = R == C
    diag[R[d]] = V[d]
    return torch.sparse_csr_tensor(crow, col, val, (3 * nb, 3 * nb)), torch.linalg.inv(diag)


def _cg(A, minv, b, tol=1e-14, most=20000):
    """Block-Jacobi conjugate gradients in 64 bits, restarted from the true residual."""
    x = torch.zeros_like(b)
    stop = tol * b.norm()
    pre = lambda r: torch.einsum("nij,nj->ni", minv, r.reshape(-1, 3)).reshape(-1)  # noqa: E731
    done = 0
    for _ in range(4):
        r = b - A @ x
        if r.norm() <= stop:
            break
        z = pre(r)
        p, rz = z.clone(), r @ z
        while done < most:
            for _ in range(50):
                q = A @ p
                a = rz / (p @ q)
                x += a * p
                r -= a * q
                z = pre(r)
                new = r @ z
                p = z + (new / rz) * p
                rz = new
            done += 50
            if not r.norm() > stop:
                break
    return x


def _exact_elements(s):
    """The exact 9x9 Hessian in F, projected by a full eigendecomposition, and the gradient, in 64 bits."""
    box_t = s["tets"].long()
    x = s["x"].reshape(-1, 3)
    Di, vol, u, r = s["rest"]
    Di = Di.reshape(-1, 3, 3)
    eps = torch.zeros((3, 3, 3), dtype=torch.float64, device="cuda")
    for a, b, c in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        eps[a, b, c], eps[a, c, b] = 1.0, -1.0
    two = torch.einsum("ikm,jln->ijklmn", eps, eps).reshape(81, 9)
    grad = torch.zeros_like(x)
    vals = torch.empty((s["nt"], 10, 9), dtype=torch.float64, device="cuda")
    for lo in range(0, s["nt"], 10000):  # batches that the eigensolver takes
        hi = min(lo + 10000, s["nt"])
        t, D = box_t[lo:hi], Di[lo:hi]
        scale = DT * DT * vol[lo:hi]
        uu, rr = u[lo:hi], r[lo:hi]
        F = torch.stack([x[t[:, k]] - x[t[:, 0]] for k in (1, 2, 3)], dim=2) @ D
        g = torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]),
                         torch.linalg.cross(F[:, 0], F[:, 1])], dim=1)
        J = (F[:, 0] * g[:, 0]).sum(1)
        k = rr * (J - 1) - uu
        Hf = rr[:, None, None] * g.reshape(-1, 9, 1) * g.reshape(-1, 1, 9)
        Hf += k[:, None, None] * (F.reshape(-1, 9) @ two.T).reshape(-1, 9, 9)
        Hf += uu[:, None, None] * torch.eye(9, dtype=torch.float64, device="cuda")
        w, Q = torch.linalg.eigh(Hf)
        Hf = (Q * w.clamp(min=0)[:, None, :]) @ Q.transpose(1, 2)
        cf = torch.cat([-D.sum(dim=1, keepdim=True), D], dim=1)
        P = uu[:, None, None] * F + k[:, None, None] * g
        f = scale[:, None, None] * torch.einsum("taj,tij->tai", cf, P)
        grad.index_put_((t.reshape(-1),), f.reshape(-1, 3), accumulate=True)
        Hf = Hf.reshape(-1, 3, 3, 3, 3)
        for q, (a, b) in enumerate(UPPER):
            K = scale[:, None, None] * torch.einsum("tj,tijkl,tl->tik", cf[:, a], Hf, cf[:, b])
            K = torch.where((t[:, a] > t[:, b])[:, None, None], K.transpose(1, 2), K)
            vals[lo:hi, q] = K.transpose(1, 2).reshape(-1, 9)
    return {"grad": grad.reshape(-1), "rows": None, "cols": None, "vals": vals.reshape(-1, 9)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "refresh"):
        return None
    s = prepare(case, seed)
    if kind == "operators":
        A, _ = _full(s["rows"], s["cols"], s["vals"], s["nb"])
        return {"y": A @ s["b"], "z": None}
    if kind == "adjoint":
        A, minv = _full(s["rows"], s["cols"], s["vals"], s["nb"])
        x = _cg(A, minv, s["b"])
        lam = _cg(A, minv, 2 * (x - s["target"]))
        r, c = s["rows"].long(), s["cols"].long()
        X, L = x.reshape(-1, 3), lam.reshape(-1, 3)
        g = -L[r][:, :, None] * X[c][:, None, :]
        g -= torch.where((r != c)[:, None, None], X[r][:, :, None] * L[c][:, None, :], torch.zeros_like(g))
        g = g.transpose(1, 2).reshape(-1, 9)
        if s["modulus"]:
            nt = len(s["E"])
            g = (g[:10 * nt] * s["vals"][:10 * nt]).sum(1).reshape(nt, 10).sum(1) / s["E"]
        return {"x": x, "grad": g, "grad_b": lam}
    if kind == "elements":
        return _exact_elements(s)
    if kind == "merge":
        key = s["rows"].long() * (1 << 31) + s["cols"].long()
        key, perm = torch.sort(key, stable=True)
        key, lengths = torch.unique_consecutive(key, return_counts=True)
        return {"rows": (key >> 31).int(), "cols": (key & ((1 << 31) - 1)).int(),
                "vals": _segments(s["vals"], perm, lengths)}
    if kind == "partition":
        p = torch.argsort(s["types"], stable=True)
        return {"rows": s["rows"][p], "cols": s["cols"][p], "vals": s["vals"][p],
                "counts": torch.bincount(s["types"], minlength=4).int().cpu()}
    return {"rows": None, "cols": None, "vals": None, **_exact_transfer(s)}


def _exact_transfer(s):
    owner, bases, masks, X = s["keep"]
    one = torch.ones((len(X), 1), dtype=torch.float64, device="cuda")
    phi = torch.cat([one, X], dim=1)
    affine = (masks == 15)[owner.long()]
    base = bases.long()[owner.long()]
    bc = torch.zeros((len(s["xc"]) // 3, 3), dtype=torch.float64, device="cuda")
    xc, b = s["xc"].reshape(-1, 3), s["b"].reshape(-1, 3)
    xf = torch.zeros_like(b)
    for a in range(4):
        k = torch.arange(len(X), device="cuda") if a == 0 else torch.nonzero(affine)[:, 0]
        bc.index_put_((base[k] + a,), phi[k, a, None] * b[k], accumulate=True)
        xf[k] += phi[k, a, None] * xc[base[k] + a]
    return {"bc": bc.reshape(-1), "xf": xf.reshape(-1)}
