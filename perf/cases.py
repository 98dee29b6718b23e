"""Timing cases of the mesh stage, through the library's public entry points.

A pass takes sphere rows (or PDB text) from host memory to a finished mesh in
host memory, as a program that meshes one structure after another does; an
open device, the warm-start model and a tuned batch configuration are what
such a program keeps between structures.  The inputs are the seeded synthetic
globules of `sesmesh_b200.workloads` (protein-like packing, C/N/O/S Bondi
radii) and its assemblies.

A case is a dict:
  path      "mesh" (compute_surface), "warm" (SurfaceEngine with the learned
            warm start), "batch" (MultiBatch) or "text" (PDB text to OBJ text)
  shape     "globule", "rings" (21 copies on rings) or "shell" (60 copies on
            an icosahedral shell)
  n         spheres (the largest structure's, for a batch); per copy for
            assemblies
  kind, probe, spacing, refine, brick: the fields of SurfaceParams
  count     structures of a batch
"""
import math

import numpy as np
import torch

from sesmesh_b200 import native, structure, surface, warm_start, workloads


def _case(name, **more):
    c = dict(path="mesh", shape="globule", n=330, kind="ses", probe=1.4, spacing=0.5, refine="exact", brick=10,
             count=1)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A ligand at the default spacing and mode: the smallest call, where latency counts.
        _case("ligand43_exact_h050", n=43),
        # A peptide or small domain at the default settings (the test suite's globule).
        _case("peptide331_exact_h050", n=331),
        # A small protein's van der Waals surface, fast mode, odd spacing.
        _case("vdw1201_fast_h035", n=1201, kind="vdw", probe=0.0, spacing=0.35, refine="fast"),
        # A protein chain at Quality::High, in both refinement modes.
        _case("protein2803_exact_h025", n=2803, spacing=0.25),
        _case("protein2803_fast_h025", n=2803, spacing=0.25, refine="fast"),
        # A protein at the finest spacing in use (figures, docking grids).
        _case("protein4999_fast_h010", n=4999, probe=1.3, spacing=0.1, refine="fast"),
        # A complex's solvent-accessible surface at the default spacing, just below the size whose
        # arrangement is built on the device.
        _case("sas16001_exact_h050", n=16001, kind="sas"),
        # A large assembly at Quality::High: exact, and fast from the learned warm start.
        _case("rings58800_exact_h025", shape="rings", n=2800, spacing=0.25),
        _case("rings58800_warm_h025", path="warm", shape="rings", n=2800, spacing=0.25, refine="fast"),
        # A virus-like shell of 2.4 M atoms at 1 A: the largest structure.
        _case("shell2400k_fast_h100", shape="shell", n=40000, spacing=1.0, refine="fast"),
        # A service's small batch of mixed sizes and spacings in one device pass.
        _case("batch10_fast", path="batch", n=5000, count=10, refine="fast", brick=16),
        # The command line's work: read PDB text, mesh, write OBJ text.
        _case("text5003_exact_h050", path="text", n=5003),
    ]


def _cost(n, spacing):
    """Grid points of a pass, up to a factor (surface bricks grow with area / spacing^2.4 in this range)."""
    return n * (0.25 / spacing) ** 2.4


def draw(rng):
    path = rng.choice(["mesh", "mesh", "mesh", "mesh", "warm", "warm", "batch", "text"])
    kind = "ses" if path != "mesh" else rng.choice(["ses", "ses", "ses", "ses", "sas", "vdw"])
    probe = 0.0 if kind == "vdw" else round(rng.uniform(1.2, 1.6), 3)
    if path == "batch":
        return _case(None, path="batch", n=rng.randint(60, 5000), count=rng.randint(3, 10), refine="fast",
                     brick=rng.choice([8, 16]))
    n = int(round(math.exp(rng.uniform(math.log(20), math.log(60000 if path != "text" else 9000)))))
    spacing = round(math.exp(rng.uniform(math.log(0.1), 0.0)), 3)
    while _cost(n, spacing) > 6e4:
        spacing = round(spacing * 1.3, 3)
    shape = "globule"
    if n > 6000 and path != "text":
        # Assemblies of 21 or 60 copies (a single chain of this size is not met).
        shape = rng.choice(["rings", "shell"])
        n = n // (21 if shape == "rings" else 60)
        spacing = max(spacing, 0.2)
    refine = "fast" if path == "warm" else rng.choice(["exact", "fast"]) if path == "mesh" else "exact"
    return _case(None, path=path, shape=shape, n=n, kind=kind, probe=probe, spacing=spacing, refine=refine,
                 brick=rng.choice([10, 10, 10, 8, 16]) if path == "mesh" else 10)


def _moved(spheres, step, rng, reach=40):
    """The spheres in another order, moved by up to `reach` whole lattice steps: other coordinates, another
    brick partition and other vertex and triangle orders, with the same numbers of vertices and triangles.
    Coordinates have the three decimals of a PDB file."""
    out = spheres[rng.permutation(len(spheres))]
    out[:, :3] = np.round(np.round(out[:, :3], 3) + rng.integers(-reach, reach + 1, 3) * step, 3)
    return out


def _spheres(case, seed):
    """The case's structure (its own walk seed), placed by the seed."""
    own = 1000 + case["n"]
    if case["shape"] == "rings":
        s = workloads.rings58800(own, case["n"])["spheres"]
    elif case["shape"] == "shell":
        s = workloads.shell2400k(own, case["n"])["spheres"]
    else:
        s = workloads.globule(own, case["n"])
    rng = np.random.default_rng(seed)
    if case["path"] == "text":
        # Whole bricks, all coordinates in 100..999: the OBJ text then has one length for every seed.
        brick = case["brick"] * case["spacing"]
        out = _moved(s, brick, rng, reach=int(300 / brick))
        out[:, :3] = np.round(out[:, :3] + math.ceil(550 / brick) * brick, 3)
        return out
    return _moved(s, case["spacing"], rng)


def _params(case):
    p = surface.SurfaceParams(probe_radius=case["probe"], spacing=case["spacing"], refine=case["refine"],
                              brick_size=case["brick"], kind=case["kind"])
    return p


def _batch_items(case, seed):
    """(spheres, probe, spacing) of a batch: sizes log-uniform from 20 to n, as `workloads.batch512` has them."""
    own = np.random.default_rng(case["n"])
    rng = np.random.default_rng(seed)
    items = []
    for k in range(case["count"]):
        # Stratified, so that batches of one size do similar work.
        u = (k + own.uniform(0.3, 0.7)) / case["count"]
        n = int(round(math.exp(math.log(20) + u * math.log(case["n"] / 20))))
        spacing = [0.25, 0.5, 0.1][k % 3]
        s = workloads.globule(case["n"] * 1009 + k, n)
        items.append((_moved(s, spacing, rng), round(float(own.uniform(1.2, 1.4)), 3), spacing))
    return items


_ATOMS = {1.7: " C", 1.55: " N", 1.52: " O", 1.8: " S"}


def _pdb_text(spheres):
    lines = []
    for k, (x, y, z, r) in enumerate(spheres):
        e = _ATOMS[round(float(r), 2)]
        lines.append("ATOM  %5d %s%-2s ALA %s%4d    %8.3f%8.3f%8.3f  1.00  0.00          %s  \n"
                     % (k + 1, e, "", "ABCDEFGH"[k // 9999 % 8], k % 9999 + 1, x, y, z, e))
    return "".join(lines).encode() + b"END\n"


def prepare(case, seed):
    dev = surface._device(0)
    state = dict(case=case, path=case["path"])
    if case["path"] == "batch":
        items = _batch_items(case, seed)
        state["structures"] = [(s, surface.SurfaceParams(probe_radius=p, spacing=h, refine="fast"))
                               for s, p, h in items]
        return state
    state["params"] = _params(case)
    state["spheres"] = _spheres(case, seed)
    if case["path"] == "text":
        state["text"] = _pdb_text(state.pop("spheres"))
    if case["path"] == "warm":
        state["mlp"] = native.Mlp(dev, warm_start.load())
    return state


def _mesh_arrays(out):
    return dict(positions=out.positions, normals=out.normals, triangles=out.triangles, vertex_atom=out.vertex_atom,
                vertex_patch=out.vertex_patch, vertex_component=out.vertex_component)


def _mesh_result(out):
    r = _mesh_arrays(out)
    r["area"], r["volume"] = out.stats["area"], out.stats["volume"]
    return r


def run(state):
    path = state["path"]
    if path == "mesh":
        return _mesh_result(surface.compute_surface(state["spheres"], state["params"]))
    if path == "warm":
        eng = surface.SurfaceEngine(state["spheres"], state["params"])
        eng.set_warm_start(state["mlp"])
        out = eng.mesh()
        eng.close()
        return _mesh_result(out)
    if path == "text":
        spheres = structure.read_bytes(state["text"], "pdb")
        out = surface.compute_surface(spheres, state["params"])
        r = _mesh_result(out)
        r["obj"] = np.frombuffer(out.obj(), np.uint8)
        return r
    batch = surface.MultiBatch(state["structures"], config=(state["case"]["brick"], 0, 4))
    batch.run()
    meshes = [_mesh_arrays(batch.surface(i)) for i in range(batch.n)]
    batch.close()
    return meshes


def work(case):
    """Spheres read and the mesh written once; per vertex the two end samples of its edge and 2.2 evaluations of
    the root search, each an f32 or f64 walk over some 30 candidates (300 operations)."""
    if case["path"] == "batch":
        sizes = [(20 * (case["n"] / 20) ** ((k + 0.5) / case["count"]), [0.25, 0.5, 0.1][k % 3])
                 for k in range(case["count"])]
    else:
        copies = {"globule": 1, "rings": 21, "shell": 60}[case["shape"]]
        sizes = [(case["n"], case["spacing"])] * copies
    spheres = vertices = 0.0
    for n, h in sizes:
        spheres += n
        # SES area about 13.5 n^0.92 A^2 (protein-like packing); about 1.5 crossing edges per h^2.  A SAS
        # keeps the outer boundary only, a van der Waals surface every atom's.
        area = {"ses": 13.5 * n ** 0.92, "sas": 30.0 * n ** 0.73, "vdw": 13.5 * n}[case["kind"]]
        vertices += 1.5 * area / (h * h)
    per_vertex = 12 + 12 + 4 + 1 + 4 + 2 * 12
    return {"bytes": 32.0 * spheres + per_vertex * vertices, "flops": vertices * (2 + 2.2) * 300.0}


# ---- the mesh vertices in 64 bits, from the definition of the surface ------------------------------------------

_BAND = 4.0   # how far beyond the probe the nearest boundary point is looked for, in spacings


class _SphereField:
    """F(x) = min |x - c| - R (van der Waals or solvent-accessible surface)."""

    def __init__(self, c, R):
        self.c, self.R = c, R

    def __call__(self, x):
        """Values and outward unit normals at x (m, 3)."""
        value = torch.empty(len(x), dtype=x.dtype, device=x.device)
        near = torch.empty(len(x), dtype=torch.long, device=x.device)
        step = max(1, 30_000_000 // len(self.c))
        for a in range(0, len(x), step):
            d = torch.cdist(x[a:a + step], self.c, compute_mode="donot_use_mm_for_euclid_dist") - self.R
            value[a:a + step], near[a:a + step] = d.min(1)
        n = x - self.c[near]
        return value, n / n.norm(dim=1, keepdim=True)

    def undecided(self, x):
        return None


class _SolventExcluded:
    """F(x) = probe - distance from x to the boundary of the union of expanded balls (probe outside the union)."""

    def __init__(self, c, r, probe, cap):
        self.c, self.R, self.probe, self.reach = c, r + probe, probe, probe + cap
        n, R = len(c), self.R
        d = torch.cdist(c, c, compute_mode="donot_use_mm_for_euclid_dist")
        i, j = torch.nonzero(torch.triu(d < R[:, None] + R[None, :], 1), as_tuple=True)
        u = (c[j] - c[i]) / d[i, j][:, None]
        t = (d[i, j] ** 2 + R[i] ** 2 - R[j] ** 2) / (2 * d[i, j])
        rho2 = R[i] ** 2 - t ** 2
        ok = rho2 > 0
        self.i, self.j, self.u, self.rho = i[ok], j[ok], u[ok], rho2[ok].sqrt()
        self.o = c[self.i] + u[ok] * t[ok][:, None]
        # Triple points: circle (i, j) against sphere k > j.
        pts = []
        for a in range(0, len(self.i), 2000):
            o, axis, rho, jj = (v[a:a + 2000] for v in (self.o, self.u, self.rho, self.j))
            ii = self.i[a:a + 2000]
            w = c[None] - o[:, None]                                   # (m, n, 3)
            along = (w * axis[:, None]).sum(2)
            flat = w - along[..., None] * axis[:, None]
            fl = flat.norm(dim=2)
            # Points at angle +-g from the direction of k in the circle's plane.
            cosg = (rho[:, None] ** 2 + (w * w).sum(2) - R[None] ** 2) / (2 * rho[:, None] * fl.clamp_min(1e-300))
            m, k = torch.nonzero((cosg.abs() < 1) & (torch.arange(n, device=c.device)[None] > jj[:, None]),
                                 as_tuple=True)
            e1 = flat[m, k] / fl[m, k][:, None]
            e2 = torch.cross(axis[m], e1, dim=1)
            g = cosg[m, k]
            s = (1 - g * g).sqrt()
            for sign in (1.0, -1.0):
                q = o[m] + rho[m][:, None] * (e1 * g[:, None] + sign * e2 * s[:, None])
                pts.append(q[self._clear(q, ii[m], jj[m], k)])
        self.v = torch.cat(pts) if pts else c[:0]

    def _clear(self, q, *own):
        """Whether q (m, 3) lies in none of the balls but those named (which it lies on)."""
        out = torch.ones(len(q), dtype=torch.bool, device=q.device)
        step = max(1, 10_000_000 // len(self.c))
        for a in range(0, len(q), step):
            d = torch.cdist(q[a:a + step], self.c, compute_mode="donot_use_mm_for_euclid_dist")
            blocked = d < self.R - 1e-9
            for o in own:
                blocked.scatter_(1, o[a:a + step, None], False)
            out[a:a + step] = ~blocked.any(1)
        return out

    def undecided(self, x):
        """Nodes whose sign the balls alone do not decide (and the sign of the others)."""
        sas, _ = _SphereField(self.c, self.R)(x)
        vdw, _ = _SphereField(self.c, self.R - self.probe)(x)
        return (sas < 0) & (vdw >= 0), vdw < 0

    def __call__(self, x):
        dist = torch.full((len(x),), self.reach, dtype=x.dtype, device=x.device)
        close = x.clone()
        inside = torch.zeros(len(x), dtype=torch.bool, device=x.device)
        step = max(1, 6_000_000 // max(len(self.i), len(self.v), len(self.c)))
        for a in range(0, len(x), step):
            y = x[a:a + step]
            found = []
            d = torch.cdist(y, self.c, compute_mode="donot_use_mm_for_euclid_dist")
            inside[a:a + step] = (d < self.R).any(1)
            m, k = torch.nonzero(((d - self.R).abs() < self.reach) & (d > 1e-12), as_tuple=True)
            q = self.c[k] + (y[m] - self.c[k]) * (self.R[k] / d[m, k])[:, None]
            ok = self._clear(q, k)
            found.append((m[ok], q[ok]))
            w = y[:, None] - self.o[None]
            along = (w * self.u[None]).sum(2)
            w -= along[..., None] * self.u[None]
            wl = w.norm(dim=2)
            dc = (along ** 2 + (wl - self.rho) ** 2).sqrt()
            m, k = torch.nonzero((dc < self.reach) & (wl > 1e-12), as_tuple=True)
            q = self.o[k] + w[m, k] * (self.rho[k] / wl[m, k])[:, None]
            ok = self._clear(q, self.i[k], self.j[k])
            found.append((m[ok], q[ok]))
            if len(self.v):
                dv = torch.cdist(y, self.v, compute_mode="donot_use_mm_for_euclid_dist")
                at, k = dv.min(1)
                m = torch.nonzero(at < self.reach)[:, 0]
                found.append((m, self.v[k[m]]))
            m, q = torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])
            if not len(m):
                continue
            dq = (q - y[m]).norm(dim=1)
            best = torch.full((len(y),), self.reach, dtype=x.dtype, device=x.device)
            best.scatter_reduce_(0, m, dq, "amin")
            hit = dq <= best[m]
            dist[a:a + step] = best
            close[a + m[hit]] = q[hit]
        value = torch.where(inside, self.probe - dist, torch.full_like(dist, self.probe))
        n = close - x
        return value, n / n.norm(dim=1, keepdim=True).clamp_min(1e-300)


def exact(case, seed):
    """Vertices (the roots of F on the lattice's crossing edges, bricks in (z, y, x) order and edges in lattice
    order within a brick) and normals in 64 bits.  The other outputs are whole numbers or follow from the
    triangulation.  None for structures too large for this direct search."""
    if case["path"] != "mesh" or case["shape"] != "globule":
        return None
    if case["kind"] == "ses" and case["n"] * (0.5 / case["spacing"]) ** 2 > 400:
        return None
    if case["kind"] != "ses" and case["n"] ** 2 * (0.5 / case["spacing"]) ** 3 > 1e7:
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    s = torch.from_numpy(_spheres(case, seed)).to(device)
    c, r, h, b = s[:, :3].contiguous(), s[:, 3].contiguous(), case["spacing"], case["brick"]
    big = r + case["probe"]
    field = _SolventExcluded(c, r, case["probe"], _BAND * h) if case["kind"] == "ses" else _SphereField(c, big)
    lo = torch.floor((c - big[:, None]).min(0).values / h).long() - 2
    hi = torch.ceil((c + big[:, None]).max(0).values / h).long() + 2
    axes = [torch.arange(int(lo[k]), int(hi[k]) + 1, device=device) for k in range(3)]
    dims = [len(a) for a in axes]
    negative = torch.empty(dims[0] * dims[1] * dims[2], dtype=torch.bool, device=device)
    layer = dims[1] * dims[2]
    for k in range(dims[0]):  # one x layer of nodes at a time
        g = torch.stack(torch.meshgrid(axes[0][k:k + 1], axes[1], axes[2], indexing="ij"), -1).reshape(-1, 3)
        x = g.double() * h
        mask = field.undecided(x)
        if mask is None:
            neg = field(x)[0].float() < 0
        else:
            neg = mask[1].clone()
            if mask[0].any():
                neg[mask[0]] = field(x[mask[0]])[0].float() < 0
        negative[k * layer:(k + 1) * layer] = neg
    negative = negative.reshape(dims)
    rows = []
    for axis in range(3):
        cross = negative.narrow(axis, 0, dims[axis] - 1) != negative.narrow(axis, 1, dims[axis] - 1)
        ijk = torch.nonzero(cross)
        rows.append(torch.cat([ijk + lo, torch.full_like(ijk[:, :1], axis)], 1))
    e = torch.cat(rows).cpu().numpy()
    ijk = e[:, :3]
    key, local = np.floor_divide(ijk, b), np.mod(ijk, b)
    e = e[np.lexsort((e[:, 3], local[:, 0], local[:, 1], local[:, 2], key[:, 0], key[:, 1], key[:, 2]))]
    e = torch.from_numpy(e).to(device)
    pa = e[:, :3].double() * h
    d = torch.zeros_like(pa).scatter_(1, e[:, 3:4], h)
    t0, t1 = torch.zeros(len(e), dtype=pa.dtype, device=device), torch.ones(len(e), dtype=pa.dtype, device=device)
    neg0 = field(pa)[0] < 0
    for _ in range(44):
        t = 0.5 * (t0 + t1)
        same = (field(pa + d * t[:, None])[0] < 0) == neg0
        t0, t1 = torch.where(same, t, t0), torch.where(same, t1, t)
    t = (0.5 * (t0 + t1)).clamp(1e-4, 1 - 1e-4)
    x = pa + d * t[:, None]
    out = dict.fromkeys(("triangles", "vertex_atom", "vertex_patch", "vertex_component", "area", "volume"))
    out["positions"], out["normals"] = x.cpu().numpy(), field(x)[1].cpu().numpy()
    return out
