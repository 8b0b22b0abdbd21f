"""Performance cases of the narrow-band elasticity solver: the calls a user of
the framework makes, through its public entry points.

Kinds (``case["kind"]``):

* ``fem``: the drop-in ``fem_solve`` on a serialized FEMInputs blob (host blob
  in, displacement field out): decode, set-up, solve and output are all in the
  pass, as they are for the reference's driver, which calls it once per
  optimizer iteration.
* ``solve``: the multigrid-preconditioned CG of a problem resident on the GPU
  (``native.Session``: set up once, solved many times), the solution copied
  into the caller's tensor.
* ``compliance``: forward and backward of the differentiable compliance of the
  PyTorch layer.
* ``simp``: one optimizer iteration through the host-array entry points: new
  densities, solve, sensitivity, filter, optimality-criteria update.
* ``band``: one iteration of the driver's loop with its narrow band: page maps,
  repacking of the solver input, the step on the band.
* ``render``: the headless renderer on a band's densities.

Domains: ``box`` (a dense cantilever), ``bridge`` (a dense box on four supports
with a loaded deck), ``shell`` (a sphere shell) and ``spheres`` (a 12-voxel band
around the union of eight spheres).  Geometry and boundary conditions are fixed
by the case; the densities come from the seed.
"""
import functools
import math

import numpy as np
import torch

from spgrid_topo_opt_b200 import configs, native
from spgrid_topo_opt_b200 import fem_interface as fi
from spgrid_topo_opt_b200.compliance import Compliance

PRECISION = {"reference": native.PRECISION_REFERENCE, "fp64": native.PRECISION_FP64, "mixed": native.PRECISION_MIXED}
YOUNG, POISSON, PENALTY, E_MIN = 1e6, 0.3, 3.0, 1e-9
VOLUME_FRACTION, STEP_LIMIT, FILTER = 0.55, 0.2, 1.5


def listed():
    return [
        # the smallest drop-in call: set-up and hundreds of short launches
        {"name": "fem_box16", "kind": "fem", "domain": "box", "nx": 16, "ny": 16, "nz": 16, "bottom": 4,
         "precision": "reference", "tol": 1e-6},
        # the reference's dense-box configuration (64^3, mg_bottom_size 16) in its default arithmetic
        {"name": "fem_box64", "kind": "fem", "domain": "box", "nx": 64, "ny": 64, "nz": 64, "bottom": 16,
         "precision": "reference", "tol": 1e-6},
        # the driver's default mg_bottom_size of 64 on an uneven box: a bottom level of 10^5 unknowns
        {"name": "fem_box83_bottom64", "kind": "fem", "domain": "box", "nx": 83, "ny": 70, "nz": 57, "bottom": 64,
         "precision": "mixed", "tol": 1e-6},
        # a mid-sized narrow band end to end through the drop-in call
        {"name": "fem_band384", "kind": "fem", "domain": "spheres", "n": 384, "bottom": 16, "precision": "mixed",
         "tol": 1e-6},
        # resident solves: a small ragged band in plain FP64, the 256^3 sphere shell, the 512^3 band in FP64
        # and the 1024^3 band (the benchmark workload) in mixed precision
        {"name": "solve_band204_fp64", "kind": "solve", "domain": "spheres", "n": 204, "bottom": 16,
         "precision": "fp64", "tol": 1e-6},
        {"name": "solve_shell256", "kind": "solve", "domain": "shell", "n": 256, "bottom": 16, "precision": "mixed",
         "tol": 1e-6},
        {"name": "solve_band512_fp64", "kind": "solve", "domain": "spheres", "n": 512, "bottom": 16,
         "precision": "fp64", "tol": 1e-6},
        {"name": "solve_band1024", "kind": "solve", "domain": "spheres", "n": 1024, "bottom": 16,
         "precision": "mixed", "tol": 1e-6},
        # gradient-based optimization in PyTorch: tight FP64 forward, adjoint backward
        {"name": "compliance_box48", "kind": "compliance", "domain": "box", "nx": 48, "ny": 48, "nz": 48,
         "bottom": 16, "precision": "fp64", "tol": 1e-10},
        # one SIMP iteration of a bridge with odd extents, host arrays in and out
        {"name": "simp_bridge97", "kind": "simp", "domain": "bridge", "nx": 97, "ny": 25, "nz": 49, "bottom": 16,
         "precision": "mixed", "tol": 1e-6},
        # one iteration of the driver's narrow-band loop on a larger bridge
        {"name": "band_bridge192", "kind": "band", "domain": "bridge", "nx": 192, "ny": 48, "nz": 96, "bottom": 16,
         "precision": "mixed", "tol": 1e-6},
        # pictures of a design: surface and volume mode
        {"name": "render_bridge256", "kind": "render", "domain": "bridge", "nx": 256, "ny": 64, "nz": 128,
         "width": 640, "height": 360, "frames": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same kinds and ranges."""
    kind = rng.choice(["fem", "fem", "solve", "solve", "compliance", "simp", "band", "render"])
    if kind == "render":
        n = _log_int(rng, 48, 256)
        width = _log_int(rng, 240, 800)
        return {"kind": kind, "domain": "bridge", "nx": n, "ny": max(12, n // 4), "nz": max(16, n // 2),
                "width": width, "height": width * 9 // 16, "frames": rng.randint(1, 8)}
    if kind in ("simp", "band"):
        n = _log_int(rng, 40, 192)
        return {"kind": kind, "domain": "bridge", "nx": n, "ny": max(12, n // rng.randint(2, 5)),
                "nz": max(12, n // rng.randint(1, 3)), "bottom": 16, "precision": rng.choice(["mixed", "fp64"]),
                "tol": 1e-6}
    if kind == "compliance":
        n = _log_int(rng, 16, 56)
        return {"kind": kind, "domain": "box", "nx": n, "ny": n - rng.randint(0, 3), "nz": n + rng.randint(0, 3),
                "bottom": 16, "precision": rng.choice(["fp64", "mixed"]), "tol": 1e-10}
    if kind == "fem" and rng.random() < 0.6:
        n = _log_int(rng, 16, 96)
        return {"kind": kind, "domain": "box", "nx": n, "ny": n - rng.randint(0, 4), "nz": n + rng.randint(0, 4),
                "bottom": rng.choice([16, 16, 32]), "precision": rng.choice(["reference", "fp64", "mixed"]),
                "tol": 1e-6}
    precision = rng.choice(["mixed", "fp64"])
    if rng.random() < 0.3:
        return {"kind": kind, "domain": "shell", "n": _log_int(rng, 64, 256), "bottom": 16, "precision": precision,
                "tol": 1e-6}
    n = 4 * _log_int(rng, 32, 120 if kind == "fem" else 200)
    return {"kind": kind, "domain": "spheres", "n": n, "bottom": 16, "precision": precision, "tol": 1e-6}


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _settings(p, case, dx):
    p.dx = dx
    p.global_mu, p.global_lambda = configs.lame(YOUNG, POISSON)
    p.krylov = fi.KrylovSolverParameters(case["tol"], 50, 0, False)
    p.extra_doubles.update({"penalty": PENALTY, "minimum_stiffness": E_MIN, "min_fraction": 0.0})
    p.extra_ints.update({"boundary_smoothing": 3, "keep_state": 0, "forced_reuse": 1,
                         "sgs_precision": PRECISION[case["precision"]]})
    p.pre_and_post_smoothing_iter = 1
    p.caller_method = "perf"


def _dense(case, rho):
    """Box or bridge with the given cell densities, packed as the driver packs them."""
    nx, ny, nz = rho.shape
    if case["domain"] == "bridge":
        prob = configs.bridge(nx, ny, nz, bottom_size=case.get("bottom", 16), support_radius=0.05)
        prob.density = rho
    else:
        cells = np.argwhere(np.ones((1, ny, nz), bool)).astype(np.int32)
        f = np.zeros(1, fi.FORCE_DTYPE)
        f["coord"][0] = (nx, ny // 2, nz // 2)
        f["f"][0] = (0.0, -1.0, 0.0)
        prob = configs.Problem("box", (nx, ny, nz), rho, cells, f, 1.0 / max(nx, ny, nz),
                               configs.mg_level_for(max(nx, ny, nz), case["bottom"]))
    p = configs.to_inputs(prob, E=YOUNG, nu=POISSON, penalty=PENALTY, minimum_stiffness=E_MIN,
                          tolerance=case.get("tol", 1e-6))
    p.extra_ints["sgs_precision"] = PRECISION[case.get("precision", "mixed")]
    return p


def _dense_density(case, seed):
    """Cell densities of a box or bridge: uniform in [0.2, 1] (a design under way)."""
    return np.random.default_rng(seed).uniform(0.2, 1.0, size=(case["nx"], case["ny"], case["nz"]))


@functools.lru_cache(maxsize=2)
def _spheres(n):
    """Geometry of the 12-voxel band around eight fixed spheres: the node blocks
    (4x4x4, block coordinates) in lexicographic order, the band cells of each
    [blocks, 64], the Dirichlet cells (the lowest band layer) and 16 loaded nodes."""
    g = np.random.default_rng(7)
    centres, radii = g.uniform(0.3, 0.7, size=(8, 3)), g.uniform(0.1, 0.3, size=8)
    dev = torch.device("cuda")
    half, nb = 6.0 / n, n // 4

    def distance(x, y, z):
        d = None
        for c, r in zip(centres, radii):
            e = ((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2).sqrt() - r
            d = e if d is None else torch.minimum(d, e)
        return d.abs()

    mid = (torch.arange(nb, device=dev, dtype=torch.float64) * 4 + 2) / n
    near = [(distance(mid[i], mid[:, None], mid[None, :]) <= half + math.sqrt(3) * 2 / n).nonzero() for i in range(nb)]
    cand = torch.cat([torch.cat([torch.full_like(k[:, :1], i), k], 1) for i, k in enumerate(near)])
    e = torch.arange(64, device=dev)
    off = torch.stack([e // 16, e // 4 % 4, e % 4], 1)
    at = (cand[:, None] * 4 + off[None] + 0.5).double() / n
    band = distance(at[..., 0], at[..., 1], at[..., 2]) <= half
    keep = band.any(1)
    cand, band = cand[keep], band[keep]
    m = nb + 1
    fwd = torch.tensor([[a, b, c] for a in (0, 1) for b in (0, 1) for c in (0, 1)], device=dev)
    key = lambda b: (b[..., 0] * m + b[..., 1]) * m + b[..., 2]
    every = torch.unique(key(cand[:, None] + fwd[None]))
    blocks = torch.stack([every // (m * m), every // m % m, every % m], 1)
    cells = torch.zeros((len(every), 64), dtype=torch.bool, device=dev)
    cells[torch.searchsorted(every, key(cand))] = band
    coord = (cand[:, None] * 4 + off[None])[band]
    low = coord[coord[:, 1] == coord[:, 1].min()].int().cpu().numpy()
    pick = coord[torch.from_numpy(g.choice(len(coord), 16, replace=False)).to(dev)] + 1
    v = g.normal(size=(16, 3))
    return (blocks.int().cpu().numpy(), cells.cpu().numpy(), low, pick.int().cpu().numpy(),
            v / np.linalg.norm(v, axis=1, keepdims=True))


@functools.lru_cache(maxsize=2)
def _shell(n, bottom):
    """The sphere shell's packed input; its densities are replaced per seed."""
    return configs.to_inputs(configs.sphere_shell(n, bottom_size=bottom))


def _inputs(case, seed):
    if case["domain"] in ("box", "bridge"):
        return _dense(case, _dense_density(case, seed))
    n = case["n"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["domain"] == "shell":
        src = _shell(n, case["bottom"])
        p = fi.FEMInputs()
        base, cells = src.density.base, src.density.data > 0
        p.resolution, p.mg_level = list(src.resolution), src.mg_level
        p.dirichlet_nodes, p.forces = src.dirichlet_nodes, src.forces
        lo = 0.2
    else:
        blocks, cells, low, pick, v = _spheres(n)
        p = fi.FEMInputs()
        base = blocks * 4 + configs.PADDING
        p.resolution, p.mg_level = [n + 7 * configs.PADDING] * 3, configs.mg_level_for(n, case["bottom"])
        p.dirichlet_nodes = configs.dirichlet_nodes_from_cells(low + configs.PADDING)
        p.forces = np.zeros(16, fi.FORCE_DTYPE)
        p.forces["coord"], p.forces["f"] = pick + configs.PADDING, v
        lo = 0.05
    rho = torch.rand(cells.shape, generator=gen, device="cuda", dtype=torch.float64) * (1 - lo) + lo
    data = torch.where(torch.from_numpy(cells).cuda(), rho, 0.0).cpu().numpy()
    p.density = fi.BlockedGrid(resolution=list(p.resolution), base=base.astype(np.int32), data=data)
    _settings(p, case, 1.0 / n)
    p.preserve_output(base.shape[0])
    return p


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "render":
        rho = _dense_density(case, seed)
        # a design: solid where a smooth random field is high, void elsewhere
        g = torch.Generator(device="cuda").manual_seed(seed)
        lattice = torch.rand((1, 1, 9, 5, 7), generator=g, device="cuda", dtype=torch.float64)
        field = torch.nn.functional.interpolate(lattice, size=rho.shape, mode="trilinear", align_corners=True)
        rho = np.where(field[0, 0].cpu().numpy() > 0.55, rho, 1e-3)
        p = _dense(case, rho)
        state["band"] = native.Band(p.density.base, p.resolution, (p.density.data > 0).astype(np.uint8),
                                    p.density.data)
        state["camera"] = native.view_matrix(20, -35, 0, 0, 0, -3.0)
        return state
    p = _inputs(case, seed)
    if kind == "fem":
        state["blob"] = fi.serialize_inputs(p)
    elif kind == "solve":
        state["session"] = native.Session(fi.serialize_inputs(p), PRECISION[case["precision"]])
        state["u"] = torch.empty(state["session"].solution_size(), dtype=torch.float64, device="cuda")
    elif kind == "compliance":
        state["model"] = Compliance(p, precision=PRECISION[case["precision"]], tolerance=case["tol"])
        state["rho"] = torch.from_numpy(p.density.data).cuda().requires_grad_(True)
    elif kind == "simp":
        state["rho"] = p.density.data.copy()
        state["session"] = native.Session(p, PRECISION[case["precision"]])
    elif kind == "band":
        rho = p.density.data
        inside = rho > 0
        # a third of the box has gone to the minimum density: its blocks leave the band
        y = (p.density.base[:, 1] - configs.PADDING)[:, None] + (np.arange(64) // 4 % 4)[None]
        x = (p.density.base[:, 0] - configs.PADDING)[:, None] + (np.arange(64) // 16)[None]
        void = (y < case["ny"] // 2) & (np.abs(x - case["nx"] / 2) < case["nx"] / 3)
        state["rho"] = np.where(inside, np.where(void, 1e-9, rho), 0.0)
        state["all"] = np.ones(len(rho), np.uint8)
        state["band"] = native.Band(p.density.base, p.resolution, inside.astype(np.uint8), state["rho"])
        p.density = fi.BlockedGrid(resolution=list(p.resolution), base=np.zeros((0, 3), np.int32),
                                   data=np.zeros((0, 64)))
        state["template"] = fi.serialize_inputs(p)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fem":
        out = native.fem_solve_outputs(state["blob"])
        if not out.success:
            raise RuntimeError(out.info)
        # the displacements; the record's fourth entry is the residual the stopping rule left over
        return out.displacements.data[..., :3]
    if kind == "solve":
        state["session"].solve()
        state["session"].solution_device(state["u"])
        return state["u"]
    if kind == "compliance":
        c = state["model"](state["rho"])
        return c, torch.autograd.grad(c, state["rho"])[0]
    if kind == "simp":
        s, rho = state["session"], state["rho"]
        s.set_density(rho)
        s.solve(tolerance=case["tol"])
        objective, dc, _ = s.sensitivity(rho)
        dc = s.filter_sensitivity(rho, -dc, FILTER)
        new, _, _ = s.oc_update(rho, dc, VOLUME_FRACTION, STEP_LIMIT)
        return objective, dc, new
    if kind == "band":
        b = state["band"]
        b.set_density(state["rho"])
        b.set_fat(state["all"])
        b.update(minimum_density=0.0)
        with b.session(state["template"], PRECISION[case["precision"]]) as s:
            r = b.step(s, tolerance=case["tol"], volume_fraction=VOLUME_FRACTION, step_limit=STEP_LIMIT,
                       filter_size=FILTER)
        return r["objective"], b.density(), np.stack(b.maps())
    kw = dict(frames=case["frames"])
    surface, _ = state["band"].render(case["width"], case["height"], state["camera"], mode=0, threshold=0.5, **kw)
    volume, _ = state["band"].render(case["width"], case["height"], state["camera"], mode=1, threshold=0.05,
                                     extinction=2.0, **kw)
    return surface.view(np.int32), volume.view(np.int32)


# --------------------------------------------------------------------------
# What a pass cannot do without, and how far another implementation may be off
# --------------------------------------------------------------------------
def _nodes(case):
    if case["domain"] in ("box", "bridge"):
        return (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    n = case["n"]
    return 0.2555 * n ** 3 + 5.65 * n ** 2 if case["domain"] == "shell" else 23.0 * n ** 2


def work(case):
    if case["kind"] == "render":
        cells = case["nx"] * case["ny"] * case["nz"]
        pixels = case["width"] * case["height"]
        # the densities in, two images out; per pixel and frame a surface ray and its ambient rays (about 100
        # voxel steps of about 10 operations) and a 1025-step volume march
        return {"bytes": 8.0 * cells + 8.0 * pixels, "flops": float(pixels * case["frames"]) * (1000 + 1025 * 10)}
    n, w = _nodes(case), 4 if case["precision"] == "mixed" else 8
    # CG iterations that the algorithm takes at the case's tolerance (a size-dependent round figure)
    its = {"box": 14, "bridge": 20, "shell": 22, "spheres": 45}[case["domain"]] * (2 if case["tol"] < 1e-8 else 1)
    # an iteration: two smoothing sweeps and a residual in the V-cycle's precision (u, b and the cell stiffness
    # once each), transfers, an FP64 matvec and the CG updates; coarse levels add about a quarter.  A node's row
    # of K holds 81 x 3 entries.
    cycle = (2 * 10 * w + 10 * w + 8 * w) * 1.25
    cg = 7 * 8 + 3 * 8 * 6
    return {"bytes": n * (its * (cycle + cg) + 2 * 8 + 3 * 8), "flops": n * its * (4 * 486 * 1.25 + 20)}


def tolerance(case):
    kind = case["kind"]
    if kind == "render":
        return "exact"
    if kind == "compliance":
        return {"rel": 1e-9, "max": 1e-7}
    # a CG solve stopped at a relative residual of 1e-6: one iteration more or fewer moves the solution by about
    # its own error, which measures up to 6e-6 of it (the 16^3 box against the exact solution)
    return {"rel": 2e-5, "max": 8e-4}


# --------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# --------------------------------------------------------------------------
def _element():
    """24 x 24 element matrix of the unit trilinear hexahedron by 2-point Gauss
    quadrature (exact), node 4x + 2y + z, dof 3 node + axis."""
    mu, la = YOUNG / (2 * (1 + POISSON)), YOUNG * POISSON / ((1 + POISSON) * (1 - 2 * POISSON))
    c = np.array([[i >> 2, (i >> 1) & 1, i & 1] for i in range(8)], float)
    K = np.zeros((8, 3, 8, 3))
    for p in np.ndindex(2, 2, 2):
        x = 0.5 + (np.array(p) - 0.5) / math.sqrt(3)
        s = np.where(c == 1, x, 1 - x)
        g = np.stack([(2 * c[:, a] - 1) * np.prod(np.delete(s, a, 1), 1) for a in range(3)], 1)
        K += 0.125 * (mu * (np.einsum("ak,bk,ij->aibj", g, g, np.eye(3)) + np.einsum("aj,bi->aibj", g, g))
                      + la * np.einsum("ai,bj->aibj", g, g))
    return torch.from_numpy(K.reshape(24, 24)).cuda()


def _corners(u):
    """[3, nodes] -> [24, cells]"""
    s = [n - 1 for n in u.shape[1:]]
    return torch.cat([u[:, a:a + s[0], b:b + s[1], c:c + s[2]].reshape(3, -1)
                      for a in (0, 1) for b in (0, 1) for c in (0, 1)])


def _gather(f, shape):
    """[24, cells] -> [3, nodes], summed"""
    out = torch.zeros((3, shape[0] + 1, shape[1] + 1, shape[2] + 1), dtype=torch.float64, device="cuda")
    for i in range(8):
        a, b, c = i >> 2, (i >> 1) & 1, i & 1
        out[:, a:a + shape[0], b:b + shape[1], c:c + shape[2]] += f[3 * i:3 * i + 3].reshape(3, *shape)
    return out


def _solve64(case, rho):
    """u [3, nodes] of K(rho) u = f by Jacobi-preconditioned CG to round-off, the force field, and u_e^T K0 u_e."""
    p = _dense(case, rho.cpu().numpy())  # its boundary conditions
    shape, K, dx = rho.shape, _element(), 1.0 / max(rho.shape)
    E = ((1 - E_MIN) * rho ** PENALTY + E_MIN).reshape(1, -1)
    free, f = (torch.zeros((3, shape[0] + 1, shape[1] + 1, shape[2] + 1), dtype=torch.float64, device="cuda")
               for _ in range(2))
    free += 1
    d = torch.from_numpy(p.dirichlet_nodes["coord"].astype(np.int64) - configs.PADDING).cuda()
    free[torch.from_numpy(p.dirichlet_nodes["axis"].astype(np.int64)).cuda(), d[:, 0], d[:, 1], d[:, 2]] = 0
    d = torch.from_numpy(p.forces["coord"].astype(np.int64) - configs.PADDING).cuda()
    f[:, d[:, 0], d[:, 1], d[:, 2]] = torch.from_numpy(np.array(p.forces["f"].T.tolist())).cuda()
    f = f * free
    apply = lambda u: dx * free * _gather(E * (K @ _corners(u)), shape)
    diag = dx * _gather(E * torch.diagonal(K)[:, None], shape)
    u, r = torch.zeros_like(f), f.clone()
    z = r / diag
    s, rho_z = z.clone(), (r * z).sum()
    stop = 1e-13 * r.abs().max()
    for it in range(6000):
        q = apply(s)
        alpha = rho_z / (s * q).sum()
        u, r = u + alpha * s, r - alpha * q
        if it % 20 == 0 and r.abs().max() <= stop:
            break
        z = r / diag
        new = (r * z).sum()
        s, rho_z = z + (new / rho_z) * s, new
    e = _corners(u)
    return u, f, (e * (K @ e)).sum(0).reshape(shape)


def _blocks(field):
    """A node or cell field [x, y, z, ...] in the input blocks' layout: all 4x4x4 blocks of the node grid in
    lexicographic order, in-block index 16 x + 4 y + z."""
    n = [4 * -(-s // 4) for s in field.shape[:3]]
    pad = torch.zeros((*n, *field.shape[3:]), dtype=field.dtype, device=field.device)
    pad[:field.shape[0], :field.shape[1], :field.shape[2]] = field
    v = pad.reshape(n[0] // 4, 4, n[1] // 4, 4, n[2] // 4, 4, -1).permute(0, 2, 4, 1, 3, 5, 6)
    return v.reshape(-1, 64, *field.shape[3:])


def exact(case, seed):
    if case["domain"] not in ("box", "bridge") or case["kind"] not in ("fem", "compliance", "simp"):
        return None
    if case["nx"] * case["ny"] * case["nz"] > 300_000:
        return None
    rho = torch.from_numpy(_dense_density(case, seed)).cuda()
    u, f, s = _solve64(case, rho)
    # cells live on the node grid's blocks: one more (empty) layer than cells on each axis
    cells = lambda c: _blocks(torch.nn.functional.pad(c, (0, 1, 0, 1, 0, 1)))
    if case["kind"] == "fem":
        return _blocks(u.permute(1, 2, 3, 0)).cpu().numpy()
    slope = PENALTY * rho ** (PENALTY - 1) * (1 - E_MIN) * s
    if case["kind"] == "compliance":
        return (f * u).sum(), cells(-slope / max(rho.shape))
    objective = (s * (E_MIN + rho ** PENALTY * (1 - E_MIN))).sum()
    # the density-weighted filter: cells within 1.5, weight 1.5 - distance
    pad = lambda a: torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))
    g, r, one = pad(-slope), pad(rho), pad(torch.ones_like(rho))
    num = den = 0
    for i in np.ndindex(3, 3, 3):
        w = max(0.0, FILTER - math.sqrt(sum((k - 1) ** 2 for k in i)))
        at = tuple(slice(k, k + m) for k, m in zip(i, rho.shape))
        num, den = num + w * g[at] * r[at], den + w * one[at] * (rho + 1e-3)
    dc = num / den
    lower, upper = 1e-20, 1e20
    while lower * (1 + 1e-7) < upper:
        mid = 0.5 * (lower + upper)
        new = (rho * ((-dc).clamp_min(0) / mid).sqrt())
        new = torch.minimum(torch.maximum(new, rho - STEP_LIMIT), rho + STEP_LIMIT).clamp(0, 1)
        if new.sum() > VOLUME_FRACTION * rho.numel():
            lower = mid
        else:
            upper = mid
    return objective, cells(dc).cpu().numpy(), cells(new).cpu().numpy()
