"""Performance cases of the framework: what its users have it compute, through its public Python API.

Every case goes through `Problem` or `Batch` with host arrays in the reference's layouts, as the drop-in C++
library, the request loop and the benchmark do.  The kinds:

  design     a whole design run (`Problem.run_global`, the reference CLI's `GLOBAL` command): the solid-domain
             solve and `loops` design iterations, in one of three solver set-ups:
               reference  the CLI's own (FP64, Adapted V-cycle, tolerance 1e-3, at most 800 iterations, the
                          reference's summation order) -- what a user gets without choosing anything
               fp64       FP64, Standard V-cycle rebuilt each iteration, every solve to 1e-6
               mixed      the same in mixed precision: the production set-up of the benchmark
  batch      many small designs of uneven size stepping together (`Batch`), the serving set-up
  matvec     one K(E)u product (`K_times_u_finest`)
  precond    multigrid set-up for new moduli and one V-cycle on it
  solve      multigrid set-up for new moduli and a converged `PCG_free` from a zero start
  elements   moduli, element compliance and sensitivities of a design (`simp`, `ComputeCompliance`, ...)
  update     sensitivity filter of two successive iterations, scaling and the OC bisection
"""
import math
import random

import numpy as np
import torch

import algorithmengineering_altproject_b200 as t3d

CSOLID = 1.172271756   # a solid domain's compliance of ordinary size (the 30 x 60 x 30 cantilever's)


def listed():
    return [
        # the smallest whole run: a smoke test or a parameter study on a toy domain; launches and latency only
        dict(name="design 6x12x6 reference", kind="design", dims="6x12x6", mode="reference", loops=3, load=0, voids=0),
        # the reference CLI's ordinary call, `GLOBAL 30 60 30 0.12`
        dict(name="design 30x60x30 reference", kind="design", dims="30x60x30", mode="reference", loops=2, load=0,
             voids=0),
        # a desktop-size reference run: every solve stops at the 800-iteration cap
        dict(name="design 64x128x64 reference", kind="design", dims="64x128x64", mode="reference", loops=1, load=0,
             voids=0),
        # converged FP64 design of a ragged domain with a passive void under a torsion couple
        dict(name="design 45x101x37 fp64", kind="design", dims="45x101x37", mode="fp64", loops=3, load=2, voids=1),
        # the benchmark's middle configuration in its production set-up
        dict(name="design 96x192x96 mixed", kind="design", dims="96x192x96", mode="mixed", loops=3, load=0, voids=0),
        # the largest: the benchmark's headline configuration, 101.6 M DOF
        dict(name="design 256x512x256 mixed", kind="design", dims="256x512x256", mode="mixed", loops=1, load=0,
             voids=0),
        # requests of a design server in flight together
        dict(name="batch of 12", kind="batch", count=12, lo=32, hi=112, shapes=7, loops=2),
        # an operator call of the drop-in library on a ragged grid
        dict(name="matvec 33x67x21", kind="matvec", dims="33x67x21"),
        # the preconditioner as a user's own solver calls it
        dict(name="precond 80x160x80", kind="precond", dims="80x160x80", cycle="adapted"),
        # a converged linear solve on a given design
        dict(name="solve 48x96x48", kind="solve", dims="48x96x48", tol=1e-8),
        # the element-wise part of a design iteration
        dict(name="elements 96x192x96", kind="elements", dims="96x192x96"),
        # the design update with the default summation order
        dict(name="update 50x100x50", kind="update", dims="50x100x50", order=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    """nely x nelx x nelz of a slender domain, as the listed ones are: nelx the longest side."""
    y = _log_int(rng, lo, hi)
    return "%dx%dx%d" % (y, max(8, int(round(y * rng.uniform(1.5, 2.5)))), max(4, int(round(y * rng.uniform(0.6, 1.2)))))


def draw(rng):
    kind = rng.choice(["design", "design", "design", "batch", "matvec", "precond", "solve", "elements", "update"])
    if kind == "design":
        mode = rng.choice(["reference", "fp64", "mixed"])
        # the reference set-up does 800 iterations a solve, the mixed one a few dozen
        return dict(kind=kind, dims=_dims(rng, 6, {"reference": 56, "fp64": 72, "mixed": 128}[mode]), mode=mode,
                    loops=rng.randint(1, 2), load=rng.randint(0, 2), voids=rng.randint(0, 1))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 16), lo=32, hi=rng.choice([48, 80, 112]),
                    shapes=rng.randrange(1000), loops=rng.randint(1, 3))
    if kind == "matvec":
        return dict(kind=kind, dims=_dims(rng, 6, 80))
    if kind == "precond":
        return dict(kind=kind, dims=_dims(rng, 6, 96), cycle=rng.choice(["adapted", "standard"]))
    if kind == "solve":
        return dict(kind=kind, dims=_dims(rng, 6, 64), tol=rng.choice([1e-6, 1e-8]))
    if kind == "elements":
        return dict(kind=kind, dims=_dims(rng, 6, 112))
    return dict(kind=kind, dims=_dims(rng, 6, 80), order=rng.randint(0, 1))


def _parse(dims):
    return tuple(int(v) for v in dims.split("x"))


# ---------------------------------------------------------------- the reference's layouts
def _padded(dims):
    """(nx, ny, nz): element counts padded to the multigrid hierarchy (at least 3 halvings)."""
    y, x, z = dims
    n, levels = x * y * z, 0
    while n >= 50000:
        levels, n = levels + 1, (n + 4) // 8
    s = 1 << max(3, levels)
    return tuple(-(-v // s) * s for v in (x, y, z))


def _elements(dims):
    """Element coordinates (ex, ey, ez) in the element arrays' order: 64-bit Morton keys, x the highest bit."""
    y, x, z = dims
    e = np.indices((z, y, x), dtype=np.int64).reshape(3, -1)
    ez, ey, ex = e
    key = np.zeros(ex.shape, dtype=np.int64)
    for b in range(max(x, y, z).bit_length()):
        key |= ((ex >> b) & 1) << (3 * b + 2) | ((ey >> b) & 1) << (3 * b + 1) | ((ez >> b) & 1) << (3 * b)
    o = np.argsort(key, kind="stable")
    return ex[o], ey[o], ez[o]


def _free_nodes(dims):
    """Coordinates (ix, iy, iz) of the nodes whose 3 DOFs are free, in ascending node number: the solid block's
    nodes off the clamped x = 0 face.  The solid block fills the padded grid from its high-y side."""
    y, x, z = dims
    _, ny, _ = _padded(dims)
    iz, iy, ix = np.meshgrid(np.arange(z + 1), np.arange(ny - y, ny + 1), np.arange(1, x + 1), indexing="ij")
    return ix.ravel(), iy.ravel(), iz.ravel()


# ---------------------------------------------------------------- inputs
def _waves(rng, coords, scale, terms=6):
    """A smooth random field in [-1, 1] at the given coordinates."""
    f = np.zeros(coords[0].shape)
    for _ in range(terms):
        k = rng.uniform(0.5, 3.0, 3) * np.pi / scale
        f += np.cos(sum(k[d] * coords[d] for d in range(3)) + rng.uniform(0, 2 * np.pi))
    return f / terms


def _density(rng, dims):
    """A design part way through its iterations: struts near 1, void near the minimum, grey between."""
    c = _elements(dims)
    f = _waves(rng, c, max(dims) / 2) + 0.05 * rng.standard_normal(c[0].size)
    return np.clip(1.0 / (1.0 + np.exp(-14.0 * (f - 0.18))), 1e-3, 1.0).astype(np.float32)


def _moduli(x):
    return 1e-6 + x.astype(np.float64) ** 3 * (1.0 - 1e-6)


def _displacement(rng, dims):
    """Bending of a clamped beam with local variation, on the free DOFs."""
    c = _free_nodes(dims)
    t = c[0] / float(dims[1])
    u = np.stack([0.3 * t * _waves(rng, c, max(dims)), 0.2 * t * _waves(rng, c, max(dims)),
                  -t * t * (1.0 + 0.2 * _waves(rng, c, max(dims)))], axis=1)
    return (u + 1e-3 * rng.standard_normal(u.shape) * t[:, None]).ravel()


def _sensitivities(rng, x):
    """Compliance sensitivities: negative, over several orders of magnitude, largest in the struts."""
    return (-0.3 * x ** 2 * np.exp(1.5 * rng.standard_normal(x.size)) - 1e-6).astype(np.float32)


def _params(mode):
    if mode == "reference":
        return {}
    p = dict(mg_vcycle=t3d.T3D_VCYCLE_STANDARD, mg_rebuild_period=1, cg_tol=1e-6, cg_max_it=2000)
    if mode == "mixed":
        p.update(precision=t3d.T3D_MIXED, oc_sum_order=t3d.T3D_SUM_FP64, mg_max_levels=6)
    return p


def _spec(dims, load, voids):
    if not load and not voids:
        return None
    y, x, z = dims
    # one ellipsoid in the middle of the domain: it never cuts the load from the support
    v = [(0.5 * x, 0.5 * y, 0.5 * z, 0.15 * x, 0.25 * y, 0.25 * z)] if voids else []
    return t3d.ProblemSpec.make(load, v)


def _batch_shapes(case):
    """Sides as the request generator draws them: nelx a multiple of 8, the others a fraction of half of it."""
    r = random.Random(case["shapes"])
    shapes = []
    for _ in range(case["count"]):
        x = 8 * r.randint(case["lo"] // 8, case["hi"] // 8)
        shapes.append((max(8, int(x / 2 * r.uniform(0.5, 1.0))), x, max(8, int(x / 2 * r.uniform(0.5, 1.0))),
                       r.randint(0, 2), r.randint(0, 1)))
    return shapes


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        shapes = _batch_shapes(case)
        p = _params("mixed")
        p.pop("precision")
        B = t3d.Batch([s[:3] for s in shapes], problems=[_spec(s[:3], s[3], s[4]) for s in shapes],
                      mg_coarse_assembly=t3d.T3D_COARSE_FULL, **p)
        return dict(case=case, B=B, V0=rng.uniform(0.08, 0.3, case["count"]).astype(np.float32))
    dims = _parse(case["dims"])
    if kind == "design":
        P = t3d.Problem(*dims, problem=_spec(dims, case["load"], case["voids"]), **_params(case["mode"]))
        return dict(case=case, P=P, V0=float(rng.uniform(0.1, 0.16)))
    x = _density(rng, dims)
    if kind == "matvec":
        return dict(case=case, P=t3d.Problem(*dims), E=_moduli(x), u=_displacement(rng, dims))
    if kind == "precond":
        std = case["cycle"] == "standard"
        P = t3d.Problem(*dims, **(dict(mg_vcycle=t3d.T3D_VCYCLE_STANDARD) if std else {}))
        r = _displacement(rng, dims) * 1e-3
        return dict(case=case, P=P, E=_moduli(x), r=r)
    if kind == "solve":
        P = t3d.Problem(*dims, mg_vcycle=t3d.T3D_VCYCLE_STANDARD)
        return dict(case=case, P=P, E=_moduli(x), b=P.bfree(), x0=np.zeros(P.nf))
    if kind == "elements":
        return dict(case=case, P=t3d.Problem(*dims), x=x, u=_displacement(rng, dims))
    P = t3d.Problem(*dims, oc_sum_order=case["order"])
    a, b = _sensitivities(rng, x), _sensitivities(rng, x)
    return dict(case=case, P=P, x=x, a=x * a, b=x * (0.5 * a + 0.5 * b), V0=float(x.mean(dtype=np.float64)))


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "batch":
        B = s["B"]
        cs = B.design_init(s["V0"])
        recs = B.run([case["loops"]] * B.n)
        return dict(c_solid=cs, obj=np.array([[r["obj"] for r in m] for m in recs]),
                    x=[m.density() for m in B.members])
    P = s["P"]
    if kind == "design":
        cs, recs, x = P.run_global(s["V0"], case["loops"])
        return dict(c_solid=cs, obj=np.array([r["obj"] for r in recs]), x=x)
    if kind == "matvec":
        return P.K_times_u_finest(s["E"], s["u"])
    if kind == "precond":
        P.make_diagonal_preconditioner_from_static(s["E"])
        return P.vcycle(s["r"])
    if kind == "solve":
        P.make_diagonal_preconditioner_from_static(s["E"])
        u, its = P.PCG_free(s["E"], s["b"], s["x0"], tol=case["tol"], maxIt=800)
        return dict(u=u, its=its)
    if kind == "elements":
        E = P.simp(s["x"])
        C, ce = P.ComputeCompliance(E, s["u"])
        return dict(E=E, C=C, ce=ce, dc=P.sensitivity(s["x"], ce, CSOLID))
    # two successive iterations' sensitivities: each filter call starts from the last one's result
    fa = P.ApplyPDEFilter(s["a"])
    fb = P.ApplyPDEFilter(s["b"])
    dc = P.dc_scale(fb, s["x"])
    xn, change, lmid, passes = P.oc_update(s["x"], dc, s["V0"])
    return dict(fa=fa, fb=fb, dc=dc, x=xn, oc=np.array([change, lmid], dtype=np.float32), passes=passes)


def work(case):
    """Bytes and operations the path cannot do without.  Solves: the iteration counts are the algorithm's
    (the cap of the reference set-up; about 45 a converged solve), each iteration reading and writing the PCG
    vectors once (x, r, p, z, Ap: 10 passes), the moduli once and the preconditioner's vectors once."""
    kind = case["kind"]

    def sizes(dims):
        y, x, z = dims
        return x * y * z, 3 * (x + 1) * (y + 1) * (z + 1)

    def solves(ne, n, mode, count):
        w, its = (4, 45) if mode == "mixed" else (8, 45 if mode == "fp64" else 800)
        if mode == "reference" and ne < 60000:
            its = 450
        return count * its * (w * (12 * n + ne)), count * its * 1152 * ne

    if kind in ("design", "batch"):
        b = f = 0
        parts = _batch_shapes(case) if kind == "batch" else [_parse(case["dims"])]
        for p in parts:
            ne, n = sizes(p[:3])
            sb, sf = solves(ne, n, "mixed" if kind == "batch" else case["mode"], case["loops"] + 1)
            b, f = b + sb + case["loops"] * (8 * n + 40 * ne), f + sf + case["loops"] * 1152 * ne
        return dict(bytes=b, flops=f)
    ne, n = sizes(_parse(case["dims"]))
    if kind == "matvec":
        return dict(bytes=8 * (2 * n + ne), flops=1152 * ne)
    if kind == "precond":
        return dict(bytes=8 * (3 * n + ne), flops=60 * n)
    if kind == "solve":
        b, f = solves(ne, n, "fp64", 1)
        return dict(bytes=b, flops=f)
    if kind == "elements":
        return dict(bytes=8 * n + 40 * ne, flops=1152 * ne)
    return dict(bytes=2 * 8 * ne + 12 * ne, flops=2 * 10 * 128 * ne)


# ---------------------------------------------------------------- the same in 64 bits, without the library
_OFF = np.array([[0, 1, 0], [1, 1, 0], [1, 0, 0], [0, 0, 0], [0, 1, 1], [1, 1, 1], [1, 0, 1], [0, 0, 1]])
_SGN = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])


def _shape_gradients(g):
    """8 x 3 derivatives of the trilinear shape functions at the natural coordinates g."""
    f = 1 + _SGN * g
    return 0.125 * np.stack([_SGN[:, 0] * f[:, 1] * f[:, 2], _SGN[:, 1] * f[:, 0] * f[:, 2],
                             _SGN[:, 2] * f[:, 0] * f[:, 1]], axis=1)


def _stiffness(nu=0.3):
    """Unit-modulus stiffness of a unit cube, 2 x 2 x 2 Gauss points."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
    D = np.diag([2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam
    K = np.zeros((24, 24))
    for g in _SGN / math.sqrt(3.0):
        d = 2 * _shape_gradients(g)
        B = np.zeros((6, 24))
        for a in range(8):
            dx, dy, dz = d[a]
            B[:, 3 * a:3 * a + 3] = [[dx, 0, 0], [0, dy, 0], [0, 0, dz], [0, dz, dy], [dz, 0, dx], [dy, dx, 0]]
        K += B.T @ D @ B / 8
    return K


def _element_nodes(dims, device):
    """ne x 8 node numbers of the elements' corners in the padded grid."""
    nx, ny, _ = _padded(dims)
    ex, ey, ez = (torch.from_numpy(v).to(device) for v in _elements(dims))
    cy = ny - 1 - ey
    return torch.stack([((ez + o[2]) * (ny + 1) + cy + o[1]) * (nx + 1) + ex + o[0] for o in _OFF.tolist()], dim=1)


def _node_count(dims):
    nx, ny, nz = _padded(dims)
    return (nx + 1) * (ny + 1) * (nz + 1)


def _exact_filter(dims, src, rmin, device):
    """The Helmholtz-filtered field: (r^2 K0 + K1) x = the elements' shares at the nodes, averaged back."""
    r = rmin / (2 * math.sqrt(3.0))
    k = np.zeros((8, 8))
    for g in _SGN / math.sqrt(3.0):
        d, N = _shape_gradients(g), 0.125 * np.prod(1 + _SGN * g, axis=1)
        k += r * r * d @ d.T + np.outer(N, N) / 8
    k = torch.from_numpy(k).to(device)
    nodes, n = _element_nodes(dims, device), _node_count(dims)
    s = torch.from_numpy(src.astype(np.float64)).to(device)

    def gather(v):
        return torch.zeros(n, dtype=torch.float64, device=device).index_add_(0, nodes.reshape(-1), v.reshape(-1))

    rhs = gather((s / 8)[:, None].expand(-1, 8))
    diag = gather(k.sum(1).expand(nodes.shape[0], -1))
    inv = torch.where(diag > 0, 1 / diag.clamp_min(1e-300), torch.ones_like(diag))
    x, res = torch.zeros_like(rhs), rhs.clone()
    p, rz = inv * res, float((res * inv * res).sum())
    for _ in range(400):
        Ap = gather(p[nodes] @ k)
        a = rz / float((p * Ap).sum())
        x += a * p
        res -= a * Ap
        if float(res.norm()) <= 1e-13 * float(rhs.norm()):
            break
        new = float((res * inv * res).sum())
        p = inv * res + (new / rz) * p
        rz = new
    return (x[nodes].sum(1) / 8).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("matvec", "elements", "update"):
        return None
    dims = _parse(case["dims"])
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    rng = np.random.default_rng(seed)
    x = _density(rng, dims)
    if kind == "update":
        a, b = _sensitivities(rng, x), _sensitivities(rng, x)
        rmin = math.sqrt(3.0)
        fa = _exact_filter(dims, x * a, rmin, device)
        fb = _exact_filter(dims, x * (0.5 * a + 0.5 * b), rmin, device)
        return dict(fa=fa, fb=fb, dc=fb / np.maximum(1e-3, x.astype(np.float64)), x=None, oc=None, passes=None)
    nx, ny, _ = _padded(dims)
    ix, iy, iz = _free_nodes(dims)
    free = torch.from_numpy((iz.astype(np.int64) * (ny + 1) + iy) * (nx + 1) + ix).to(device)
    u = torch.zeros((_node_count(dims), 3), dtype=torch.float64, device=device)
    u[free] = torch.from_numpy(_displacement(rng, dims).reshape(-1, 3)).to(device)
    nodes = _element_nodes(dims, device)
    ue = u[nodes].reshape(-1, 24)
    f = ue @ torch.from_numpy(_stiffness()).to(device)
    E = torch.from_numpy(_moduli(x)).to(device)
    if kind == "matvec":
        y = torch.zeros_like(u).index_add_(0, nodes.reshape(-1), (f * E[:, None]).reshape(-1, 3))
        return y[free].reshape(-1).cpu().numpy()
    ce = (f * ue).sum(1)
    xd = torch.from_numpy(x.astype(np.float64)).to(device)
    dc = ce / CSOLID * xd ** 2 * (1e-6 - 1.0) * 3.0
    return dict(E=E.cpu().numpy(), C=float((E * ce).sum()), ce=ce.cpu().numpy(), dc=dc.cpu().numpy())
