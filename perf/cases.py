"""The work that performance is measured on: calls of the public entry points of
angstromcube_b200 over the range of sizes, precisions and options that its users have.

A case is a dict of plain values:

  call                 "action" (action_t.multiply), "solve", "batch" (solve_batched), "vjp" or
                       "density" (get_projection_coefficients)
  nx, ny, nz           4x4x4-point cubes of the cell
  bc                   boundary conditions of x, y, z: 0 isolated, 1 periodic, 2 vacuum, 3 repeat
  hx, hy, hz           grid spacings in Bohr
  r_trunc              truncation radius in Bohr
  sx, sy, sz           box of source cubes (64 columns each)
  order                reach of the finite differences (4: 8th order, 8: 16th order)
  atoms, numax, sigma  atoms, their largest basis size (mixed: each atom its own, up to it), spread
  lattice              atoms on a jittered lattice (True) or anywhere in the cell
  Ere, Eim, kx, ky, kz energy in Hartree, k-point in units of 2 pi / cell
  dtype                "float32" or "float64": blocks of an action, recurrences of a solve
  and of the solves: tolerance, precondition, pairs (of a batch), iterations (tfQMR iterations the
  work is counted for)

`exact` evaluates the same operator in plain torch with 64 bits: the truncation and the order of
the blocks from the geometry, the finite differences along the lines of target cubes, and the
projectors as dense products.
"""
import math

import numpy as np
import torch

from angstromcube_b200 import green_action, green_function, workloads

PROJECTION_RADIUS = 6.0          # in units of each atom's spread
GRID = 0.25                      # Bohr


# ------------------------------------------------------------------ the cases

def _case(call, n, sources, **kw):
    c = dict(call=call, nx=n[0], ny=n[1], nz=n[2], bc="111", hx=GRID, hy=GRID, hz=GRID, r_trunc=12.0,
             sx=sources[0], sy=sources[1], sz=sources[2], order=4, atoms=0, numax=5, mixed=False, sigma=0.6,
             lattice=True, Ere=-0.2, Eim=0.02, kx=0.0, ky=0.0, kz=0.0, dtype="float64")
    c.update(kw)
    return c


def listed():
    L = []

    def add(name, *a, **kw):
        L.append(dict(_case(*a, **kw), name=name))

    # the smallest cell in use, one atom and one source cube: launches and latency count
    add("action_f64_cell4", "action", (4, 4, 4), (1, 1, 1), r_trunc=6.0, atoms=1, numax=3, sigma=0.5, Ere=-0.3, Eim=0.05)
    # an ordinary small periodic cell away from Gamma, in the FP32 recurrences of a mixed solve
    add("action_f32_cell8", "action", (8, 8, 8), (2, 2, 1), atoms=8, kx=0.1, ky=0.2, kz=-0.15, dtype="float32")
    # a slab-like cell: every direction with another boundary condition, spacing and length, a
    # truncation sphere that leaves z-lines of many lengths, atoms of several basis sizes
    add("action_f64_ragged", "action", (9, 7, 11), (3, 2, 2), bc="012", hx=0.25, hy=0.3, hz=0.2, r_trunc=2.4, atoms=9,
        mixed=True, lattice=False, ky=0.2)
    # a molecule in an isolated box with the 16th-order kinetic energy
    add("action_f64_fd16", "action", (12, 12, 12), (2, 2, 2), bc="000", r_trunc=4.0, order=8, atoms=5, numax=3,
        sigma=0.5, lattice=False)
    # the periodic cell of 64 atoms with 8 source cubes (the contour's cell) in both precisions
    add("action_f32_cell16", "action", (16, 16, 16), (2, 2, 2), atoms=64, dtype="float32")
    add("action_f64_cell16", "action", (16, 16, 16), (2, 2, 2), atoms=64, kx=0.1, ky=0.2, kz=-0.15)
    # the largest cell: 32^3 cubes, 256 atoms, 32 source cubes inside their truncation spheres
    add("action_f32_wrapped32", "action", (32, 32, 32), (4, 4, 2), atoms=256, dtype="float32")
    # a whole solve of the smallest cell, plain FP64
    add("solve_f64_cell4", "solve", (4, 4, 4), (1, 1, 1), r_trunc=6.0, atoms=1, numax=3, sigma=0.5, Ere=-0.3, Eim=0.05,
        tolerance=1e-9, precondition=False, iterations=220)
    # one point of the contour on the 64-atom cell, one source cube: FP32 recurrences with the FP64
    # solution and the preconditioner
    add("solve_mixed_cell16", "solve", (16, 16, 16), (1, 1, 1), atoms=64, Ere=-0.5, Eim=0.5, kx=0.1, ky=0.2, kz=-0.15,
        tolerance=1e-8, precondition=True, iterations=120, dtype="float32")
    # a contour's worth of (energy, k-point) pairs of the smallest cell as one batch
    add("batch_f64_cell4", "batch", (4, 4, 4), (1, 1, 1), r_trunc=6.0, atoms=1, numax=3, sigma=0.5, Ere=-0.5, Eim=0.5,
        tolerance=1e-8, precondition=True, pairs=16, iterations=60)
    # gradients: potential, atom matrices and positions of the 64-atom cell, one source cube
    add("vjp_cell16", "vjp", (16, 16, 16), (1, 1, 1), atoms=64, kx=0.1, ky=0.2, kz=-0.15)
    # atomic density matrices of a molecule in an isolated box
    add("density_iso10", "density", (10, 10, 10), (3, 3, 3), bc="000", r_trunc=3.0, atoms=8, lattice=False)
    return L


def draw(rng):
    def size(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))

    def kpoint():
        return {k: (0.0 if rng.random() < 0.3 else round(rng.uniform(-0.5, 0.5), 4)) for k in ("kx", "ky", "kz")}

    what = rng.choice(["action"]*6 + ["solve", "batch", "vjp", "density"])
    numax = rng.randint(1, 5)
    sigma = round(rng.uniform(0.35, 0.65), 3)
    if what == "action":
        while True:
            periodic = rng.random() < 0.5
            n = tuple(size(3, 18) for _ in range(3))
            c = _case("action", n, tuple(rng.randint(1, min(4, m)) for m in n),
                      bc="111" if periodic else "".join(rng.choice("0123") for _ in range(3)),
                      hx=round(rng.uniform(0.2, 0.32), 3), hy=round(rng.uniform(0.2, 0.32), 3),
                      hz=round(rng.uniform(0.2, 0.32), 3),
                      r_trunc=12.0 if periodic and rng.random() < 0.5 else round(rng.uniform(1.5, 4.5), 2),
                      order=8 if rng.random() < 0.2 else 4, atoms=size(1, 64), numax=numax, mixed=rng.random() < 0.5,
                      sigma=sigma, lattice=False, dtype=rng.choice(["float32", "float64"]), **kpoint())
            if _layout(c)["blocks"] <= 60000:
                return c
    if what == "solve":
        n = tuple(rng.randint(3, 5) for _ in range(3))
        return _case("solve", n, (rng.randint(1, 2), 1, 1), atoms=rng.randint(0, 2), numax=min(numax, 3), sigma=sigma,
                     lattice=False, Ere=round(rng.uniform(-0.8, -0.2), 3), Eim=round(rng.uniform(0.3, 0.5), 3), tolerance=1e-8,
                     precondition=rng.random() < 0.5, iterations=150, dtype=rng.choice(["float32", "float64"]), **kpoint())
    if what == "batch":
        n = tuple(rng.randint(3, 5) for _ in range(3))
        return _case("batch", n, (1, 1, 1), atoms=rng.randint(0, 2), numax=min(numax, 3), sigma=sigma, lattice=False,
                     Ere=-0.5, Eim=round(rng.uniform(0.35, 0.5), 3), tolerance=1e-8, precondition=rng.random() < 0.5,
                     pairs=rng.randint(2, 16), iterations=100)
    if what == "vjp":
        n = tuple(rng.randint(5, 14) for _ in range(3))
        return _case("vjp", n, (1, 1, rng.randint(1, 2)), atoms=size(1, 40), numax=numax, mixed=rng.random() < 0.5,
                     sigma=sigma, lattice=False, **kpoint())
    n = tuple(rng.randint(5, 12) for _ in range(3))
    return _case("density", n, tuple(rng.randint(1, 3) for _ in range(3)), bc="000", r_trunc=round(rng.uniform(1.5, 3.5), 2),
                 atoms=size(1, 20), numax=numax, sigma=sigma, lattice=False)


# ------------------------------------------------------------------ inputs

def _nsho(numax):
    return (numax + 1)*(numax + 2)*(numax + 3)//6


def _system(case, seed):
    """Geometry, potential [nz, ny, nx], atom matrices and their offsets: Gaussian wells with a
    little noise, symmetric random matrices with a positive overlap, SHO prefactors included.  The
    atoms are the case's own, whatever the seed: which of them a truncated region touches decides
    the shapes of what comes back."""
    rng, place = np.random.default_rng(seed), np.random.default_rng(case["atoms"])
    n = np.array([case["nx"], case["ny"], case["nz"]])
    h = np.array([case["hx"], case["hy"], case["hz"]])
    ng = 4*n
    L = ng*h
    wells = max(4, min(256, int(round(np.prod(L)/64))))
    centres = rng.uniform(-L/2, L/2, size=(wells, 3))
    g = []
    for d in range(3):
        x = (np.arange(ng[d]) - ng[d]/2 + 0.5)*h[d]
        dx = x[None, :] - centres[:, d:d + 1]
        dx -= L[d]*np.round(dx/L[d])
        g.append(np.exp(-dx*dx/(2*1.5*1.5)))
    V = -np.einsum("cz,cyx->zyx", g[2], g[1][:, :, None]*g[0][:, None, :], optimize=True)
    V += rng.uniform(-1e-3, 1e-3, size=V.shape)
    na = case["atoms"]
    atoms = np.zeros((na, 8))
    if case["lattice"] and na > 1:
        m = (8, 8, 4) if na == 256 else (int(round(na**(1/3))),)*3
        assert np.prod(m) == na
        a = np.indices(m).reshape(3, -1).T
        atoms[:, :3] = (a + 0.5)*(L/np.array(m)) - L/2 + place.uniform(-0.3, 0.3, size=(na, 3))
    elif na > 1 or not case["lattice"]:
        atoms[:, :3] = place.uniform(-L/2, L/2, size=(na, 3))
    atoms[:, 3] = 1
    atoms[:, 4] = np.arange(na)
    atoms[:, 5] = place.integers(min(1, case["numax"]), case["numax"] + 1, size=na) if case["mixed"] else case["numax"]
    atoms[:, 6] = case["sigma"]
    mats, offsets, off = [], [], 0
    for a in range(na):
        numax = int(atoms[a, 5])
        ns = _nsho(numax)
        H, S = (np.triu(B) + np.triu(B, 1).T for B in rng.normal(0.0, 0.1, size=(2, ns, ns)))
        S = S + (0.1 - np.linalg.eigvalsh(S)[0])*np.eye(ns)
        f = workloads.sho_prefactors(numax, case["sigma"])
        mats += [(np.outer(f, f)*H).ravel(), (np.outer(f, f)*S).ravel()]
        offsets.append(off)
        off += 2*ns*ns
    mats = np.concatenate(mats) if mats else np.zeros(1)
    geometry = workloads.Geometry(tuple(int(v) for v in ng), tuple(int(b) for b in case["bc"]), tuple(float(v) for v in h),
                                  case["r_trunc"], (case["sx"], case["sy"], case["sz"]), case["order"],
                                  PROJECTION_RADIUS, atoms)
    return geometry, V, mats, np.array(offsets, np.int64), float(np.prod(h))


def _blocks(nnzb, seed, dtype, device):
    gen = torch.Generator(device=device).manual_seed(seed)
    return torch.randn((nnzb, 2, 64, 64), device=device, dtype=dtype, generator=gen)


def _pairs(case, seed):
    """The (energy, k-point) pairs of a batch: the upper arc of the contour from -1 to 0 Hartree."""
    rng = np.random.default_rng(seed)
    n = case["pairs"]
    theta = np.pi*(0.25 + 0.5*(np.arange(n) + 0.5)/n)
    return case["Ere"] + case["Eim"]*np.exp(1j*theta), rng.uniform(-0.5, 0.5, size=(n, 3))


def prepare(case, seed):
    geometry, V, mats, offsets, dVol = _system(case, seed)
    plan = green_function.construct_Green_function(geometry)
    some = len(offsets) > 0
    green_function.update_potential(plan, V, mats if some else None, offsets if some else None)
    green_function.update_energy_parameter(plan, complex(case["Ere"], case["Eim"]), dVol)
    green_function.update_phases(plan, (case["kx"], case["ky"], case["kz"]))
    plan.upload()
    s = {"case": case, "plan": plan, "dVol": dVol}
    dtype = getattr(torch, case["dtype"])
    if case["call"] == "action":
        s["op"] = green_action.action_t(plan, case["dtype"])
        s["x"] = _blocks(plan.nnzb, seed, dtype, "cuda")
        s["y"] = torch.empty_like(s["x"])
        s["colindx"] = torch.from_numpy(plan.export()["colindx"].astype(np.int16)).cuda()
    elif case["call"] == "solve":
        s["X"] = torch.empty((plan.nnzb, 2, 64, 64), device="cuda", dtype=torch.float64)
        s["stream"] = torch.cuda.Stream()
    elif case["call"] == "batch":
        s["E"], s["K"] = _pairs(case, seed)
        s["stream"] = torch.cuda.Stream()
    elif case["call"] == "vjp":
        s["L"] = _blocks(plan.nnzb, seed, dtype, "cuda")
        s["G"] = _blocks(plan.nnzb, seed + 1000003, dtype, "cuda")
    else:
        s["G"] = _blocks(plan.nnzb, seed, dtype, "cuda")
    return s


def run(state):
    case, plan = state["case"], state["plan"]
    if case["call"] == "action":
        state["op"].multiply(state["y"], state["x"], state["colindx"], plan.nnzb, plan.nCols)
        return state["y"]
    if case["call"] in ("solve", "batch"):
        options = dict(tolerance=case["tolerance"], max_iterations=2000, precision=case["dtype"],
                       precondition=case["precondition"], stream=state["stream"])
        if case["call"] == "solve":
            _, rho = green_action.solve(plan, X=state["X"], **options)
            return state["X"], rho
        _, rho = green_action.solve_batched(plan, state["E"], state["K"], state["dVol"], want_rho=True, **options)
        return rho
    if case["call"] == "vjp":
        g = green_action.vjp(plan, state["L"], state["G"])
        return g["V"], np.concatenate([m.ravel() for m in g["M"]]), g["R"]
    D = green_action.get_projection_coefficients(plan, state["G"])
    return np.concatenate([m.ravel() for m in D])


# ------------------------------------------------------------------ work and tolerances

def _truncated(case):
    """Spacings of the truncation test and boundary conditions with it (4: a periodic direction
    that the truncation sphere fits into)."""
    h, bc = [case["hx"], case["hy"], case["hz"]], [int(b) for b in case["bc"]]
    n = [case["nx"], case["ny"], case["nz"]]
    for d in range(3):
        if bc[d] == 1:
            if 2*case["r_trunc"] > h[d]*4*n[d]:
                h[d] = 0.0
            else:
                bc[d] = 4
    return h, bc


def _layout(case):
    """The blocks of the Green function in their order: target cubes t (in cells of the grid) and
    sources s, rows in z, y, x order and the sources ascending in a row."""
    n = np.array([case["nx"], case["ny"], case["nz"]])
    h, bc = _truncated(case)
    ns = np.minimum(np.array([case["sx"], case["sy"], case["sz"]]), n)
    off = (n - ns)//2
    src = np.array([[x, y, z] for z in range(ns[2]) for y in range(ns[1]) for x in range(ns[0])]) + off
    rbcs = 1.5*math.sqrt(case["hx"]**2 + case["hy"]**2 + case["hz"]**2)
    r = case["r_trunc"]
    axes = []
    for d in range(3):
        it = int(math.floor((r + 2*rbcs)/(4*h[d]))) if h[d] > 0 else int(n[d]) - 1
        if bc[d] == 1:
            it = min(it, int(n[d]) - 1)
        axes.append(np.arange(-it, it + 1))
    bz, by, bx = (v.ravel() for v in np.meshgrid(axes[2], axes[1], axes[0], indexing="ij"))
    b = (bx, by, bz)
    d2 = (4*bx*h[0])**2 + (4*by*h[1])**2 + (4*bz*h[2])**2
    far = d2 > (3*rbcs)**2

    def nearest(d):
        ends = np.minimum(((4*b[d] - 3)*h[d])**2, ((4*b[d] + 3)*h[d])**2)
        return np.where(far, ends, np.minimum(ends, (4*b[d]*h[d])**2))

    inside = (d2 < (r + 2*rbcs)**2) & (nearest(0) + (nearest(1) + nearest(2)) < r*r)
    offsets = np.stack([v[inside] for v in b], axis=1)
    t, s = [], []
    for i, c in enumerate(src):
        q = offsets + c
        keep = np.ones(len(q), bool)
        for d in range(3):
            if bc[d] in (0, 1):
                keep &= (q[:, d] >= 0) & (q[:, d] < n[d])
        t.append(q[keep])
        s.append(np.full(int(keep.sum()), i))
    t, s = np.concatenate(t), np.concatenate(s)
    order = np.lexsort((s, t[:, 0], t[:, 1], t[:, 2]))
    return {"t": t[order], "s": s[order], "sources": src, "blocks": len(s), "bc": bc, "n": n}


def _images(case, atoms, lay):
    """The atom images that touch a target cube: position, atom copy, shift of the phase and the
    target cubes touched (one of the 8 corner points of the cube inside the projection sphere)."""
    n, bc = lay["n"], lay["bc"]
    h = np.array([case["hx"], case["hy"], case["hz"]])
    cell = 4*n*h
    rbcs = 1.5*math.sqrt(float((h*h).sum()))
    rows, inv = np.unique(lay["t"][:, ::-1], axis=0, return_inverse=True)
    rows = rows[:, ::-1] - 0.5*n
    src = lay["sources"]
    reach = math.sqrt(float(((((src - 0.5*(src.min(0) + src.max(0)))*4*h))**2).sum(1).max()))
    radius = case["r_trunc"] + reach + 2*case["sigma"]*PROJECTION_RADIUS + 2*rbcs
    m = [int(max(0, math.ceil(radius/cell[d]))) for d in range(3)]
    nimg = [m[d] if bc[d] == 1 else 0 for d in range(3)]
    ncpy = [m[d] if bc[d] == 3 else (1 if bc[d] == 4 else 0) for d in range(3)]

    def box(k):
        return [np.array([x, y, z]) for z in range(-k[2], k[2] + 1) for y in range(-k[1], k[1] + 1)
                for x in range(-k[0], k[0] + 1)]

    found = []
    corner = [(rows*4 + i)*h for i in (0.5, 3.5)]
    for shift in box(nimg):
        for a in range(len(atoms)):
            for ic, copy in enumerate(box(ncpy)):
                pos = atoms[a, :3] + (shift + copy)*cell
                rp = PROJECTION_RADIUS*atoms[a, 6]
                near = (((rows*4 + 2.0)*h - pos)**2).sum(1) <= (rp + rbcs)**2
                best = sum(np.minimum((corner[0][:, d] - pos[d])**2, (corner[1][:, d] - pos[d])**2) for d in range(3))
                hit = np.flatnonzero(near & (best < rp*rp))
                if len(hit):
                    found.append({"pos": pos, "copy": (a, ic), "shift": shift, "rows": hit})
    return found, rows, inv


def work(case):
    lay = _layout(case)
    blocks, cols = lay["blocks"], len(lay["sources"])*64
    size = 8 if case["dtype"] == "float64" else 4
    vector = blocks*8192*size
    # projection spheres cover this many cubes of a source's targets, 944 multiply-adds a column
    # at the basis size 5 (sum-factorized), each way
    sphere = 4/3*math.pi*(PROJECTION_RADIUS*case["sigma"])**3
    density = case["atoms"]/(64.0*case["nx"]*case["ny"]*case["nz"]*case["hx"]*case["hy"]*case["hz"])
    l, ns = case["numax"], _nsho(case["numax"])
    pair = 64*(l + 1) + 8*(l + 1)*(l + 2) + 4*ns
    pairs = blocks*density*sphere
    local = blocks*4096*2*2*(3*(2*case["order"] + 1) + 3)
    action = local + 2*pairs*128*pair*2 + case["atoms"]*cols*8*ns*ns
    if case["call"] == "action":
        return {"bytes": 2*vector, "flops": action}
    if case["call"] in ("solve", "batch"):
        k = case["iterations"]*case.get("pairs", 1)
        passes = 21 + 2*2*(2 if case["precondition"] else 1)
        return {"bytes": k*passes*vector, "flops": k*2*action}
    if case["call"] == "vjp":
        return {"bytes": 2*vector, "flops": blocks*4096*8 + 8*pairs*128*pair*2 + case["atoms"]*cols*(4*8 + 8)*ns*ns}
    return {"bytes": vector, "flops": pairs*128*pair*2 + case["atoms"]*cols*4*ns*ns}


def tolerance(case):
    if case["call"] in ("solve", "batch"):
        # the solution to a relative residual of 1e-8 or 1e-9, whatever the iterates' rounding
        return {"rel": 100*case["tolerance"], "max": 4000*case["tolerance"]}
    # measured against exact(): 1.1e-7 and 2.6e-16 for the actions, 2.1e-15 for the sums over all
    # columns of the gradients and density matrices
    if case["call"] == "action":
        return {"rel": 5e-7} if case["dtype"] == "float32" else {"rel": 2e-15}
    return {"rel": 1e-14}


# ------------------------------------------------------------------ the operator in plain torch

def _weights(case, d, periodic):
    """One half of the finite-difference second derivative of direction d times -1/2."""
    h = (case["hx"], case["hy"], case["hz"])[d]
    if case["order"] == 8 and not periodic:
        w = np.array([-924708642, 538137600, -94174080, 22830080, -5350800, 1053696, -156800, 15360, -735])/302702400
    else:
        w = np.array([-14350, 8064, -1008, 128, -9])/5040
    return -0.5/(h*h)*w


class _Operator:
    """(H - E S) of a case on its blocks [nnzb, 64 points, 64 columns], complex 64-bit torch."""

    def __init__(self, case, seed, E, k, device):
        geometry, V, mats, offsets, dVol = _system(case, seed)
        self.case, self.device, self.E = case, device, complex(E)
        lay = self.lay = _layout(case)
        n, bc, t = lay["n"], lay["bc"], lay["t"]
        self.source = torch.from_numpy(lay["s"]).to(device)
        given = np.ones(len(t), bool)
        for d in range(3):
            if bc[d] in (0, 2):
                given &= (t[:, d] >= 0) & (t[:, d] < n[d])
        m = t % n
        cells = torch.from_numpy(V.reshape(n[2], 4, n[1], 4, n[0], 4).transpose(0, 2, 4, 1, 3, 5).reshape(-1, 64)).to(device)
        self.cell = torch.from_numpy((m[:, 2]*n[1] + m[:, 1])*n[0] + m[:, 0]).to(device)
        self.given = torch.from_numpy(given).to(device)
        self.V = torch.where(self.given[:, None], cells[self.cell], torch.zeros((), dtype=torch.float64, device=device))
        self.phase = [complex(math.cos(2*math.pi*v), math.sin(2*math.pi*v)) for v in k]
        self.periodic = [b == 1 for b in bc]
        # the block before and after each one on its line (-1: none): the cubes of a source that follow
        # each other on a line of the truncated region are neighbours, and the ends of a periodic
        # direction meet
        self.next, self.ends = [], []
        for d in range(3):
            a, b = (t[:, e] for e in range(3) if e != d)
            o = np.lexsort((t[:, d], a, b, lay["s"]))
            same = (a[o][1:] == a[o][:-1]) & (b[o][1:] == b[o][:-1]) & (lay["s"][o][1:] == lay["s"][o][:-1])
            nxt, ends = np.full((2, len(o)), -1), np.ones((2, len(o)), bool)
            nxt[0, o[1:][same]], nxt[1, o[:-1][same]] = o[:-1][same], o[1:][same]
            ends[0, o[1:][same]] = ends[1, o[:-1][same]] = False
            if bc[d] == 1:
                first, last = o[np.r_[True, ~same]], o[np.r_[~same, True]]
                nxt[0, first], nxt[1, last] = last, first
            self.next.append(torch.from_numpy(nxt).to(device))
            self.ends.append(torch.from_numpy(ends).to(device))
        self.images, rows, inv = _images(case, geometry.xyzZinso, lay)
        order = np.argsort(inv, kind="stable")
        first = np.searchsorted(inv[order], np.arange(len(rows) + 1))
        self.copies = sorted({im["copy"] for im in self.images})
        self.numax = [int(geometry.xyzZinso[a, 5]) for a, _ in self.copies]
        self.M = []
        for (a, _), l in zip(self.copies, self.numax):
            ns = _nsho(l)
            H = mats[offsets[a]:offsets[a] + ns*ns].reshape(ns, ns)
            S = mats[offsets[a] + ns*ns:offsets[a] + 2*ns*ns].reshape(ns, ns)
            self.M.append(torch.from_numpy((H - self.E*S)*dVol).to(device))
        for im in self.images:
            im["l"] = int(geometry.xyzZinso[im["copy"][0], 5])
            im["sigma"] = float(geometry.xyzZinso[im["copy"][0], 6])
            count = first[im["rows"] + 1] - first[im["rows"]]
            im["blocks"] = torch.from_numpy(np.concatenate([order[first[r]:first[r + 1]] for r in im["rows"]])).to(device)
            im["slot"] = torch.from_numpy(np.repeat(np.arange(len(count)), count)).to(device)
            im["corner"] = rows[im["rows"]]
            im["phase"] = complex(np.prod([self.phase[d]**int(im["shift"][d]) for d in range(3)]))

    def functions(self, im, corner, derivative=None):
        """Projector functions [cubes, nSHO, 64] of an image on cubes; derivative: with respect to
        that coordinate of the atom's position."""
        l, sinv = im["l"], 1/im["sigma"]
        h = (self.case["hx"], self.case["hy"], self.case["hz"])
        R2 = PROJECTION_RADIUS**2
        f, x2 = [], []
        for d in range(3):
            xi = sinv*((corner[:, d:d + 1]*4 + np.arange(4) + 0.5)*h[d] - im["pos"][d])
            H = [np.where(xi*xi < R2, np.exp(-0.5*xi*xi), 0.0)]
            for nu in range(l):
                H.append(xi*H[nu] - (0.5*nu*H[nu - 1] if nu else 0.0))
            if derivative == d:
                H = [-sinv*((nu*H[nu - 1] if nu else 0.0) - xi*H[nu]) for nu in range(l + 1)]
            f.append(np.stack(H, axis=1))
            x2.append((xi*xi).astype(np.float32))
        # the mask of the sphere is decided in 32 bits
        z = (x2[2] - np.float32(R2))[:, :, None, None]
        mask = (x2[0][:, None, None, :] + (x2[1][:, None, :, None] + z)) < 0
        P = [f[2][:, iz, :, None, None]*f[1][:, iy, None, :, None]*f[0][:, ix, None, None, :]
             for iz in range(l + 1) for iy in range(l + 1 - iz) for ix in range(l + 1 - iz - iy)]
        return torch.from_numpy((np.stack(P, axis=1)*mask[:, None]).reshape(len(corner), -1, 64)).to(self.device)

    def project(self, X, conj=False, derivative=None):
        """Coefficients of every atom copy: [sources, nSHO, 64 columns], the images' phases included."""
        cols = len(self.lay["sources"])
        out = [torch.zeros((cols, _nsho(l), 64), dtype=torch.complex128, device=self.device) for l in self.numax]
        for im in self.images:
            P = self.functions(im, im["corner"], derivative)
            x = X[im["blocks"]]
            c = torch.view_as_complex(torch.bmm(P[im["slot"]], torch.view_as_real(x).reshape(len(x), 64, 128))
                                      .reshape(len(x), -1, 64, 2))
            ph = im["phase"].conjugate() if conj else im["phase"]
            out[self.copies.index(im["copy"])].index_add_(0, self.source[im["blocks"]], c*ph)
        return out

    def _window(self, X, d, reach, at):
        """The points of cubes `at` and of their neighbours up to `reach` points along direction d:
        [cubes, 4 + 2 reach, ...] with the direction's points second."""
        axis = 3 - d
        parts = []
        for side in (0, 1):
            phase = self.phase[d] if side == 0 else self.phase[d].conjugate()
            at_side, wrapped = at, torch.zeros(len(at), dtype=torch.bool, device=self.device)
            for _ in range(0, reach, 4):
                nxt = torch.where(at_side < 0, at_side, self.next[d][side][at_side])
                wrapped = wrapped | ((at_side >= 0) & self.ends[d][side][at_side])
                at_side = nxt
                x = X[at_side.clamp(min=0)]
                x[at_side < 0] = 0
                x[wrapped] *= phase
                x = x.reshape(-1, 4, 4, 4, 64).movedim(axis, 1)
                parts = [x] + parts if side == 0 else parts + [x]
            if side == 0:
                parts.append(X[at].reshape(-1, 4, 4, 4, 64).movedim(axis, 1))
        return torch.cat(parts, dim=1)

    def local(self, X):
        Y = torch.empty_like(X)
        for k in range(0, len(X), 4096):
            at = torch.arange(k, min(k + 4096, len(X)), device=self.device)
            total = ((self.V[at][:, :, None] - self.E)*X[at]).reshape(-1, 4, 4, 4, 64)
            for d in range(3):
                w = _weights(self.case, d, self.periodic[d])
                R = len(w) - 1
                p = self._window(X, d, R, at)
                y = w[0]*p[:, R:R + 4]
                for i in range(1, R + 1):
                    y += w[i]*(p[:, R - i:R - i + 4] + p[:, R + i:R + i + 4])
                total += y.movedim(1, 3 - d)
            Y[at] = total.reshape(-1, 64, 64)
        return Y

    def action(self, X):
        Y = self.local(X)
        C = [torch.matmul(M, c) for M, c in zip(self.M, self.project(X))]
        for im in self.images:
            P = self.functions(im, im["corner"])
            c = (C[self.copies.index(im["copy"])]*im["phase"].conjugate())[self.source[im["blocks"]]]
            c = torch.view_as_real(c).reshape(len(c), -1, 128)
            y = torch.bmm(P[im["slot"]].transpose(1, 2), c).reshape(len(c), 64, 64, 2)
            Y[im["blocks"]] += torch.view_as_complex(y)
        return Y


def _to_complex(x):
    x = x.double()
    return torch.complex(x[:, 0], x[:, 1])


def _solutions(case, seed, E, k, device):
    """Blocks of the inverse of the operator on an untruncated cell, by a dense solve."""
    n = (case["nx"], case["ny"], case["nz"])
    every = dict(case, sx=n[0], sy=n[1], sz=n[2])
    op = _Operator(every, seed, E, k, device)
    cubes = n[0]*n[1]*n[2]
    eye = torch.zeros((cubes*cubes, 64, 64), dtype=torch.complex128, device=device)
    eye[torch.arange(cubes, device=device)*(cubes + 1)] = torch.eye(64, dtype=torch.complex128, device=device)
    A = op.action(eye).reshape(cubes, cubes, 64, 64).permute(0, 2, 1, 3).reshape(cubes*64, cubes*64)
    lay = _layout(case)
    cube = (lay["sources"][:, 2]*n[1] + lay["sources"][:, 1])*n[0] + lay["sources"][:, 0]
    B = torch.zeros((cubes, 64, len(cube), 64), dtype=torch.complex128, device=device)
    for i, c in enumerate(cube):
        B[int(c), :, i] = torch.eye(64, dtype=torch.complex128, device=device)
    X = torch.linalg.solve(A, B.reshape(cubes*64, -1)).reshape(cubes, 64, len(cube), 64)
    rho = np.stack([torch.diagonal(X[int(c), :, i]).cpu().numpy()/math.pi for i, c in enumerate(cube)])
    return X.permute(0, 2, 1, 3).reshape(-1, 64, 64), rho


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    E, k = complex(case["Ere"], case["Eim"]), (case["kx"], case["ky"], case["kz"])
    if case["call"] in ("solve", "batch"):
        if case["nx"]*case["ny"]*case["nz"] > 125 or any(_truncated(case)[0]):
            return None                   # too large for a dense inverse, or truncated
        if case["call"] == "solve":
            X, rho = _solutions(case, seed, E, k, device)
            return torch.stack([X.real, X.imag], dim=1), rho
        energies, kpoints = _pairs(case, seed)
        return np.stack([_solutions(case, seed, e, q, device)[1] for e, q in zip(energies, kpoints)])
    op = _Operator(case, seed, E, k, device)
    dtype = getattr(torch, case["dtype"])
    if case["call"] == "action":
        Y = op.action(_to_complex(_blocks(op.lay["blocks"], seed, dtype, device)))
        return torch.stack([Y.real, Y.imag], dim=1)
    if case["call"] == "density":
        C = op.project(_to_complex(_blocks(op.lay["blocks"], seed, dtype, device)))
        corner = op.lay["sources"] - 0.5*op.lay["n"]
        out = []
        for im in sorted(op.images, key=lambda im: im["copy"]):
            P = op.functions(im, corner).to(torch.complex128)
            c = C[op.copies.index(im["copy"])]
            out.append(torch.einsum("sic,sjc->ij", c, P).imag.cpu().numpy().ravel())
        return np.concatenate(out)
    L = _to_complex(_blocks(op.lay["blocks"], seed, dtype, device))
    G = _to_complex(_blocks(op.lay["blocks"], seed + 1000003, dtype, device))
    dV = torch.zeros((case["nx"]*case["ny"]*case["nz"], 64), dtype=torch.complex128, device=device)
    dV.index_add_(0, op.cell[op.given], (L*G).sum(2)[op.given])
    l, g = op.project(L, conj=True), op.project(G)
    dM = [torch.einsum("sic,sjc->ij", a, b) for a, b in zip(l, g)]
    dR = torch.zeros((len(l), 3), dtype=torch.complex128, device=device)
    for d in range(3):
        dl, dg = op.project(L, conj=True, derivative=d), op.project(G, derivative=d)
        for a, M in enumerate(op.M):
            dR[a, d] = (dl[a]*torch.matmul(M, g[a])).sum() + (l[a]*torch.matmul(M, dg[a])).sum()
    return dV.cpu().numpy(), np.concatenate([m.cpu().numpy().ravel() for m in dM]), dR.cpu().numpy()
