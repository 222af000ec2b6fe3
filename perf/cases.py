"""The work this framework is timed on: calls of its public entry points over the sizes, forms and
precisions its decks, tests and benchmark use.

Every case is one of six calls a program makes:

``divtau``      ``ks_divtau_noalloc`` on caller-owned device buffers (the allocation-free viscous term);
``projection``  ``ApplyProjection``, the nodal projection of a given velocity;
``steps``       one Evolve step from each of two stored snapshots of a run (``set_field``, step, ``get_field``), as a
                program does that restarts members of an ensemble or forms one-step targets from stored data:
                Taylor-Green, neutral ABL, MOL and stratified ABL decks;
``farm``        the same for the ABL with a wind farm (actuator disks, fixed dt);
``adjoint``     one reverse step at a stored state from stored terminal adjoints, as a gradient driver
                calls it (the step recomputes its own forward step).

The pressure of these boxes (periodic or Neumann everywhere) is defined up to a constant, so ``p`` is
returned without its mean.  The mixed-precision form states its fields to single precision and they are
handed on as FP32 tensors; FP64 forms return FP64.
"""
import ctypes
import math

import numpy as np
import torch

import kynema_sgf_gb300 as ks
from kynema_sgf_gb300 import decks

MEMBERS = 2  # snapshots of one pass, each advanced by one Evolve step
APART = 3  # steps of the run between them


def listed():
    return [
        # the smallest call: the viscous term of a plug-in's 32 x 32 x 16 block, three kernels' worth of launches
        {"name": "divtau_32", "kind": "divtau", "nx": 32, "ny": 32, "nz": 16, "wall": True},
        # small Taylor-Green boxes (tests, the reference's own verification case): bound by launches and host waits
        {"name": "tgv_32", "kind": "steps", "flow": "tgv", "nx": 32, "ny": 32, "nz": 32, "dz": 1.0, "mixed": False, "semi": False},
        {"name": "tgv_64", "kind": "steps", "flow": "tgv", "nx": 64, "ny": 64, "nz": 64, "dz": 1.0, "mixed": False, "semi": False},
        # one nodal projection on counts that are no powers of two
        {"name": "projection_160x96x80", "kind": "projection", "nx": 160, "ny": 96, "nz": 80, "dz": 20.0, "wall": True},
        # MOL predictor-corrector on the benchmark's 20 x 20 x 10 m cells (two MAC and two nodal solves a step)
        {"name": "mol_128", "kind": "steps", "flow": "mol", "nx": 128, "ny": 128, "nz": 64, "dz": 10.0, "mixed": False, "semi": False},
        # the reference's abl_godunov physics (temperature, buoyancy, Crank-Nicolson diffusion), 96^3
        {"name": "stratified_96", "kind": "steps", "flow": "stratified", "nx": 96, "ny": 96, "nz": 96, "dz": 1.0, "mixed": False, "semi": False},
        # the benchmark box: 256 x 256 x 128 cells of 20 x 20 x 10 m, FP64 and mixed precision
        {"name": "abl_256_fp64", "kind": "steps", "flow": "abl", "nx": 256, "ny": 256, "nz": 128, "dz": 10.0, "mixed": False, "semi": False},
        {"name": "abl_256_mixed", "kind": "steps", "flow": "abl", "nx": 256, "ny": 256, "nz": 128, "dz": 10.0, "mixed": True, "semi": False},
        # ragged counts with the deck's MAC semicoarsening on
        {"name": "abl_192x160x96_semi", "kind": "steps", "flow": "abl", "nx": 192, "ny": 160, "nz": 96, "dz": 10.0, "mixed": False, "semi": True},
        # reverse step of the three-disk gradient check (FP64) and of a 16-disk farm (mixed precision)
        {"name": "adjoint_c3_128", "kind": "adjoint", "nx": 128, "ny": 128, "nz": 64, "walls": False, "mixed": False},
        {"name": "adjoint_farm_256", "kind": "adjoint", "nx": 256, "ny": 256, "nz": 128, "walls": True, "mixed": True},
        # production wind farm: 67 million cells, 16 disks, mixed precision
        {"name": "farm_512_mixed", "kind": "farm", "nx": 512, "ny": 512, "nz": 256, "mixed": True},
    ]


def _count(rng, lo, hi, mult):
    """A cell count between lo and hi, spread over its logarithm, a multiple of mult."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, mult * round(x / mult))))


def _box(rng, hi, zhi, mixed):
    """Counts of a box.  FP64 boxes take counts that multigrid coarsens far enough for its solves to reach the
    tolerance of an FP64 result; single precision is met on counts of larger odd factors too."""
    if mixed:
        return _count(rng, 32, hi, 16), _count(rng, 32, hi, 16), _count(rng, 32, zhi, 16)
    xy = [n for n in (32, 64, 96, 128, 160, 192, 256) if n <= hi]
    z = [n for n in (32, 64, 96, 128) if n <= zhi]
    return rng.choice(xy), rng.choice(xy), rng.choice(z)


def draw(rng):
    kind = rng.choice(["divtau", "projection", "tgv", "abl", "abl", "mol", "stratified", "farm", "adjoint"])
    if kind == "divtau":
        return {"kind": "divtau", "nx": _count(rng, 8, 128, 2), "ny": _count(rng, 8, 64, 2), "nz": _count(rng, 4, 32, 2), "wall": rng.random() < 0.5}
    if kind == "tgv":
        n = _count(rng, 16, 96, 8)
        return {"kind": "steps", "flow": "tgv", "nx": n, "ny": n, "nz": n, "dz": 1.0, "mixed": rng.random() < 0.3, "semi": False}
    mixed = rng.random() < 0.5 and kind in ("abl", "farm", "adjoint")
    nx, ny, nz = _box(rng, 192 if kind == "adjoint" else 256, 96, mixed)
    if kind == "projection":
        return {"kind": "projection", "nx": nx, "ny": ny, "nz": nz, "dz": rng.choice([10.0, 20.0]), "wall": rng.random() < 0.7}
    if kind in ("abl", "mol"):
        return {"kind": "steps", "flow": kind, "nx": nx, "ny": ny, "nz": nz, "dz": rng.choice([10.0, 20.0]), "mixed": mixed, "semi": mixed and rng.random() < 0.5}
    if kind == "stratified":
        return {"kind": "steps", "flow": "stratified", "nx": min(nx, 128), "ny": min(ny, 128), "nz": nz, "dz": 1.0, "mixed": False, "semi": False}
    if kind == "farm":
        return {"kind": "farm", "nx": max(96, nx), "ny": max(96, ny), "nz": max(64, nz), "mixed": mixed}
    return {"kind": "adjoint", "nx": max(64, nx), "ny": max(64, ny), "nz": nz, "walls": rng.random() < 0.5, "mixed": mixed}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _smooth_noise(shape, g, amp):
    """Uniform noise with its neighbours averaged in along every axis: resolved turbulence rather than white noise."""
    v = 2.0 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 1.0
    for ax in (1, 2, 3):
        v = 0.5 * v + 0.25 * (torch.roll(v, 1, ax) + torch.roll(v, -1, ax))
    return amp * v


def _shared_keys(case):
    # dt starts at its CFL limit instead of growing to it over the first 25 steps
    out = "time.init_shrink = 1.0\n"
    if case.get("mixed"):
        out += "ks.precision = mixed\n"
    if case.get("semi"):
        out += "mac_proj.do_semicoarsening = true\n"
    return out


def _flow_deck(case, seed):
    nx, ny, nz, flow = case["nx"], case["ny"], case["nz"], case["flow"]
    steps = 10 ** 8
    if flow == "tgv":
        deck = decks.tgv(nx, steps=steps)
    elif flow == "abl":
        deck = decks.abl(nx, ny, nz, steps=steps, dz=case["dz"], seed=seed % 100003)
    elif flow == "mol":
        deck = decks.mol(decks.abl(nx, ny, nz, steps=steps, dz=case["dz"], cfl=0.45, seed=seed % 100003))
    else:
        h = 1000.0 / 48
        deck = decks.abl_temperature((nx, ny, nz), steps=steps, diffusion_type=1, size=(nx * h, ny * h, 1000.0))
    return deck + _shared_keys(case)


def _farm_deck(case, seed, ngrid):
    """The wind-farm ABL on 10 m cells: an ngrid x ngrid array of disks that spans the box, hub height one diameter."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    pitch = min(nx, ny) // ngrid
    dcells = max(4, pitch // 7)
    return decks.abl_disks(nx, ny, nz, dcells=dcells, ngrid=ngrid, spacing=pitch / dcells, seed=seed % 100003,
                           precision="mixed" if case["mixed"] else "fp64")


def _stir(sim, seed, amp):
    """Resolved turbulence added to the whole initial velocity, as a spun-up precursor run leaves it."""
    v = sim.get_field("velocity", out=torch.empty(sim.layout("velocity"), dtype=torch.float64, device="cuda"))
    v += _smooth_noise(tuple(v.shape), _gen(seed), amp)
    torch.cuda.synchronize()
    sim.set_field("velocity", v)


def _snapshot(sim, names):
    return {f: sim.get_field(f, out=torch.empty(sim.layout(f), dtype=torch.float64, device="cuda")) for f in names}


def _buffers(state, names):
    return {f: torch.empty_like(state[f]) for f in names}


def prepare(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind == "divtau":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        g = _gen(seed)
        vel = _smooth_noise((3, nz, ny, nx), g, 0.5)
        vel[0] += 8.0
        mu = 0.5 + torch.rand((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64)
        wg = 0.1 * torch.rand((2, ny, nx), generator=g, device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        return {"case": case, "lib": ks.load_library(), "vel": vel, "mu": mu, "wg": wg, "out": torch.empty_like(vel)}
    if kind == "projection":
        deck = decks.abl(case["nx"], case["ny"], case["nz"], steps=10 ** 8, dz=case["dz"])
        if not case["wall"]:
            deck = deck.replace("geometry.is_periodic = 1 1 0", "geometry.is_periodic = 1 1 1")
        sim = ks.Incflo(deck)
        names = ("velocity", "gp", "p")
        first = _snapshot(sim, names)
        first["velocity"] = _projection_velocity(case, seed)
        torch.cuda.synchronize()
        return {"case": case, "sim": sim, "first": first, "out": _buffers(first, names)}
    if kind == "adjoint":
        if case["walls"]:
            deck, lo, hi, _ = _farm_deck(case, seed, 4)
        else:
            deck, lo, hi, _ = decks.adjoint_c3(case["nx"], case["ny"], case["nz"], dcells=case["nx"] // 8, seed=seed % 100003)
            if case["mixed"]:
                deck += "ks.precision = mixed\n"
        sim = ks.Incflo(deck)
        _stir(sim, seed, 0.5)
        sim.InitData()
        sim.set_objective_box(lo, hi)
        first = _snapshot(sim, ("velocity", "gp"))
        # the adjoints a sweep carries into this step: the objective's own seed and a pressure-gradient part
        sim.objective(seed=True)
        bar = _snapshot(sim, ("velocity_adjoint", "gp_adjoint"))
        bar["gp_adjoint"] = _smooth_noise(tuple(bar["gp_adjoint"].shape), _gen(seed), 0.1 * float(bar["velocity_adjoint"].abs().max()))
        torch.cuda.synchronize()
        return {"case": case, "sim": sim, "first": first, "bar": bar, "out": _buffers(bar, ("velocity_adjoint", "gp_adjoint"))}
    if kind == "farm":
        deck, _, _, _ = _farm_deck(case, seed, 4)
        names = ("velocity", "gp", "p")
        sim = ks.Incflo(deck)
        _stir(sim, seed, 0.5)
    else:
        deck = _flow_deck(case, seed)
        names = ("velocity", "gp", "p") + (("temperature",) if case["flow"] == "stratified" else ())
        sim = ks.Incflo(deck)
        if case["flow"] in ("tgv", "stratified"):  # decks without a noise seed of their own
            _stir(sim, seed, 0.05)
    sim.InitData()
    members = [_snapshot(sim, names)]
    while len(members) < MEMBERS:
        sim.Evolve(APART)
        members.append(_snapshot(sim, names))
    return {"case": case, "sim": sim, "members": members, "out": _buffers(members[0], names)}


# ---------------------------------------------------------------- one pass
def _read(state, names):
    """The fields as the program hands them on (see the module docstring)."""
    got = {}
    for f in names:
        x = state["sim"].get_field(f, out=state["out"][f])
        if f == "p":
            x = x - x.mean()
        got[f] = x.float() if state["case"].get("mixed") else x.clone()
    return got


def run(state):
    case = state["case"]
    if case["kind"] == "divtau":
        def ptr(t):
            return ctypes.c_void_p(t.data_ptr())
        rc = state["lib"].ks_divtau_noalloc(ptr(state["vel"]), ptr(state["mu"]), ptr(state["wg"]) if case["wall"] else None, ptr(state["out"]),
                                            case["nx"], case["ny"], case["nz"], 20.0, 20.0, 10.0, 0, 1 if case["wall"] else 0,
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError("ks_divtau_noalloc: status %d" % rc)
        return state["out"]
    sim = state["sim"]
    if "members" in state:
        got = []
        for member in state["members"]:
            for f, x in member.items():
                sim.set_field(f, x)
            sim.Evolve(1)
            got.append(_read(state, tuple(member)))
        return got
    for f, x in state["first"].items():
        sim.set_field(f, x)
    if case["kind"] == "projection":
        sim.ApplyProjection(0.0, 1.0, False)
        return _read(state, ("velocity", "gp", "p"))
    if case["kind"] == "adjoint":
        sim.adjoint_reset()
        for f, x in state["bar"].items():
            sim.set_field(f, x)
        sim.adjoint_step()
        got = _read(state, ("velocity_adjoint", "gp_adjoint"))
        got["ct_gradient"] = sim.ct_gradient().astype(np.float32 if case["mixed"] else np.float64)
        return got
    raise ValueError(case["kind"])


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    n = float(case["nx"]) * case["ny"] * case["nz"]
    real = 8.0
    if case["kind"] == "divtau":
        # read the velocity and the viscosity, write the term; nine face fluxes of about 20 flops and their differences
        return {"bytes": real * 7 * n, "flops": 250.0 * n}
    # a Poisson problem on a uniform periodic-by-periodic grid: transforms along two directions and back
    # (2.5 log2 n flops a real value each way), a tridiagonal solve along the third
    solve = (5.0 * math.log2(float(case["nx"]) * case["ny"]) + 8.0) * n
    if case["kind"] == "projection":
        return {"bytes": real * 14 * n, "flops": solve + 80.0 * n}
    # one Godunov step: edges, traces, transverse corrections and fluxes of three components on three face
    # sets (about 900 flops a cell), two viscous terms, viscosity and sources (about 600), two Poisson solves
    step = 1500.0 * n + 2 * solve
    if case["kind"] == "adjoint":
        # the forward step, and its transpose at twice the arithmetic
        return {"bytes": real * 24 * n, "flops": 3 * step}
    if case["kind"] == "farm":
        return {"bytes": MEMBERS * real * 14 * n, "flops": MEMBERS * step}
    if case["flow"] == "mol":
        return {"bytes": MEMBERS * real * 14 * n, "flops": MEMBERS * (1000.0 * n + 4 * solve)}
    if case["flow"] == "stratified":
        return {"bytes": MEMBERS * real * 16 * n, "flops": MEMBERS * (step + 900.0 * n)}
    return {"bytes": MEMBERS * real * 14 * n, "flops": MEMBERS * step}


# ---------------------------------------------------------------- the same in 64 bits, without the library
def _projection_velocity(case, seed):
    """A boundary-layer profile with resolved turbulence: what the nodal projection meets."""
    shape = (3, case["nz"], case["ny"], case["nx"])
    v = _smooth_noise(shape, _gen(seed), 0.5)
    z = (torch.arange(case["nz"], device="cuda", dtype=torch.float64) + 0.5) * case["dz"]
    v[0] += (1.5 * torch.log1p(z / 0.1) * 0.41)[:, None, None]
    return v


def _pad(a, lo, hi):
    """One ghost layer: periodic x and y, the given layers in z."""
    a = torch.cat([lo[None], a, hi[None]], 0)
    a = torch.cat([a[:, -1:], a, a[:, :1]], 1)
    return torch.cat([a[:, :, -1:], a, a[:, :, :1]], 2)


def _exact_divtau(case, seed):
    s = prepare(case, seed)
    u, mu, wg = s["vel"], s["mu"], s["wg"]
    h = (20.0, 20.0, 10.0)
    q = []
    for n in range(3):
        lo, hi = u[n, 0], u[n, -1]
        if n == 2:
            lo, hi = -lo, -hi
        elif case["wall"]:
            lo = lo - wg[n] * h[2]
        q.append(_pad(u[n], lo, hi))
    m = _pad(mu, mu[0], mu[-1])
    axis = (2, 1, 0)  # x, y, z of the (z, y, x) arrays
    nx, ny, nz = case["nx"], case["ny"], case["nz"]

    def sh(a, off):
        """The padded array at every face's high-side cell plus off (x, y, z), over the faces of direction d."""
        ext = [nz, ny, nx]
        ext[axis[d]] += 1
        st = [1 + off[2], 1 + off[1], 1 + off[0]]
        return a[st[0]:st[0] + ext[0], st[1]:st[1] + ext[1], st[2]:st[2] + ext[2]]

    out = torch.zeros_like(u)
    for d in range(3):
        e = [0, 0, 0]
        e[d] = -1
        mf = 0.5 * (sh(m, (0, 0, 0)) + sh(m, e))
        gr = [[None] * 3 for _ in range(3)]
        for n in range(3):
            for k in range(3):
                if k == d:
                    gr[k][n] = (sh(q[n], (0, 0, 0)) - sh(q[n], e)) / h[k]
                else:
                    f = [0, 0, 0]
                    f[k] = 1
                    up = sh(q[n], f) + sh(q[n], [a + b for a, b in zip(e, f)])
                    dn = sh(q[n], [-a for a in f]) + sh(q[n], [a - b for a, b in zip(e, f)])
                    gr[k][n] = 0.25 * (up - dn) / h[k]
        dv = gr[0][0] + gr[1][1] + gr[2][2]
        for n in range(3):
            F = mf * (2.0 * gr[d][d] - (2.0 / 3.0) * dv) if n == d else mf * (gr[d][n] + gr[n][d])
            out[n] += torch.diff(F, dim=axis[d]) / h[d]
    return out


def _exact_projection(case, seed):
    """The nodal projection by Fourier transforms in x and y and a direct solve in z."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = (20.0, 20.0, case["dz"])
    sigma = 1.0 / 1.225
    u = _projection_velocity(case, seed)
    wall = case["wall"]
    if wall:  # mirror images: w odd, u and v even
        g = torch.stack([torch.cat([u[n, :1] * s, u[n], u[n, -1:] * s]) for n, s in ((0, 1.0), (1, 1.0), (2, -1.0))])
    else:
        g = torch.cat([u[:, -1:], u], 1)

    def back(a, ax):
        return torch.roll(a, 1, ax)

    def avg(a, ax):
        return 0.5 * (a + back(a, ax))

    def dif(a, ax):
        return a - back(a, ax)

    def zavg(a):
        return 0.5 * (a[1:] + a[:-1])

    rhs = zavg(avg(dif(g[0], 2), 1)) / h[0] + zavg(avg(dif(g[1], 1), 2)) / h[1] + avg(avg(g[2, 1:] - g[2, :-1], 2), 1) / h[2]
    nn = rhs.shape[0]
    tx = 2 * math.pi * torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64) / nx
    ty = 2 * math.pi * torch.arange(ny, device="cuda", dtype=torch.float64) / ny
    kx, ky = (2 - 2 * torch.cos(tx)) / h[0] ** 2, (2 - 2 * torch.cos(ty)) / h[1] ** 2
    mx, my = (2 + torch.cos(tx)) / 3, (2 + torch.cos(ty)) / 3
    s = ky[:, None] * mx[None, :] + my[:, None] * kx[None, :]
    t = my[:, None] * mx[None, :]
    R = torch.fft.rfft2(rhs) / sigma
    if wall:
        off, dia = -(s / 6 - t / h[2] ** 2), -(2 * s / 3 + 2 * t / h[2] ** 2)
        P = torch.empty_like(R)
        c = torch.zeros((nn,) + tuple(s.shape), device="cuda", dtype=torch.float64)
        # elimination from the bottom node; the end rows couple to their neighbour twice (mirror image)
        dia = dia.clone()
        dia[0, 0] = 1.0  # the mean mode is solved below
        c[0], P[0] = 2 * off / dia, R[0] / dia
        for k in range(1, nn):
            a = 2 * off if k == nn - 1 else off
            den = dia - a * c[k - 1]
            den[0, 0] = 1.0
            c[k] = off / den
            P[k] = (R[k] - a * P[k - 1]) / den
        for k in range(nn - 2, -1, -1):
            P[k] -= c[k] * P[k + 1]
        r0 = R[:, 0, 0].real.cpu().numpy()
        A = np.zeros((nn, nn))
        for k in range(nn):
            A[k, k] = -2.0
            A[k, k - 1 if k else 1] += 1.0
            A[k, k + 1 if k + 1 < nn else nn - 2] += 1.0
        w = np.ones(nn)
        w[0] = w[-1] = 0.5
        r0 = r0 - (w @ r0) / w.sum()
        P[:, 0, 0] = torch.from_numpy(np.linalg.lstsq(A / h[2] ** 2, r0, rcond=None)[0]).to(P)
    else:
        tz = 2 * math.pi * torch.arange(nn, device="cuda", dtype=torch.float64) / nn
        lam = -(s[None] * ((2 + torch.cos(tz)) / 3)[:, None, None] + t[None] * ((2 - 2 * torch.cos(tz)) / h[2] ** 2)[:, None, None])
        lam[0, 0, 0] = 1.0
        Z = torch.fft.fft(R, dim=0) / lam
        Z[0, 0, 0] = 0.0
        P = torch.fft.ifft(Z, dim=0)
    p = torch.fft.irfft2(P, s=(ny, nx))
    n = p if wall else torch.cat([p, p[:1]])

    def fwd(a, ax):
        return torch.roll(a, -1, ax)

    gx = zavg(0.5 * ((fwd(n, 2) - n) + fwd(fwd(n, 2) - n, 1))) / h[0]
    gy = zavg(0.5 * ((fwd(n, 1) - n) + fwd(fwd(n, 1) - n, 2))) / h[1]
    dz = n[1:] - n[:-1]
    gz = 0.25 * (dz + fwd(dz, 2) + fwd(dz, 1) + fwd(fwd(dz, 1), 2)) / h[2]
    gp = torch.stack([gx, gy, gz])
    return {"velocity": u - sigma * gp, "gp": gp, "p": (p - p.mean())[None]}


def exact(case, seed):
    if case["kind"] == "divtau":
        return _exact_divtau(case, seed)
    if case["kind"] == "projection":
        return _exact_projection(case, seed)
    return None  # a whole time step has no reference outside the library's own restatement
