"""Performance cases: what a user of this framework has the GPU do in a substep, through the public entry points.

A substep solves the potential, projects the velocity, extrapolates it, enforces the collider, advects the level set
and the velocity and redistances the level set; the learned form adds the network's forward and training passes.
Every array is resident on the GPU (the device entry points), as in the sequence driver and the benchmark.

Inputs are the repository's scenes (a pool with a sphere, box walls on the grid faces, a dipole's applied field)
built on the GPU, with the pool, the sphere and the velocities drawn from the seed.
"""
import importlib
import math
import os

import numpy as np
import torch

sf = importlib.import_module("simferrofluid-cuda_gb300")
scenes = importlib.import_module("simferrofluid-cuda_gb300.scenes")
sequence = importlib.import_module("simferrofluid-cuda_gb300.sequence")

F64 = torch.float64
CHI = 2.0  # the benchmark scene's susceptibility


def listed():
    return [
        # the smallest grid of the benchmark configurations, every option at its default (FP64 form, tolerance 1e-8):
        # about a hundred short launches per iteration
        dict(name="project_fp64_64", kind="project", nx=64, ny=64, nz=64, precision="fp64", tol=1e-8),
        # a domain that is no multiple of the kernels' tiles, defaults (FP64 form, tolerance 1e-6)
        dict(name="potential_fp64_ragged", kind="potential", nx=131, ny=97, nz=117, precision="fp64", tol=1e-6),
        # the benchmark's scene in the form it is tuned for; to 1e-10, where the answer is that of the system rather
        # than that of the iteration at which the solver stops
        dict(name="project_mixed_256", kind="project", nx=256, ny=256, nz=256, precision="mixed", tol=1e-10),
        dict(name="potential_mixed_256", kind="potential", nx=256, ny=256, nz=256, precision="mixed", tol=1e-10),
        # a long sequence's resolution range: every field is ten times the L2 cache
        dict(name="potential_mixed_512", kind="potential", nx=512, ny=512, nz=512, precision="mixed", tol=1e-10),
        # after the projection: six layers of extrapolation, then the collider's boundary condition
        dict(name="velocity_256", kind="velocity", nx=256, ny=256, nz=256),
        # the interface coupling: magnetic pressures at the contour's vertices and the jump on every face
        dict(name="interface_256", kind="interface", nx=256, ny=256, nz=256),
        # advection of the level set (tricubic) and of the velocity by itself (trilinear)
        dict(name="advect_levelset_192", kind="advect_levelset", nx=192, ny=192, nz=192, depth=0.25),
        dict(name="advect_velocity_160", kind="advect_velocity", nx=160, ny=160, nz=160, depth=0.25),
        # redistancing with its default ten steps: the longest part of a substep
        dict(name="reinitialize_128", kind="reinitialize", nx=128, ny=128, nz=128, steps=10),
        # the learned form: one forward at the benchmark's size, one training step at the training size
        dict(name="unet_forward_256", kind="unet_forward", nx=256, ny=256, nz=256),
        dict(name="unet_train_128", kind="unet_train", nx=128, ny=128, nz=128),
    ]


def draw(rng):
    """One more case: sizes spread over the logarithm, half of them ragged boxes with odd sides."""
    kind = rng.choice(["project", "potential", "velocity", "interface", "advect_levelset", "advect_velocity",
                       "reinitialize", "unet_forward", "unet_train"])
    lo, hi = {"project": (32, 288), "potential": (32, 288), "velocity": (32, 256), "interface": (32, 256),
              "advect_levelset": (24, 200), "advect_velocity": (24, 170), "reinitialize": (24, 128),
              "unet_forward": (32, 224), "unet_train": (32, 120)}[kind]

    def side():
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if rng.random() < 0.5:
        n = side()
        n = max(lo, n - n % 8)
        c = dict(kind=kind, nx=n, ny=n, nz=n)
    else:
        n = side()
        c = dict(kind=kind, nx=n, ny=min(hi, max(24, int(n * rng.uniform(0.7, 1.3)))),
                 nz=min(hi, max(24, int(n * rng.uniform(0.7, 1.3)))))
    if kind in ("project", "potential"):
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["tol"] = 1e-10 if c["precision"] == "mixed" else (1e-8 if kind == "project" else 1e-6)
    elif kind in ("advect_levelset", "advect_velocity"):
        c["depth"] = round(rng.uniform(0.1, 0.6), 3)
    elif kind == "reinitialize":
        c["steps"] = rng.choice([3, 5, 10])
    return c


# ------------------------------------------------------------------------------------------------ inputs
_stream = None


def _use_stream():
    """Torch and the library share one stream, as in the benchmark (the default stream cannot be borrowed)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    torch.cuda.set_stream(_stream)
    return _stream.cuda_stream


def _grid(c):
    return sf.StaggeredGrid.from_origin(1.0 / c["nx"], (c["nx"], c["ny"], c["nz"]))


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _centres(g):
    return [torch.from_numpy(scenes.cell_centres(g, a)).cuda() for a in range(3)]


def _pool_sphere(g, rng, depth=None):
    """Distance to a pool united with a sphere (the benchmark's scene, its measures moved a little by the seed)."""
    x, y, z = _centres(g)
    top = float(y[-1])
    depth = (0.2 if depth is None else depth) + rng.uniform(-0.02, 0.02)
    c = [rng.uniform(0.4, 0.6), rng.uniform(0.5, 0.6), rng.uniform(0.4, 0.6)]
    r = rng.uniform(0.12, 0.18)
    s = ((x.view(-1, 1, 1) - c[0]) ** 2 + (y.view(1, -1, 1) - c[1]) ** 2 + (z.view(1, 1, -1) - c[2]) ** 2).sqrt() - r
    return torch.minimum(y.view(1, -1, 1) - depth * min(1.0, top), s).contiguous()


def _dipole(g, pos=(0.5, -0.3, 0.5)):
    """Field of a dipole of moment (0, 1, 0) below the pool, on every face."""
    out = []
    for a in range(3):
        p = [torch.from_numpy(v).cuda() for v in scenes.face_positions(g, a)]
        r = [p[0].view(-1, 1, 1) - pos[0], p[1].view(1, -1, 1) - pos[1], p[2].view(1, 1, -1) - pos[2]]
        r2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2
        h = 3 * r[1] * r[a] / r2 ** 2.5
        if a == 1:
            h = h - 1 / r2 ** 1.5
        out.append(h.contiguous())
    return out


def _moving(g, phi, gen):
    """A smooth velocity as the extrapolation leaves it: |u| <= 0.5 within six cells of the liquid, zero beyond."""
    near = (phi < 6 * g.spacing).to(F64)
    out = []
    for a, u in enumerate(sequence.smooth_velocity(torch, g, torch.device("cuda"), gen)):
        pad = [0, 0, 0, 0, 0, 0]
        pad[2 * (2 - a)] = pad[2 * (2 - a) + 1] = 1
        m = torch.nn.functional.pad(near[None, None], pad, mode="replicate")[0, 0]
        out.append((u * torch.maximum(m.narrow(a, 0, u.shape[a]), m.narrow(a, 1, u.shape[a]))).contiguous())
    return out


def _rippled(g, phi, gen):
    """The distance after an advection: stretched by up to a tenth and rippled by a fiftieth of the domain."""
    lat = torch.rand((1, 2, 9, 9, 9), generator=gen, device="cuda", dtype=F64) * 2 - 1
    s = torch.nn.functional.interpolate(lat, size=g.shape, mode="trilinear", align_corners=True)[0]
    return (phi * (1 + 0.1 * s[0]) + 0.02 * s[1]).contiguous()


def _contour(g, phi):
    """The contour's vertices, one on each cell-grid edge that the interface cuts: edge marks and positions, in a
    mesh buffer of a capacity that depends on the grid alone (its rest repeats the vertices)."""
    inside = phi <= 0
    marks, pos, count = [], [], 0
    o = torch.tensor([v + 0.5 * g.spacing for v in g.origin], dtype=F64, device="cuda")
    for a in range(3):
        n = phi.shape[a] - 1
        p0, p1 = phi.narrow(a, 0, n), phi.narrow(a, 1, n)
        at = (inside.narrow(a, 0, n) != inside.narrow(a, 1, n)).nonzero()
        m = torch.full(p0.shape, -1, dtype=torch.int32, device="cuda")
        m[at[:, 0], at[:, 1], at[:, 2]] = torch.arange(count, count + len(at), dtype=torch.int32, device="cuda")
        f0, f1 = p0[at[:, 0], at[:, 1], at[:, 2]], p1[at[:, 0], at[:, 1], at[:, 2]]
        q = at.to(F64)
        q[:, a] += f0 / (f0 - f1)
        marks.append(m)
        pos.append(o + q * g.spacing)
        count += len(at)
    pos = torch.cat(pos)
    room = 2 * g.shape[0] * g.shape[2] + g.shape[0] ** 2
    return marks, pos[torch.arange(room, device="cuda") % count].contiguous()


def _weights(seed):
    """The trained network's weights moved by a hundredth of their size (another user's training run)."""
    w = np.fromfile(os.path.join(os.path.dirname(sf.__file__), "weights", "unet.f32"), dtype=np.float32)
    return (w * (1 + 0.01 * np.random.default_rng(seed).standard_normal(w.size))).astype(np.float32)


def _features(g, phi, gen):
    """Network features of a pressure-like system: rhs, active mask, lower couplings over D, excess over D."""
    n = g.num_cells
    act = (phi <= 0).to(F64).reshape(-1)
    f = torch.zeros((n, 16), dtype=F64, device="cuda")
    f[:, 0] = torch.randn(n, generator=gen, device="cuda", dtype=F64) * act
    f[:, 1] = act
    for a in range(3):
        f[:, 2 + a] = act / 6
    f[:, 5] = act * torch.rand(n, generator=gen, device="cuda", dtype=F64) * 0.1
    return f.to(torch.bfloat16)


def _inputs(case, seed):
    g, gen, rng = _grid(case), _gen(seed), np.random.default_rng(int(seed))
    phi = _pool_sphere(g, rng, case.get("depth"))
    kind, s = case["kind"], dict(g=g, phi=phi)
    if kind == "project":
        s["vel"] = [torch.randn(g.face_shape(a), generator=gen, device="cuda", dtype=F64) * 0.5 for a in range(3)]
        s["frac"] = sequence.box_fractions_device(sf, scenes, torch, g, torch.device("cuda"))
    elif kind == "potential":
        s["hext"] = _dipole(g, (0.5 + 0.1 * rng.uniform(-1, 1), -0.3, 0.5))
    elif kind == "velocity":
        s["vel"] = sequence.smooth_velocity(torch, g, torch.device("cuda"), gen)
        s["frac"] = sequence.box_fractions_device(sf, scenes, torch, g, torch.device("cuda"))
        s["normal"] = sequence.box_normals_device(sf, scenes, torch, g, torch.device("cuda"))
    elif kind == "interface":
        s["H"] = _dipole(g, (0.5 + 0.1 * rng.uniform(-1, 1), -0.3, 0.5))
        s["marks"], s["pos"] = _contour(g, phi)
        nrm = torch.randn(s["pos"].shape, generator=gen, device="cuda", dtype=F64)
        s["nrm"] = nrm / nrm.norm(dim=1, keepdim=True)
        s["kappa"] = torch.randn(len(nrm), generator=gen, device="cuda", dtype=F64) * 8
    elif kind in ("advect_levelset", "advect_velocity"):
        s["vel"] = _moving(g, phi, gen)
    elif kind == "reinitialize":
        s["phi"] = _rippled(g, phi, gen)
    elif kind == "unet_forward":
        s["feat"] = _features(g, phi, gen)
    elif kind == "unet_train":
        s["feat"] = _features(g, phi, gen)
        s["target"] = (phi.reshape(-1) * s["feat"][:, 1].to(F64)).float()
    return s


SIGMA, DENSITY, DT = 0.072, 1.0, 0.004  # surface tension, density and time step of the jump
LR = 1e-3  # the trainer's learning rate


def prepare(case, seed):
    handle = _use_stream()
    s = _inputs(case, seed)
    g, kind = s["g"], case["kind"]
    s["kind"] = kind
    s["ctx"] = ctx = sf.Context(0, stream=handle)
    zeros = lambda shape: torch.zeros(shape, dtype=F64, device="cuda")  # noqa: E731
    if kind == "project":
        s["op"] = sf.Pressure(g, ctx)
        s["opts"] = sf.options("pressure", precision=case["precision"], tol=case["tol"])
        s["u"], s["p"] = [torch.empty_like(v) for v in s["vel"]], zeros(g.shape)
    elif kind == "potential":
        s["op"] = sf.MagneticField(g, CHI, 2 * g.spacing, ctx)
        # from zero: a repeated solve that starts from its own answer would take no iteration
        s["opts"] = sf.options("magnetic", precision=case["precision"], tol=case["tol"], warm_start=0)
        s["psi"], s["H"] = zeros(g.shape), [zeros(g.face_shape(a)) for a in range(3)]
    elif kind == "velocity":
        s["ext"], s["enf"] = sf.Extrapolation(g, ctx), sf.ColliderEnforce(g, s["frac"], s["normal"], ctx=ctx)
        s["u"] = [torch.empty_like(v) for v in s["vel"]]
    elif kind == "interface":
        s["op"] = sf.MagneticField(g, CHI, 2 * g.spacing, ctx)
        s["pm"], s["jump"] = zeros(len(s["pos"])), [zeros(g.face_shape(a)) for a in range(3)]
    elif kind == "advect_levelset":
        s["op"], s["out"] = sf.Advection(g, ctx), torch.empty_like(s["phi"])
    elif kind == "advect_velocity":
        s["op"], s["u"] = sf.Advection(g, ctx), [torch.empty_like(v) for v in s["vel"]]
    elif kind == "reinitialize":
        s["op"], s["out"], s["steps"] = sf.Reinitialization(g, ctx), torch.empty_like(s["phi"]), case["steps"]
    else:
        s["net"] = sf.Network(ctx)
        s["net"].set_params(_weights(seed))
        s["out"] = torch.zeros(g.num_cells, dtype=torch.float32, device="cuda")
    return s


def run(s):
    """One pass; arrays that a call updates in place start from a fresh copy of the inputs, as in a substep."""
    kind = s["kind"]
    if kind == "project":
        for u, v in zip(s["u"], s["vel"]):
            u.copy_(v)
        s["op"].project(s["u"], s["phi"], s["frac"], opts=s["opts"], device=True, p_out=s["p"])
        return {"u": s["u"], "p": s["p"]}
    if kind == "potential":
        s["op"].solve(s["phi"], s["hext"], opts=s["opts"], device=True, psi_out=s["psi"], H_out=s["H"])
        return {"psi": s["psi"], "H": s["H"]}
    if kind == "velocity":
        for u, v in zip(s["u"], s["vel"]):
            u.copy_(v)
        s["ext"].solve(s["u"], s["phi"], s["frac"], device=True)
        s["enf"].enforce(s["u"], device=True)
        return {"u": s["u"]}
    if kind == "interface":
        s["op"].calculate_vertex_pressures(s["pos"], s["nrm"], H=s["H"], device=True, out=s["pm"])
        sf.pressure_jump(s["g"], s["marks"], s["kappa"], s["pm"], SIGMA, DENSITY, DT, ctx=s["ctx"], device=True,
                         out=s["jump"])
        return {"pm": s["pm"], "jump": s["jump"]}
    if kind == "advect_levelset":
        s["out"].copy_(s["phi"])
        s["op"].solve_levelset(s["out"], s["vel"], s["g"].spacing, device=True)
        return {"phi": s["out"]}
    if kind == "advect_velocity":
        for u, v in zip(s["u"], s["vel"]):
            u.copy_(v)
        s["op"].solve_velocity(s["u"], s["g"].spacing, device=True)
        return {"u": s["u"]}
    if kind == "reinitialize":
        s["out"].copy_(s["phi"])
        s["op"].solve(s["out"], s["steps"], device=True)
        return {"phi": s["out"]}
    if kind == "unet_forward":
        return {"out": s["net"].forward(s["g"], s["feat"], s["out"])}
    loss = s["net"].train_step(s["g"], s["feat"], s["target"], LR)
    return {"loss": loss, "params": s["net"].get_params()}


def work(case):
    """Each input read once, each output written once; arithmetic that the method cannot do without, per cell."""
    n = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    edges = 4 * 3 * n
    per_cell = {
        # arrays of doubles in and out; operations
        "project": (8 * (1 + 3 + 3 + 3 + 1), 60),          # phi, u, fractions -> u, p; assembly and update alone
        "potential": (8 * (1 + 3 + 1 + 3), 60),             # phi, Hext -> psi, H
        "velocity": (8 * (3 + 1 + 3 + 3), 6),               # u, phi, fractions -> u (normals at the walls only)
        "interface": (8 * 3, 3),                            # jump out (the edge marks below)
        "advect_levelset": (8 * (1 + 3 + 1), 450),          # six trilinear samples, 64 points
        "advect_velocity": (8 * (3 + 3), 3 * 250),
        "reinitialize": (16, 500 * 3 * case.get("steps", 10)),
        "unet_forward": (2 * 16 + 4, 87048),
        "unet_train": (2 * 16 + 4, 3 * 87048),
    }[kind]
    return {"bytes": float(per_cell[0] * n + (edges if kind == "interface" else 0)), "flops": float(per_cell[1] * n)}


# ------------------------------------------------------------------------------------------------ 64-bit answers
def _sl(a, lo, hi):
    return tuple(slice(lo, hi) if b == a else slice(None) for b in range(3))


def _pcg(low, diag, b, tol=1e-14, most=6000):
    """Jacobi-preconditioned CG on the 7-point operator with lower-face couplings low[a]."""
    inv = torch.where(diag > 0, 1 / diag.clamp_min(1e-300), torch.zeros_like(diag))

    def mul(v):
        y = diag * v
        for a in range(3):
            w = low[a][_sl(a, 1, None)]
            y[_sl(a, 1, None)] -= w * v[_sl(a, None, -1)]
            y[_sl(a, None, -1)] -= w * v[_sl(a, 1, None)]
        return y

    x, r = torch.zeros_like(b), b.clone()
    z = inv * r
    p, rz, bn = z.clone(), (r * z).sum(), b.norm()
    for it in range(most):
        q = mul(p)
        alpha = rz / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        if it % 20 == 19 and not r.norm() > tol * bn:
            break
        z = inv * r
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_project(s):
    phi, g = s["phi"], s["g"]
    liq = phi <= 0
    w = [1 - f for f in s["frac"]]
    diag, b = torch.zeros_like(phi), torch.zeros_like(phi)
    low = [torch.zeros_like(phi) for _ in range(3)]
    for a in range(3):
        n = phi.shape[a]
        wi, ui = w[a][_sl(a, 1, n)], s["vel"][a][_sl(a, 1, n)]
        lo, hi = _sl(a, 0, n - 1), _sl(a, 1, n)
        both = liq[lo] & liq[hi]
        low[a][hi] = torch.where(both, wi, torch.zeros_like(wi))
        for me, nb, side in ((hi, lo, -1.0), (lo, hi, 1.0)):
            theta = (phi[me] / (phi[me] - phi[nb])).clamp_min(1e-3)
            diag[me] += torch.where(liq[me], torch.where(liq[nb], wi, wi / theta), torch.zeros_like(wi))
            b[me] -= torch.where(liq[me], side * wi * ui, torch.zeros_like(wi))
    diag = torch.where(liq & (diag == 0), torch.ones_like(diag), diag)
    p = _pcg(low, diag, b)
    out = []
    for a in range(3):
        n = phi.shape[a]
        lo, hi = _sl(a, 0, n - 1), _sl(a, 1, n)
        u = s["vel"][a].clone()
        wi = w[a][_sl(a, 1, n)]
        t_lo = (phi[lo] / (phi[lo] - phi[hi])).clamp_min(1e-3)
        t_hi = (1 - phi[lo] / (phi[lo] - phi[hi])).clamp_min(1e-3)
        du = torch.where(liq[lo] & liq[hi], (p[hi] - p[lo]) * wi,
                         torch.where(liq[lo], -p[lo] / t_lo * wi, torch.where(liq[hi], p[hi] / t_hi * wi, 0 * wi)))
        u[_sl(a, 1, n)] -= du
        out.append(u)
    return {"u": out, "p": torch.where(liq, p, torch.zeros_like(p))}


def _exact_potential(s):
    phi, g, h = s["phi"], s["g"], s["g"].spacing
    bw = 2 * h
    diag, b = torch.zeros_like(phi), torch.zeros_like(phi)
    low = [torch.zeros_like(phi) for _ in range(3)]
    for a in range(3):
        n = phi.shape[a]
        lo, hi = _sl(a, 0, n - 1), _sl(a, 1, n)
        f = 0.5 * (phi[lo] + phi[hi])
        t = (f / bw).clamp(-1, 1)
        mu = 1 + (1 - 0.5 * (1 + t + torch.sin(math.pi * t) / math.pi)) * CHI
        low[a][hi] = mu
        diag[lo] += mu
        diag[hi] += mu
        flux = (mu - 1) * s["hext"][a][_sl(a, 1, n)] * h
        b[hi] += flux
        b[lo] -= flux
    psi = _pcg(low, diag, b)
    psi = psi - psi[0, 0, 0]
    H = []
    for a in range(3):
        n = phi.shape[a]
        v = s["hext"][a].clone()
        v[_sl(a, 1, n)] -= (psi[_sl(a, 1, n)] - psi[_sl(a, 0, n - 1)]) / h
        H.append(v)
    return {"psi": psi, "H": H}


def _coords(p, origin, h, off):
    t = (p - origin) / h
    lo = torch.floor(t - off)
    return lo.long(), t - lo


def _trilinear(g, f, b, p):
    lo, w = [], []
    for a in range(3):
        o = g.origin[a] + (0 if a == b else 0.5 * g.spacing)
        i, fr = _coords(p[a], o, g.spacing, 0.0)
        lo.append(i)
        w.append((1 - fr, fr))
    val = 0
    for q in range(8):
        d = [(q >> a) & 1 for a in range(3)]
        i = [(lo[a] + d[a]).clamp(0, f.shape[a] - 1) for a in range(3)]
        val = val + f[i[0], i[1], i[2]] * w[0][d[0]] * w[1][d[1]] * w[2][d[2]]
    return val


def _tricubic(g, f, p):
    lo, w = [], []
    for a in range(3):
        i, r = _coords(p[a], g.origin[a] + 0.5 * g.spacing, g.spacing, 1.0)
        lo.append(i)
        w.append(((r - 1) * (r - 2) * (r - 3) / -6, r * (r - 2) * (r - 3) / 2, r * (r - 1) * (r - 3) / -2,
                  r * (r - 1) * (r - 2) / 6))
    val = 0
    for k in range(4):
        for j in range(4):
            for i in range(4):
                q = [(lo[a] + v).clamp(0, f.shape[a] - 1) for a, v in enumerate((i, j, k))]
                val = val + f[q[0], q[1], q[2]] * (w[0][i] * w[1][j] * w[2][k])
    return val


def _trace(g, u, p, dt):
    v0 = [_trilinear(g, u[b], b, p) for b in range(3)]
    v1 = [_trilinear(g, u[b], b, [p[a] + v0[a] * dt for a in range(3)]) for b in range(3)]
    return [p[a] + 0.5 * dt * (v0[a] + v1[a]) for a in range(3)]


def _points(g, face=None):
    q = scenes.face_positions(g, face) if face is not None else [scenes.cell_centres(g, a) for a in range(3)]
    return list(torch.meshgrid(*[torch.from_numpy(v).cuda() for v in q], indexing="ij"))


def _weno(d):
    """WENO5 derivative from five one-sided differences, nearest the upwind side first."""
    eps = torch.stack([v * v for v in d]).amax(0) * 1e-6 + 1e-99
    p = (d[0] / 3 - d[1] * 7 / 6 + d[2] * 11 / 6, -d[1] / 6 + d[2] * 5 / 6 + d[3] / 3,
         d[2] / 3 + d[3] * 5 / 6 - d[4] / 6)
    s = ((d[0] - 2 * d[1] + d[2]) ** 2 * 13 / 12 + (d[0] - 4 * d[1] + 3 * d[2]) ** 2 / 4,
         (d[1] - 2 * d[2] + d[3]) ** 2 * 13 / 12 + (d[1] - d[3]) ** 2 / 4,
         (d[2] - 2 * d[3] + d[4]) ** 2 * 13 / 12 + (3 * d[2] - 4 * d[3] + d[4]) ** 2 / 4)
    al = [c / (v + eps) ** 2 for c, v in zip((0.1, 0.6, 0.3), s)]
    return (al[0] * p[0] + al[1] * p[1] + al[2] * p[2]) / (al[0] + al[1] + al[2])


def _advance(g, f):
    tot = torch.zeros_like(f)
    for a in range(3):
        n = f.shape[a]
        v = [f.index_select(a, (torch.arange(n, device="cuda") + q).clamp(0, n - 1)) for q in range(-3, 4)]
        dm = _weno([v[i + 1] - v[i] for i in range(5)]) / g.spacing
        dp = _weno([v[6 - i] - v[5 - i] for i in range(5)]) / g.spacing
        neg = f < 0
        tot += torch.where(neg, dm.clamp_max(0) ** 2 + dp.clamp_min(0) ** 2, dm.clamp_min(0) ** 2 + dp.clamp_max(0) ** 2)
    m = tot.sqrt()
    return f + 0.5 * g.spacing * f / (f * f + (g.spacing * m) ** 2).sqrt() * (1 - m)


def _exact_velocity(s):
    g, phi = s["g"], s["phi"]
    liq = phi <= 0
    us = []
    for a in range(3):
        u, n = s["vel"][a].clone(), phi.shape[a]
        valid = torch.zeros(u.shape, dtype=torch.bool, device="cuda")
        valid[_sl(a, 0, n)] |= liq
        valid[_sl(a, 1, n + 1)] |= liq
        valid &= s["frac"][a] < 1
        for _ in range(6):
            tot, cnt = torch.zeros_like(u), torch.zeros_like(u)
            for b in range(3):
                m = u.shape[b]
                lo, hi = _sl(b, 0, m - 1), _sl(b, 1, m)
                vu = torch.where(valid, u, torch.zeros_like(u))
                tot[hi] += vu[lo]
                cnt[hi] += valid[lo].to(F64)
                tot[lo] += vu[hi]
                cnt[lo] += valid[hi].to(F64)
            u = torch.where(valid, u, torch.where(cnt > 0, tot / cnt.clamp_min(1), torch.zeros_like(u)))
            valid = valid | (cnt > 0)
        us.append(u)
    out = []
    for a in range(3):
        at = s["frac"][a] == 1
        idx = at.nonzero()
        o = [g.origin[b] + (0 if b == a else 0.5 * g.spacing) for b in range(3)]
        p = [o[b] + idx[:, b].to(F64) * g.spacing for b in range(3)]
        v = [_trilinear(g, us[b], b, p) for b in range(3)]
        nrm = [_trilinear(g, s["normal"][b], b, p) for b in range(3)]
        ln = (nrm[0] ** 2 + nrm[1] ** 2 + nrm[2] ** 2).sqrt()
        nrm = [torch.where(ln > 0, q / ln.clamp_min(1e-300), q) for q in nrm]
        dn = v[0] * nrm[0] + v[1] * nrm[1] + v[2] * nrm[2]
        u = us[a].clone()
        u[at] = v[a] - dn * nrm[a]
        out.append(u)
    return {"u": out}


def _exact_interface(s):
    g = s["g"]
    p = [s["pos"][:, a] for a in range(3)]
    H = torch.stack([_trilinear(g, s["H"][b], b, p) for b in range(3)], 1)
    hn = (H * s["nrm"]).sum(1)
    pm = 4e-7 * math.pi / 2 * CHI * ((H * H).sum(1) + CHI ** 2 / (4 * CHI + 4) * hn * hn)
    per = (s["kappa"] * SIGMA - pm) / DENSITY / g.spacing * DT
    jump = []
    for a in range(3):
        j = torch.zeros(g.face_shape(a), dtype=F64, device="cuda")
        m = s["marks"][a].long()
        j[_sl(a, 1, g.shape[a])] = torch.where(m >= 0, per[m.clamp_min(0)], torch.zeros((), dtype=F64, device="cuda"))
        jump.append(j)
    return {"pm": pm, "jump": jump}


LAYERS = ((16, 16, 27), (16, 16, 27), (16, 32, 27), (32, 32, 27), (32, 64, 27), (64, 64, 27), (64, 64, 27),
          (64, 64, 27), (64, 64, 27), (64, 32, 27), (32, 32, 27), (32, 16, 27), (16, 16, 27), (16, 16, 27), (16, 1, 1))


def _net64(x, w):
    """The network in 64 bits (no rounding of weights or activations); x (1, 16, X, Y, Z), w the flat weights."""
    F = torch.nn.functional
    at, ws = 0, []
    for ci, co, taps in LAYERS:
        k = w[at:at + taps * co * ci].reshape(taps, co, ci)
        at += taps * co * ci
        side = 3 if taps == 27 else 1
        ws.append((k.permute(1, 2, 0).reshape(co, ci, side, side, side), w[at:at + co]))
        at += co
    layer = iter(ws)

    def conv(v):
        k, b = next(layer)
        return F.relu(F.conv3d(v, k, b, padding=1))

    def pool(v):
        odd = [q for d in (4, 3, 2) for q in (0, v.shape[d] % 2)]
        return F.avg_pool3d(F.pad(v, odd), 2)

    def up(v, like):
        for d in (2, 3, 4):
            v = v.repeat_interleave(2, d).narrow(d, 0, like.shape[d])
        return v + like

    s0 = conv(conv(x))
    s1 = conv(conv(pool(s0)))
    s2 = conv(conv(pool(s1)))
    v = conv(conv(pool(s2)))
    for s in (s2, s1, s0):
        v = conv(conv(up(v, s)))
    k, b = next(layer)
    return F.conv3d(v, k, b)[0, 0].reshape(-1)


def exact(case, seed):
    """The same pass in 64-bit torch, without the library; None where that takes too long."""
    cells, kind = case["nx"] * case["ny"] * case["nz"], case["kind"]
    if (kind in ("project", "potential") and cells > 300 ** 3) or (kind.startswith("unet") and cells > 96 ** 3):
        return None
    _use_stream()
    s = _inputs(case, seed)
    g = s["g"]
    if kind == "project":
        return _exact_project(s)
    if kind == "potential":
        return _exact_potential(s)
    if kind == "velocity":
        return _exact_velocity(s)
    if kind == "interface":
        return _exact_interface(s)
    if kind == "advect_levelset":
        return {"phi": _tricubic(g, s["phi"], _trace(g, s["vel"], _points(g), -g.spacing))}
    if kind == "advect_velocity":
        return {"u": [_trilinear(g, s["vel"][a], a, _trace(g, s["vel"], _points(g, a), -g.spacing)) for a in range(3)]}
    if kind == "reinitialize":
        f = s["phi"].clone()
        for _ in range(case["steps"]):
            a = _advance(g, _advance(g, f))
            a = (3 * f + a) / 4
            f = (f + 2 * _advance(g, a)) / 3
        return {"phi": f}
    x = s["feat"].to(F64).T.reshape(1, 16, *g.shape)
    w = torch.from_numpy(_weights(seed)).cuda().to(F64)
    if kind == "unet_forward":
        return {"out": _net64(x, w)}
    w.requires_grad_(True)
    out, t = _net64(x, w), s["target"].to(F64)
    loss = 1 - (out @ t) ** 2 / ((out @ out) * (t @ t))
    loss.backward()
    # Adam's first step: the moments' bias corrections leave the gradient over its own size
    return {"loss": loss.detach(), "params": (w - LR * w.grad / (w.grad.abs() + 1e-8)).detach()}
