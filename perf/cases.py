"""Workloads of the library as its users run them: what perf measurements time.

Every case goes through the public Python mirror of the C ABI (``GpuSolver``, ``Ensemble``,
``Cnn``), on seeded synthetic problems of the package's own generator: the homogeneous
infiltration box with a ponded top, and heterogeneous blocks (lognormal conductivity with
exponential correlation, random van Genuchten soils, a water table in the lower part, rain on
top).  A time-stepping case starts every pass from the same saved state, so all passes of one
state do the same work.
"""
import dataclasses
import math
import os

import numpy as np
import torch

from msg123_b200.config import make_config
from msg123_b200.ensemble import Ensemble
from msg123_b200.learned import Cnn, unpack
from msg123_b200.solver import GpuSolver

_WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "msg123_b200", "weights", "guess_cnn.npy")

# The value path of the benchmark: mixed-precision V-cycle, hierarchy kept for `lag` steps,
# two-pow kr, the line-search slope from the linear solve.
_VALUE = dict(precision=1, vg_form=1, jv_mode=1)


def listed():
    return [
        # the infiltration box at its own size: 20 000 cells, FP64, DILU, ponded top and free
        # drainage -- the smallest problem, where launches and host round trips are the time
        dict(name="box_ponded", kind="box", nx=20, ny=20, nz=50, steps=4),
        # the reference's default preconditioner (DILU) on a heterogeneous block too large for
        # one thread block
        dict(name="dilu_block", kind="block", nx=96, ny=81, nz=40, sigma=1.0, steps=1, warm=2, precon=0, lag=0, mixed=0,
             guess=0),
        # the drop-in call of a Fortran host: heads in, one Newton solve of the reference's
        # method (FP64, AMG rebuilt at every Newton iteration), state and mass balance out
        dict(name="host_newton", kind="host", nx=97, ny=75, nz=37, sigma=1.0),
        # the finer drop-in: residual, Jacobian in the reference's CSR order and linear solve as
        # separate calls on host arrays
        dict(name="host_linear", kind="linear", nx=64, ny=57, nz=33, sigma=1.0),
        # a step of the reference's method on the 4.2M-cell block
        dict(name="reference_block", kind="block", nx=256, ny=256, nz=64, sigma=1.0, steps=1, warm=2, precon=1, lag=0,
             mixed=0, guess=0),
        # one realisation of an ensemble by itself, ragged, with the ensemble's settings
        dict(name="member", kind="block", nx=113, ny=87, nz=37, sigma=0.9, steps=4, warm=3, precon=1, lag=4, mixed=1,
             guess=1),
        # eight uneven realisations advanced together over worker threads
        dict(name="ensemble", kind="ensemble", members=8, first=0, steps=4),
        # the 4.2M-cell block with everything but the network, one rebuild in twelve steps
        dict(name="value_block", kind="block", nx=256, ny=256, nz=64, sigma=1.0, steps=12, warm=4, precon=1, lag=12,
             mixed=1, guess=1),
        # the benchmark's block of 25.2M cells on its value path, learned guess included
        dict(name="value_large", kind="block", nx=512, ny=512, nz=96, sigma=1.5, steps=12, warm=4, precon=1, lag=12,
             mixed=1, guess=2),
        # an output time: per-cell mass volumes, velocities, water table
        dict(name="outputs", kind="outputs", nx=200, ny=150, nz=50, sigma=1.0),
        # the network by itself: one forward pass on a ragged grid ...
        dict(name="guess_forward", kind="forward", nx=251, ny=237, nz=61),
        # ... and loss and gradient on a field of its training set
        dict(name="guess_gradient", kind="gradient", nx=128, ny=128, nz=96),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, then sizes over the range that its listed cases stand for."""
    kind = rng.choice(["box", "dilu", "host", "linear", "reference", "member", "ensemble", "value", "outputs", "forward",
                       "gradient"])

    def box(xy, z):
        return dict(nx=_log_int(rng, *xy), ny=_log_int(rng, *xy), nz=_log_int(rng, *z))

    sigma = round(rng.uniform(0.5, 1.5), 3)
    if kind == "box":
        return dict(kind="box", **box((8, 48), (20, 80)), steps=rng.randint(1, 6))
    if kind == "dilu":
        return dict(kind="block", **box((32, 128), (16, 48)), sigma=sigma, steps=1, warm=2, precon=0, lag=0, mixed=0,
                    guess=0)
    if kind == "host":
        return dict(kind="host", **box((24, 160), (16, 48)), sigma=sigma)
    if kind == "linear":
        return dict(kind="linear", **box((24, 160), (16, 48)), sigma=sigma)
    if kind == "reference":
        return dict(kind="block", **box((64, 256), (24, 64)), sigma=sigma, steps=1, warm=2, precon=1, lag=0, mixed=0,
                    guess=0)
    if kind == "member":
        return dict(kind="block", **box((64, 160), (32, 48)), sigma=sigma, steps=4, warm=3, precon=1, lag=4, mixed=1,
                    guess=1)
    if kind == "ensemble":
        return dict(kind="ensemble", members=rng.randint(3, 8), first=rng.randint(1, 60), steps=4)
    if kind == "value":
        lag = rng.choice([4, 8, 12])
        return dict(kind="block", **box((96, 360), (32, 96)), sigma=sigma, steps=lag, warm=4, precon=1, lag=lag, mixed=1,
                    guess=rng.choice([1, 2]))
    if kind == "outputs":
        return dict(kind="outputs", **box((32, 256), (16, 64)), sigma=sigma)
    return dict(kind=kind, **box((24, 256), (16, 96)))


# ---- inputs ---------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _block(case, seed):
    """The generator's heterogeneous block with its random fields drawn on the GPU: a one-column
    problem gives the geometry, rain and parameters, the fields replace its soils."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    S, N = nx * ny, nx * ny * nz
    col = make_config("hetero", shape=(1, 1, nz), seed=1)
    ls = col.params["len_scal"]
    g = _generator(seed)

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand(N, generator=g, device="cuda", dtype=torch.float64)

    k2 = 0
    for n, corr, axis, freq in ((nz, 4, 0, torch.fft.fftfreq), (ny, 20, 1, torch.fft.fftfreq), (nx, 20, 2, torch.fft.rfftfreq)):
        k = freq(n, device="cuda", dtype=torch.float64) * (2 * math.pi * corr)
        k2 = k2 + (k * k).reshape([-1 if a == axis else 1 for a in range(3)])
    noise = torch.randn((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.irfftn(torch.fft.rfftn(noise) / (1.0 + k2), s=(nz, ny, nx)).reshape(-1)
    lnk = math.log(1.0e-5) + case["sigma"] * (f - f.mean()) / f.std()

    def host(t):
        return t.to(torch.float32).cpu().numpy()

    lsf = np.float32(ls)
    ks = host(torch.exp(lnk)) * (np.float32(1.0) / lsf)
    per_cell = {k: np.repeat(getattr(col, k), S) for k in ("cell_top", "cell_vol", "head0", "resi", "ss")}
    per_face = {k: np.repeat(getattr(col, k).reshape(6, nz), S, axis=1).reshape(-1) for k in ("dis2face", "face_area")}
    per_col = {k: np.repeat(getattr(col, k)[:1], S) for k in ("area_r", "surf_top", "surf_bott", "surf_reli", "surf_parm",
                                                             "sea_head", "rech")}
    return dataclasses.replace(col, nx=nx, ny=ny, nz=nz, reta=host(uniform(1.0, 5.0)) * lsf, retn=host(uniform(1.3, 2.5)),
                               poro=host(uniform(0.35, 0.45)), ksx=ks, ksy=ks, ksz=ks, lnk=host(lnk), phys=None,
                               **per_cell, **per_face, **per_col)


def _heads(p, seed, span):
    """Heads around the water table: within +-span (nondimensional) of the hydrostatic start."""
    u = torch.rand(p.ncalc, generator=_generator(seed + 7919), device="cuda", dtype=torch.float64).cpu().numpy()
    return p.head0 + span * (2.0 * u - 1.0)


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _drop_geometry(p):
    p.dis2face = p.face_area = None   # only needed while a context is made


def prepare(case, seed):
    kind = case["kind"]
    if kind == "box":
        p = make_config("box", shape=(case["nx"], case["ny"], case["nz"]))
        u = np.random.default_rng(seed).random(p.ncalc)
        head = p.cell_top + (p.head0 - p.cell_top) * (0.9 + 0.1 * u)     # initial suction within 10 %
        return dict(case=case, g=GpuSolver(p), head=head)
    if kind == "ensemble":
        e = Ensemble(seeds=[case["first"] + k for k in range(case["members"])])
        up = np.random.default_rng(seed).uniform(-0.5, 0.5, len(e.members))      # water tables, m
        heads = [g.prob.head0 + u / g.params["len_scal"] for g, u in zip(e.members, up)]
        return dict(case=case, e=e, heads=heads, out=[dict(head_new=_pinned(g.n)) for g in e.members])
    if kind in ("forward", "gradient"):
        n = case["nx"] * case["ny"] * case["nz"]
        x = torch.zeros((n, 16), device="cuda")
        x[:, :7] = 0.7 * torch.randn((n, 7), generator=_generator(seed), device="cuda")
        y = 0.3 * torch.randn(n, generator=_generator(seed + 1), device="cuda")
        net = Cnn(seed=0)
        w = _network_weights(seed)
        net.set_weights(w)
        net.add_sample((case["nx"], case["ny"], case["nz"]), x.cpu().numpy(), y.cpu().numpy())
        return dict(case=case, net=net, n=n)
    p = _block(case, seed)
    if kind == "block":
        kw = dict(precon_type=case["precon"], amg_lag=case["lag"], guess_mode=case["guess"], guess_select=0)
        if case["mixed"]:
            kw.update(_VALUE)
        net = None
        if case["guess"] == 2:
            net = Cnn(seed=0)
            net.set_weights(np.load(_WEIGHTS))
        g, saved = GpuSolver(p, **kw), GpuSolver(p, **kw)
        _drop_geometry(p)
        if net is not None:
            net.attach(g)
            net.attach(saved)
        saved.init_state()
        saved.advance(nsteps=case["warm"])
        out = dict(head_new=_pinned(p.ncalc), srat_new=_pinned(p.ncalc))
        return dict(case=case, g=g, saved=saved, net=net, out=out)
    g = GpuSolver(p)
    _drop_geometry(p)
    if kind == "outputs":
        head = _heads(p, seed, 0.02)
        g.init_state(_heads(p, seed + 1, 0.02))
        g.set_state(head_new=head, delt=600.0)
        return dict(case=case, g=g)
    g.init_state()
    if kind == "linear":
        return dict(case=case, g=g, head=_heads(p, seed, 1.0e-3))
    g.advance(nsteps=2)
    s = g.get_state()
    return dict(case=case, g=g, state=s, delt=600.0)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "box":
        g = state["g"]
        g.init_state(state["head"])
        _, stats = g.advance(nsteps=case["steps"])
        s = g.get_state()
        return [s["head_new"], s["srat_new"], stats["current_t"]]
    if kind == "block":
        g = state["g"]
        g.copy_state_from(state["saved"])
        _, stats = g.advance(nsteps=case["steps"])
        s = g.get_state(state["out"])
        return [s["head_new"], s["srat_new"], stats["current_t"], stats["delt"]]
    if kind == "ensemble":
        e = state["e"]
        for g, h in zip(e.members, state["heads"]):
            g.init_state(h)
        _, stats = e.advance(case["steps"])
        heads = [g.get_state(out)["head_new"] for g, out in zip(e.members, state["out"])]
        return [heads, [s["current_t"] for s in stats]]
    if kind == "host":
        g, s = state["g"], state["state"]
        g.set_state(head_new=s["head_new"], head_old=s["head_new"], srat_old=s["srat_new"], surf_head=s["surf_head"],
                    delt=state["delt"])
        g.calc_numsol()
        r = g.get_state()
        return [r["head_new"], r["srat_new"], g.calc_mass()]
    if kind == "linear":
        g = state["g"]
        f = g.calc_func(state["head"])
        g.set_state(head_new=state["head"])
        d, lu, rhs = g.make_matvec()
        x, _, _, _ = g.solve_linalg(float(np.dot(rhs, rhs)), 1.0e-3)
        return [f, d, lu, rhs, x]
    if kind == "outputs":
        g = state["g"]
        m = g.cell_mass()
        fv, pv = g.velocity()
        return [m[k] for k in ("sto", "con", "sea", "wel", "rec", "sur", "riv", "lak", "drn")] + [fv, pv, g.water_table()]
    if kind == "forward":
        return state["net"].infer(0, state["n"])
    loss, grad, out = state["net"].loss_grad(0, want_out=True, n=state["n"])
    return [loss, grad, out]


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    """Bytes and operations of one pass.  Per cell and Newton iteration: the assembly reads the
    state, soils and face coefficients and writes the seven bands and the right-hand side (280 B);
    two Jacobi sweeps before and after, the residual and the transfers of a V-cycle on the level-1
    bands and on coarse levels worth a quarter of them (280 B with FP32 bands, 500 B with FP64);
    the matrix-vector product (72 B) and the Krylov and line-search vectors (180 B).  A hierarchy
    is built from the bands (100 B in, 150 B out).  Iterations per step: 10 on the blocks, 3 in the
    box; a DILU solve takes about 10 Krylov iterations of two solves and products each."""
    kind = case["kind"]
    if kind == "ensemble":
        n = case["members"] * 500_000
        return dict(bytes=n * case["steps"] * (8 * 812.0) + n * 250.0, flops=n * case["steps"] * 8 * 700.0)
    n = float(case["nx"] * case["ny"] * case["nz"])
    if kind == "box":
        return dict(bytes=n * case["steps"] * 3 * (460.0 + 20 * 250.0), flops=n * case["steps"] * 3 * 1500.0)
    if kind == "block":
        it = n * case["steps"] * 10
        if case["precon"] == 0:
            return dict(bytes=it * (460.0 + 10 * 450.0), flops=it * 1500.0)
        if case["lag"] == 0:
            return dict(bytes=it * (280 + 500 + 72 + 180 + 250.0), flops=it * 900.0)
        conv = n * case["steps"] * (34.6e3 if case["guess"] == 2 else 0.0)
        return dict(bytes=it * (280 + 280 + 72 + 180.0) + n * 250.0, flops=it * 700.0 + conv)
    if kind == "host":
        return dict(bytes=n * (10 * 1282.0 + 56.0), flops=n * 9000.0)
    if kind == "linear":
        return dict(bytes=n * (164 + 280 + 250 + 3 * 750 + 8 * 13.0), flops=n * 3000.0)
    if kind == "outputs":
        return dict(bytes=n * (2 * 60 + 80 + 13 * 8.0), flops=n * 400.0)
    if kind == "forward":
        return dict(bytes=n * (32 + 4.0), flops=n * 34.6e3)
    return dict(bytes=n * (32 + 4 + 4.0), flops=n * 3 * 34.6e3)


# ---- the same in 64 bits, from the equations -------------------------------------------------
def _soil(p, h):
    """Saturation, relative permeability and active storage coefficient at heads h."""
    c = lambda a: torch.as_tensor(np.asarray(a), device="cuda").double()  # noqa: E731
    psi = h - c(p.cell_top)
    n = c(p.retn)
    m = 1.0 - 1.0 / n
    dry = psi < 0
    se = torch.where(dry, (1.0 + (psi.clamp(max=0).abs() * c(p.reta)) ** n) ** (-m), torch.ones_like(psi))
    poro, resi = c(p.poro), c(p.resi)
    srat = torch.where(dry, (resi + (poro - resi) * se) / poro, torch.ones_like(psi))
    kr = torch.where(dry, se.sqrt() * (1.0 - (1.0 - se ** (1.0 / m)) ** m) ** 2, torch.ones_like(psi))
    return srat, kr, torch.where(dry, torch.zeros_like(psi), c(p.ss))


def _faces(p, h, kr):
    """Per direction (up, north, west, east, south, down), as [nz, ny, nx]: the velocity into the
    cell through its interior faces and the flow (velocity times area)."""
    shape = (p.nz, p.ny, p.nx)
    c = lambda a: torch.as_tensor(np.asarray(a), device="cuda").double()  # noqa: E731
    dis, area = c(p.dis2face).reshape((6,) + shape), c(p.face_area).reshape((6,) + shape)
    h, kr = h.reshape(shape), kr.reshape(shape)
    vel, flow = [], []
    for d, (axis, step, ks) in enumerate(((0, -1, p.ksz), (1, -1, p.ksy), (2, -1, p.ksx), (2, 1, p.ksx), (1, 1, p.ksy),
                                          (0, 1, p.ksz))):
        k = c(ks).reshape(shape)
        n = shape[axis]
        own = [slice(None)] * 3
        nb = [slice(None)] * 3
        own[axis], nb[axis] = (slice(1, n), slice(0, n - 1)) if step < 0 else (slice(0, n - 1), slice(1, n))
        own, nb = tuple(own), tuple(nb)
        d1, d2 = dis[(d,) + own], dis[(5 - d,) + nb]
        k12 = k[own] * k[nb] * (d1 + d2) / (d1 * k[nb] + d2 * k[own])
        dh = h[nb] - h[own]
        v = k12 * torch.where(dh <= 0, kr[own], kr[nb]) * dh / (d1 + d2)
        full, q = torch.zeros(shape, device="cuda", dtype=torch.float64), torch.zeros(shape, device="cuda", dtype=torch.float64)
        full[own] = v
        q[own] = v * area[(d,) + own]
        vel.append(full)
        flow.append(q)
    return vel, sum(flow)


def _storage(p, h, h_old, delt, old_alp_is_new):
    """Storage term: the residual takes the new level's storage coefficient at both levels, the
    mass balance each level's own."""
    s, kr, alp = _soil(p, h)
    s_old, _, alp_old = _soil(p, h_old)
    alp_old = alp if old_alp_is_new else alp_old
    poro = torch.as_tensor(p.poro, device="cuda").double()
    vol = torch.as_tensor(p.cell_vol, device="cuda").double()
    ch = alp * s * h - alp_old * s_old * h_old + poro * (s - s_old)
    return -ch * vol / delt, s, kr


def _network_weights(seed):
    """Weights of a trained network's size: the shipped ones, each scaled by a few per cent."""
    w = np.load(_WEIGHTS).astype(np.float32)
    return (w * (1.0 + 0.05 * np.random.default_rng(seed).standard_normal(w.shape))).astype(np.float32)


def _network(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    x = torch.zeros((n, 16), device="cuda")
    x[:, :7] = 0.7 * torch.randn((n, 7), generator=_generator(seed), device="cuda")
    y = 0.3 * torch.randn(n, generator=_generator(seed + 1), device="cuda")
    params = [(torch.tensor(W, device="cuda", dtype=torch.float64, requires_grad=True),
               torch.tensor(b, device="cuda", dtype=torch.float64, requires_grad=True))
              for W, b in unpack(_network_weights(seed))]
    a = x.double().reshape(nz, ny, nx, 16)
    for layer, (W, b) in enumerate(params):
        pad = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
        a = b
        for tap in range(27):
            dz, dy, dx = tap // 9, (tap // 3) % 3, tap % 3
            a = a + pad[dz:dz + nz, dy:dy + ny, dx:dx + nx] @ W[tap].T
        if layer < 3:
            a = torch.nn.functional.gelu(a)
    return a[..., 0].reshape(-1), y.double(), params


def exact(case, seed):
    kind = case["kind"]
    if kind == "forward":
        with torch.no_grad():
            return _network(case, seed)[0]
    if kind == "gradient":
        out, y, params = _network(case, seed)
        loss = ((out - y) ** 2).mean()
        loss.backward()
        return [loss.detach(), torch.cat([t.grad.reshape(-1) for pair in params for t in pair]), out.detach()]
    if kind not in ("linear", "outputs"):
        return None   # iterated to a tolerance: no value to be had apart from the iteration
    p = _block(case, seed)
    S = p.ncals
    if kind == "linear":
        h = torch.as_tensor(_heads(p, seed, 1.0e-3), device="cuda")
        sto, _, kr = _storage(p, h, torch.as_tensor(p.head0, device="cuda"), p.params["ini_step"], True)
        f = sto + _faces(p, h, kr)[1].reshape(-1)
        f[:S] += torch.as_tensor(p.rech, device="cuda")
        return [f, None, None, -f, None]
    h_old = torch.as_tensor(_heads(p, seed + 1, 0.02), device="cuda")
    h = torch.as_tensor(_heads(p, seed, 0.02), device="cuda")
    sto, s, kr = _storage(p, h, h_old, 1.0, False)
    vel, flow = _faces(p, h, kr)
    d1 = torch.as_tensor(p.dis2face[:S], device="cuda").double()
    ksz = torch.as_tensor(p.ksz[:S], device="cuda").double()
    vel[0][0] = (ksz * (h_old[:S] - h[:S]) / d1 * kr[:S]).reshape(p.ny, p.nx)
    face = torch.stack(vel).reshape(6, -1)
    point = []
    for a, b, sign in ((2, 3, 1.0), (1, 4, 1.0), (0, 5, -1.0)):
        u, w = face[a], face[b]
        point.append(sign * torch.where(u * w < 0, 0.5 * (u - w), u - w))
    wt = h[:S].clone()
    for k in range(p.nz):
        layer = slice(k * S, (k + 1) * S)
        wt = torch.where(s[layer] != 1.0, h[layer], wt)
    rec = torch.as_tensor(p.rech, device="cuda") * 600.0
    return [sto, flow.reshape(-1) * 600.0, None, None, rec, None, None, None, None, face, torch.stack(point), wt]
