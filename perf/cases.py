"""What the speed of this framework is measured on: calls of its public entry
points as a flow solver's program makes them, from one step on a small host
array to time loops on 2048 x 2048 grids.

Kinds of case (``kind``):
  rhs      F and check_conservation of a state: what a program evaluates after
           every step to log the residual, momentum and energy
  poisson  one pressure_poisson solve
  step     time_ERK, ``steps`` steps in one call (RK44)
  ens      ``steps`` steps of an ensemble of uneven flows
  network  the learned guess's network: a forward pass, and loss and gradient

Flows (``flow``): ``periodic`` (uniform grid; decaying turbulence or the
inviscid Taylor-Green vortex), ``cavity`` (lid-driven), ``channel`` (inflow
left, outflow right; also the backward-facing step's inflow profile).  Bounded
flows have tanh-stretched grids where ``stretch`` is not 0.
"""
import math

import numpy as np
import torch

import ins2d_b200
from ins2d_b200 import cases as flows
from ins2d_b200 import ensembles, learned


def listed():
    return [
        # one step per call on host arrays, as a MATLAB-style program makes it: the 40 x 40 periodic shear-layer grid
        dict(name="step_shear_40_host", kind="step", flow="periodic", nx=40, ny=40, Re=1e3, poisson=6, steps=1, host=True, precision="fp64"),
        # the per-step diagnostics of the 64 x 64 lid-driven cavity: launches and round trips
        dict(name="rhs_cavity_64", kind="rhs", flow="cavity", nx=64, ny=64, Re=1e3, stretch=0.0),
        # the same diagnostics of the 2048 x 2048 turbulence run
        dict(name="rhs_periodic_2048", kind="rhs", flow="periodic", nx=2048, ny=2048, Re=2e3, stretch=0.0),
        # a transform solve on a grid whose sides are no powers of two
        dict(name="poisson_fft_1000x600", kind="poisson", flow="periodic", nx=1000, ny=600, poisson=6, stretch=0.0),
        # a conjugate-gradient solve on an odd-sized stretched channel
        dict(name="poisson_channel_301x257", kind="poisson", flow="channel", nx=301, ny=257, poisson=4, stretch=1.5),
        # time loops: the 64 x 64 cavity, small and bound by latency
        dict(name="step_cavity_64", kind="step", flow="cavity", nx=64, ny=64, Re=1e3, stretch=0.0, poisson=4, steps=10, host=False, precision="fp64"),
        # the inviscid 512 x 512 Taylor-Green vortex
        dict(name="step_taylor_green_512", kind="step", flow="periodic", nx=512, ny=512, Re=1e30, poisson=6, steps=10, host=False, precision="fp64"),
        # the stretched backward-facing step
        dict(name="step_bfs_512", kind="step", flow="channel", nx=512, ny=512, Re=800.0, stretch=1.02, bfs=True, poisson=4, steps=2, host=False, precision="fp64"),
        # 2048 x 2048 decaying turbulence, in FP64 and with FP32 stencils
        dict(name="step_turbulence_2048", kind="step", flow="periodic", nx=2048, ny=2048, Re=2e3, poisson=6, steps=2, host=False, precision="fp64"),
        dict(name="step_turbulence_2048_fp32", kind="step", flow="periodic", nx=2048, ny=2048, Re=2e3, poisson=6, steps=2, host=False, precision="fp32"),
        # snapshot generation: cavities and channels of many sizes advanced together
        dict(name="ensemble_24", kind="ens", members=24, smallest=64, largest=256, pick=4, steps=10),
        # inference and one training batch of the learned guess's network
        dict(name="network_4x512", kind="network", batch=4, height=512, width=512),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi]; one in three a power of two or a multiple of 8, the others as they fall."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    r = rng.random()
    if r < 0.2:
        n = 1 << int(round(math.log2(n)))
    elif r < 0.33:
        n = 8 * max(1, n // 8)
    return min(max(n, lo), hi)


def draw(rng):
    kind = rng.choice(["rhs", "poisson", "step", "step", "ens", "network"])
    flow = rng.choice(["periodic", "cavity", "channel"])
    per = flow == "periodic"
    if kind == "network":
        return dict(kind=kind, batch=rng.randint(1, 4), height=_size(rng, 32, 512), width=_size(rng, 32, 512))
    if kind == "ens":
        small = rng.randint(24, 64)
        return dict(kind=kind, members=rng.randint(4, 20), smallest=small, largest=rng.randint(small + 16, 192), pick=rng.randint(0, 999), steps=rng.randint(4, 10))
    Re = round(math.exp(rng.uniform(math.log(100.0), math.log(5000.0))), 1)
    stretch = 0.0 if per else rng.choice([0.0, 1.05, 1.5])
    if kind == "rhs":
        nx, ny = _size(rng, 16, 2048), _size(rng, 16, 2048)
        return dict(kind=kind, flow=flow, nx=nx, ny=ny, Re=Re, stretch=stretch)
    while True:
        top = 2048 if per else 400
        nx, ny = _size(rng, 24, top), _size(rng, 24, top)
        pow2 = nx & (nx - 1) == 0 and ny & (ny - 1) == 0
        if not per or pow2 or nx * ny * (nx + ny) <= 1000 * 600 * 1600:
            break
    if kind == "poisson":
        return dict(kind=kind, flow=flow, nx=nx, ny=ny, poisson=6 if per else 4, stretch=stretch)
    host = rng.random() < 0.2
    return dict(kind=kind, flow=flow, nx=nx, ny=ny, Re=Re, stretch=stretch, poisson=6 if per else 4, steps=1 if host else rng.randint(1, 4),
                host=host, precision=rng.choice(["fp64", "fp64", "fp32"]))


# --- grids, boundary conditions and states ----------------------------------------
def _case_options(case):
    """Keyword arguments of Options for a rhs, poisson or step case."""
    nx, ny, st = case["nx"], case["ny"], case.get("stretch", 0.0)
    kw = dict(Re=case.get("Re", 1e3), poisson=case.get("poisson", 6 if case["flow"] == "periodic" else 4), precision=case.get("precision", "fp64"))
    if case["flow"] == "periodic":
        # the unit square, stretched with the grid so that the cells stay square
        kw.update(x=flows.uniform_grid(nx, 0.0, 1.0), y=flows.uniform_grid(ny, 0.0, ny / nx), BC=flows.BC_PERIODIC)
    elif case["flow"] == "cavity":
        kw.update(x=flows.tanh_grid(nx, 0.0, 1.0, st), y=flows.tanh_grid(ny, 0.0, 1.0, st), BC=flows.BC_CAVITY, uBC=flows.lid_uBC(1.0, 1.0))
    else:
        kw.update(x=flows.tanh_grid(nx, 0.0, 30.0 if case.get("bfs") else 4.0, st), y=flows.tanh_grid(ny, -0.5, 0.5, st), BC=flows.BC_CHANNEL,
                  uBC=flows.channel_uBC(lambda y: _inflow(y, case.get("bfs", False))))
    return kw


def _inflow(y, bfs, U=1.0):
    y = np.asarray(y, dtype=np.float64)
    return np.where(y > 0.0, 24.0 * y * (0.5 - y), 0.0) if bfs else U * (1.0 - 4.0 * y ** 2)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _streamfunction(nx, ny, gen):
    """Random-phase streamfunction at (ny, nx) points with the energy spectrum k^4 exp(-2 (k/10)^2), rms 1."""
    kx = torch.fft.rfftfreq(nx, d=1.0 / nx, dtype=torch.float64, device="cuda")
    ky = torch.fft.fftfreq(ny, d=1.0 / ny, dtype=torch.float64, device="cuda")
    k = torch.sqrt(kx[None, :] ** 2 + ky[:, None] ** 2)
    amp = torch.where(k > 0, k ** 0.5 * torch.exp(-((k / 10.0) ** 2)), torch.zeros_like(k))
    ph = torch.rand(amp.shape, dtype=torch.float64, device="cuda", generator=gen) * (2 * math.pi)
    psi = torch.fft.irfft2(amp * torch.exp(1j * ph), s=(ny, nx))
    return psi / psi.square().mean().sqrt()


def _state(x, y, flow, gen, inflow=None, noise=0.0, taylor_green=False):
    """(V, p) on the GPU: a discretely divergence-free velocity of order one, and zero pressure."""
    hx = torch.tensor(np.diff(x), device="cuda")
    hy = torch.tensor(np.diff(y), device="cuda")
    nx, ny = len(hx), len(hy)
    if taylor_green:  # perturbed by the seed, so that another seed is another state
        X = torch.arange(nx, dtype=torch.float64, device="cuda") * (2 * math.pi / nx)
        Y = torch.arange(ny, dtype=torch.float64, device="cuda") * (2 * math.pi / ny)
        psi = torch.cos(X)[None, :] * torch.cos(Y)[:, None] + 1e-3 * _streamfunction(nx, ny, gen)
    else:
        psi = _streamfunction(nx, ny, gen)
    if flow == "periodic":
        u = (torch.roll(psi, -1, 0) - psi) / hy[:, None]
        v = -(torch.roll(psi, -1, 1) - psi) / hx[None, :]
        s = torch.sqrt((u.square().mean() + v.square().mean()) / 2)
        u, v = u / s + 0.1, v / s - 0.05
    else:
        # corner values, smoothly zero at the walls
        P = torch.zeros((ny + 1, nx + 1), dtype=torch.float64, device="cuda")
        P[:ny, :nx] = psi
        X = torch.tensor((x - x[0]) / (x[-1] - x[0]), device="cuda")
        Y = torch.tensor((y - y[0]) / (y[-1] - y[0]), device="cuda")
        P = P * (torch.sin(math.pi * X) ** 2)[None, :] * (torch.sin(math.pi * Y) ** 2)[:, None]
        P[0] = P[-1] = 0.0
        P[:, 0] = P[:, -1] = 0.0
        u = (P[1:] - P[:-1]) / hy[:, None]
        v = -(P[:, 1:] - P[:, :-1]) / hx[None, :]
        s = 4.0 * torch.maximum(u.abs().max(), v.abs().max())
        u, v = u / s, v / s
        if inflow is not None:
            u = u + torch.tensor(inflow, device="cuda")[:, None]
        u, v = (u[:, 1:-1] if flow == "cavity" else u[:, 1:]), v[1:-1]
    V = torch.cat([u.reshape(-1), v.reshape(-1)]).contiguous()
    if noise:
        V = V + noise * torch.randn(V.shape, dtype=torch.float64, device="cuda", generator=gen)
    return V, torch.zeros(nx * ny, dtype=torch.float64, device="cuda")


def _time_step(kw, U):
    """CFL 0.5 on periodic grids; the explicit RK4 limit on bounded ones."""
    if kw["BC"] is flows.BC_PERIODIC:
        return 0.5 * min(np.min(np.diff(kw["x"])), np.min(np.diff(kw["y"]))) / U
    return ensembles.stable_dt(kw, U)


def _flow_inputs(case, seed):
    kw = _case_options(case)
    gen = _gen(seed)
    yp = (kw["y"][1:] + kw["y"][:-1]) / 2
    inflow = _inflow(yp, case.get("bfs", False)) if case["flow"] == "channel" else None
    V, p = _state(kw["x"], kw["y"], case["flow"], gen, inflow, noise=1e-2 if case["kind"] == "rhs" else 0.0, taylor_green=kw["Re"] > 1e20)
    if case["kind"] == "rhs":
        p = torch.randn(p.shape, dtype=torch.float64, device="cuda", generator=gen)
    f = None
    if case["kind"] == "poisson":  # a right-hand side in the range of the operator: of mean zero on a closed domain
        f = torch.randn(p.shape, dtype=torch.float64, device="cuda", generator=gen)
        if case["flow"] != "channel":
            f = f - f.mean()
    return kw, V, p, f


def _ens_members(case):
    lo, hi = case["smallest"], case["largest"]
    sizes = tuple(sorted({lo, hi, (lo + hi) // 2, (3 * lo + hi) // 4, (lo + 3 * hi) // 4}))
    return ensembles.random_members(case["members"], seed=case["pick"], sizes=sizes, CG_acc=1e-12)


def _ens_inputs(case, seed):
    """Per member: Options' keyword arguments, its state and its time step."""
    out = []
    for m, kw in enumerate(_ens_members(case)):
        cavity = m % 2 == 0
        yp = (kw["y"][1:] + kw["y"][:-1]) / 2
        V, p = _state(kw["x"], kw["y"], "cavity" if cavity else "channel", _gen(1000 * seed + m), None if cavity else _inflow(yp, False, kw["_U"]))
        out.append((kw, V, p, min(5e-4, ensembles.stable_dt(kw, kw["_U"] + 0.5))))
    return out


def _net_inputs(case, seed):
    g = np.random.default_rng(seed)
    fan = [9] + [288] * 5
    shapes = [32 * 9] + [32 * 9 * 32] * 4 + [9 * 32]
    w = np.concatenate([g.standard_normal(n) * math.sqrt(2.0 / f) for n, f in zip(shapes, fan)]).astype(np.float32)
    gen = _gen(seed)
    shape = (case["batch"], case["height"], case["width"])
    return w, 0.7, torch.randn(shape, device="cuda", generator=gen), torch.randn(shape, device="cuda", generator=gen)


def prepare(case, seed):
    if case["kind"] == "network":
        w, scale, inp, tgt = _net_inputs(case, seed)
        net = learned.ConvNet()
        net.set_params(w, scale)
        return dict(kind="network", net=net, inp=inp, tgt=tgt)
    if case["kind"] == "ens":
        members = _ens_inputs(case, seed)
        ens = ins2d_b200.Ensemble([kw for kw, _, _, _ in members])
        for m, (_, V, p, dt) in enumerate(members):
            ens.set_state(m, V, p)
            ens.set_member_dt(m, dt)
        # where the program collects the members' snapshots
        return dict(kind="ens", ens=ens, steps=case["steps"], out=[(torch.empty_like(V), torch.empty_like(p)) for _, V, p, _ in members])
    kw, V, p, f = _flow_inputs(case, seed)
    s = dict(kind=case["kind"], m=ins2d_b200.Options(**kw), V=V, p=p, f=f, t=0.0, steps=case.get("steps", 0))
    if case["kind"] == "step":
        s["dt"] = _time_step(kw, 4.0 if case["flow"] == "periodic" else 1.5)
        if case["host"]:
            s["V"], s["p"] = V.cpu().numpy(), p.cpu().numpy()
    return s


def run(s):
    if s["kind"] == "network":
        y = s["net"].forward(s["inp"])
        loss, grad = s["net"].loss_grad(s["inp"], s["tgt"])
        return dict(y=y, loss=loss, grad=grad)
    if s["kind"] == "ens":
        s["ens"].time_ERK(0.0, 5e-4, s["steps"])
        return [s["ens"].get_state(m, V, p) for m, (V, p) in enumerate(s["out"])]
    m = s["m"]
    if s["kind"] == "rhs":
        maxres, F = m.F(s["V"], None, s["p"])
        return dict(maxres=maxres, F=F, conservation=m.check_conservation(s["V"]))
    if s["kind"] == "poisson":
        return m.pressure_poisson(s["f"])
    # the time loop goes on from where it is
    s["V"], s["p"] = m.time_ERK(s["V"], s["p"], s["t"], s["dt"], s["steps"])
    s["t"] += s["steps"] * s["dt"]
    return s["V"], s["p"]


# --- what a pass cannot do without ----------------------------------------------------
_RHS_FLOPS = 100  # per cell: convection, diffusion and pressure gradient of both components


def _solve_flops(nx, ny):
    """A transform solve: forward and inverse 2D transforms of nx x ny real values."""
    return 2 * 2.5 * nx * ny * math.log2(nx * ny) + 4 * nx * ny


def _step_work(nx, ny, steps):
    # per RK44 step: four right-hand sides beside the stage combinations, four projections and four solves; the
    # state (V and p: 24 bytes a cell) read and written
    return dict(bytes=48.0 * nx * ny * steps, flops=4 * steps * (nx * ny * (_RHS_FLOPS + 30) + _solve_flops(nx, ny)))


def work(case):
    if case["kind"] == "network":
        n = case["batch"] * case["height"] * case["width"]
        fwd = 2 * 9 * (32 + 4 * 32 * 32 + 32) * n
        # two forward passes, the backward pass to the data and that to the weights
        return dict(bytes=4.0 * (4 * n) + 3 * 4 * 37440, flops=4.0 * fwd)
    if case["kind"] == "ens":
        ws = [_step_work(len(kw["x"]) - 1, len(kw["y"]) - 1, case["steps"]) for kw in _ens_members(case)]
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    if case["kind"] == "rhs":
        return dict(bytes=40.0 * n, flops=(_RHS_FLOPS + 12.0) * n)
    if case["kind"] == "poisson":
        return dict(bytes=16.0 * n, flops=_solve_flops(nx, ny))
    return _step_work(nx, ny, case["steps"])


# --- the same in 64 bits, from the discretisation's definition -----------------------
class _Exact:
    """The second-order staggered discretisation on explicit ghost values, fields as (row j, column i) tensors.  The normal
    velocity is zero at walls, the tangential one that of the lid; inflow on the left, zero normal derivative at the outflow."""

    def __init__(self, x, y, flow, Re, lid=0.0, inflow=None):
        t = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")  # noqa: E731
        self.flow, self.Re, self.lid = flow, Re, lid
        hx, hy = np.diff(x), np.diff(y)
        self.nx, self.ny = nx, ny = len(hx), len(hy)
        per, out = flow == "periodic", flow == "channel"
        # spacing of the unknowns, and of the points beside them
        mid = lambda h: (h[1:] + h[:-1]) / 2  # noqa: E731
        gx, gy = mid(hx), mid(hy)
        self.gx = t(np.r_[(hx[0] + hx[-1]) / 2, gx] if per else np.r_[gx, hx[-1] / 2] if out else gx)
        self.gy = t(np.r_[(hy[0] + hy[-1]) / 2, gy] if per else gy)
        self.hx, self.hy = t(hx), t(hy)
        wx, wy = ((hx[0] + hx[-1]) / 2, (hy[0] + hy[-1]) / 2) if per else (hx[0], hy[0])
        wx1, wy1 = (wx, wy) if per else (hx[-1], hy[-1])
        self.dvx, self.duy = t(np.r_[wx, gx, wx1]), t(np.r_[wy, gy, wy1])  # between staggered neighbours, over the boundaries
        self.dux = t(np.r_[hx[-1], hx] if per else np.r_[hx, hx[-1]] if out else hx)
        self.dvy = t(np.r_[hy[-1], hy] if per else hy)
        self.ex = t(np.r_[hx[-1], hx, hx[0]] if per else np.r_[hx[0], hx, hx[-1]])  # cell widths with the ghost cells'
        self.ey = t(np.r_[hy[-1], hy, hy[0]] if per else np.r_[hy[0], hy, hy[-1]])
        self.inflow = t(inflow) if inflow is not None else None
        self.nxu = {"periodic": nx, "cavity": nx - 1, "channel": nx}[flow]
        self.mv = ny if per else ny - 1

    def split(self, V):
        n = self.nxu * self.ny
        return V[:n].reshape(self.ny, self.nxu), V[n:].reshape(self.mv, self.nx)

    def _left(self, u):
        b = torch.zeros_like(u[:, :1])
        return b if self.inflow is None else b + self.inflow[:, None]

    def u_lines(self, u):
        """u on all grid lines x_0 .. x_nx."""
        if self.flow == "periodic":
            return torch.cat([u, u[:, :1]], 1)
        if self.flow == "channel":
            return torch.cat([self._left(u), u], 1)
        return torch.cat([self._left(u), u, torch.zeros_like(u[:, :1])], 1)

    def v_lines(self, v):
        if self.flow == "periodic":
            return torch.cat([v, v[:1]], 0)
        z = torch.zeros_like(v[:1])
        return torch.cat([z, v, z], 0)

    def u_ghost_x(self, u):
        if self.flow == "periodic":
            return torch.cat([u[:, -1:], u, u[:, :1]], 1)
        if self.flow == "channel":
            return torch.cat([self._left(u), u, u[:, -1:]], 1)
        return self.u_lines(u)

    def v_ghost_y(self, v):
        return torch.cat([v[-1:], v, v[:1]], 0) if self.flow == "periodic" else self.v_lines(v)

    def u_ghost_y(self, u):
        if self.flow == "periodic":
            return torch.cat([u[-1:], u, u[:1]], 0)
        return torch.cat([-u[:1], u, 2 * self.lid - u[-1:]], 0)

    def v_ghost_x(self, v):
        if self.flow == "periodic":
            return torch.cat([v[:, -1:], v, v[:, :1]], 1)
        return torch.cat([-v[:, :1], v, v[:, -1:] if self.flow == "channel" else -v[:, -1:]], 1)

    def rhs(self, V):
        """-convection + diffusion of u and v."""
        u, v = self.split(V)
        dx, dy = (lambda a: a[:, 1:] - a[:, :-1]), (lambda a: a[1:] - a[:-1])
        mx, my = (lambda a: 0.5 * (a[:, 1:] + a[:, :-1])), (lambda a: 0.5 * (a[1:] + a[:-1]))
        per, out = self.flow == "periodic", self.flow == "channel"
        ux, uy, vx, vy = self.u_ghost_x(u), self.u_ghost_y(u), self.v_ghost_x(v), self.v_ghost_y(v)
        fu = dx(self.hy[:, None] * mx(ux) ** 2)
        c = mx(self.v_ghost_x(self.v_lines(v)) * self.ex[None, :])  # flux of v through the corners' u columns
        if out:
            c = torch.cat([c[:, :-1], 0.5 * c[:, -1:]], 1)
        c = c[:, :-1] if per else c[:, 1:] if out else c[:, 1:-1]
        fu = fu + dy(c * my(uy))
        c = my(self.u_ghost_y(self.u_lines(u)) * self.ey[:, None])
        c = c[:-1] if per else c[1:-1]
        fv = dx(c * mx(vx)) + dy(self.hx[None, :] * my(vy) ** 2)
        du = self.hy[:, None] * dx(dx(ux) / self.dux[None, :]) + self.gx[None, :] * dy(dy(uy) / self.duy[:, None])
        dv = self.gy[:, None] * dx(dx(vx) / self.dvx[None, :]) + self.hx[None, :] * dy(dy(vy) / self.dvy[:, None])
        return torch.cat([(du / self.Re - fu).reshape(-1), (dv / self.Re - fv).reshape(-1)])

    def gradient(self, p):
        p = p.reshape(self.ny, self.nx)
        if self.flow == "periodic":
            px, py = torch.cat([p[:, -1:], p], 1), torch.cat([p[-1:], p], 0)
        else:
            px = torch.cat([p, torch.zeros_like(p[:, :1])], 1) if self.flow == "channel" else p
            py = p
        return torch.cat([(self.hy[:, None] * (px[:, 1:] - px[:, :-1])).reshape(-1), (self.hx[None, :] * (py[1:] - py[:-1])).reshape(-1)])

    def volume(self):
        return torch.cat([(self.hy[:, None] * self.gx[None, :]).reshape(-1), (self.gy[:, None] * self.hx[None, :]).reshape(-1)])

    def divergence(self, V, boundary=True):
        u, v = self.split(V)
        if not boundary:
            keep, self.inflow = self.inflow, None
        ul, vl = self.u_lines(u), self.v_lines(v)
        if not boundary:
            self.inflow = keep
        return (self.hy[:, None] * (ul[:, 1:] - ul[:, :-1]) + self.hx[None, :] * (vl[1:] - vl[:-1])).reshape(-1)

    def _basis(self, h, g):
        """Eigenvectors of the 1D pressure operator in the cell widths' inner product."""
        n = len(h)
        D = torch.zeros((n, len(g)), dtype=torch.float64, device="cuda")
        k = torch.arange(len(g), device="cuda")
        D[k, k] = 1.0
        r = k[: n - 1]
        D[r + 1, r] = -1.0
        T = (D / g[None, :]) @ D.T
        s = 1.0 / torch.sqrt(h)
        lam, W = torch.linalg.eigh(s[:, None] * T * s[None, :])
        return lam, s[:, None] * W

    def solve(self, f):
        """dp with M Om^-1 G dp = f; on closed domains without the constant, on periodic ones with its transform's mean."""
        f = f.reshape(self.ny, self.nx)
        if self.flow == "periodic":
            dx, dy = float(self.hx[0]), float(self.hy[0])
            I = torch.arange(self.nx // 2 + 1, dtype=torch.float64, device="cuda")
            J = torch.arange(self.ny, dtype=torch.float64, device="cuda")
            a = 4 * dx * dy * (torch.sin(math.pi * J / self.ny)[:, None] ** 2 / dy ** 2 + torch.sin(math.pi * I / self.nx)[None, :] ** 2 / dx ** 2)
            a[0, 0] = 1.0
            return torch.fft.irfft2(-torch.fft.rfft2(f) / a, s=(self.ny, self.nx)).reshape(-1)
        if not hasattr(self, "_bases"):
            self._bases = self._basis(self.hx, self.gx) + self._basis(self.hy, self.gy)
        lx, Qx, ly, Qy = self._bases
        lam = ly[:, None] + lx[None, :]
        w = Qy.T @ f @ Qx
        w = torch.where(lam > 1e-11 * lam.max(), -w / lam, torch.zeros_like(w))
        return (Qy @ w @ Qx.T).reshape(-1)

    def step(self, V, p, dt):
        """One classical Runge-Kutta step with a projection per stage and a final pressure solve."""
        vol = self.volume()
        Vn, U, k = V, V, []
        c = [0.5, 0.5, 1.0, 1.0]
        for i in range(4):
            k.append(self.rhs(U) / vol)
            T = (0.5 * k[0], 0.5 * k[-1], k[-1])[i] if i < 3 else (k[0] + 2 * k[1] + 2 * k[2] + k[3]) / 6
            dp = p if i == 0 else self.solve(self.divergence(Vn / dt + T, False) / c[i] + self._boundary() / dt / c[i])
            U = Vn + dt * (T - c[i] * self.gradient(dp) / vol)
        R = (self.rhs(U) - self.gradient(p)) / vol
        return U, p + self.solve(self.divergence(R, False))

    def _boundary(self):
        return self.divergence(torch.zeros_like(self.volume()))

    def conservation(self, V):
        u, v = self.split(V)
        vol = self.volume()
        wu, wv = self.split(vol)
        mom, k = (wu * u).sum(), 0.5 * (vol * V.square()).sum()
        if self.inflow is not None:
            mom = mom + (self.inflow * self.hy).sum() * self.hx[0] / 2
            k = k + 0.5 * (self.inflow.square() * self.hy).sum() * self.hx[0] / 2
        return tuple(float(a) for a in (self.divergence(V).abs().max(), mom, (wv * v).sum(), k))


def _exact_of(kw, flow, inflow=None, lid=1.0):
    return _Exact(kw["x"], kw["y"], flow, kw["Re"], lid if flow == "cavity" else 0.0, inflow)


def _exact_network(case, seed):
    w, scale, inp, tgt = _net_inputs(case, seed)
    w = torch.tensor(w, dtype=torch.float64, device="cuda", requires_grad=True)
    a, at = inp.double()[:, None], 0
    taps = [(1, 32)] + [(32, 32)] * 4 + [(32, 1)]
    for n, (ci, co) in enumerate(taps):
        k = w[at:at + 9 * ci * co].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        at += 9 * ci * co
        a = torch.nn.functional.conv2d(a, k, padding=1)
        a = torch.relu(a) if n < 5 else scale * a[:, 0]
    loss = (a - tgt.double()).square().mean()
    loss.backward()
    return dict(y=a.detach(), loss=float(loss.detach()), grad=w.grad.cpu().numpy())


def exact(case, seed):
    if case["kind"] == "network":
        return _exact_network(case, seed)
    if case["kind"] == "ens":
        out = []
        for m, (kw, V, p, dt) in enumerate(_ens_inputs(case, seed)):
            yp = (kw["y"][1:] + kw["y"][:-1]) / 2
            e = _exact_of(kw, "channel", _inflow(yp, False, kw["_U"])) if m % 2 else _exact_of(kw, "cavity", lid=kw["_U"])
            for _ in range(case["steps"]):
                V, p = e.step(V, p, dt)
            out.append((V, p))
        return out
    kw, V, p, f = _flow_inputs(case, seed)
    yp = (kw["y"][1:] + kw["y"][:-1]) / 2
    e = _exact_of(kw, case["flow"], _inflow(yp, case.get("bfs", False)) if case["flow"] == "channel" else None)
    if case["kind"] == "rhs":
        F = e.rhs(V) - e.gradient(p)
        return dict(maxres=float(F.abs().max()), F=F, conservation=e.conservation(V))
    if case["kind"] == "poisson":
        return e.solve(f)
    dt = _time_step(kw, 4.0 if case["flow"] == "periodic" else 1.5)
    for _ in range(case["steps"]):
        V, p = e.step(V, p, dt)
    return (V.cpu().numpy(), p.cpu().numpy()) if case["host"] else (V, p)
