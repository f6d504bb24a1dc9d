"""The calls whose speed is followed: time steps, Poisson solves, output-side
reductions and ensembles, each through the public interface of paratc_b200.

A case is a dict of plain values; listed() gives the fixed ones, draw() more of
the same ranges.  prepare() makes what a program holds before the call (the
context and the state, on the GPU), run() is one pass, exact() the same result
by plain torch in 64 bits.

kinds
  step      state in, `steps` calls of ChannelIterate, state out (device arrays)
  poisson   one pressure solve, source and potential in device arrays
  output    what a run does every ivstats / SaveVisu steps: clcStat's moments,
            the 1-D spectra and two dump_visu quantities of the current state
  ensemble  `members` independent channels advanced together
flows
  channel   closed channel, constant flow rate, fixed dt
  lock      half channel with a settling scalar, CFL-controlled dt, no flow-rate
            forcing (gravity current)
  turbidity as lock with the flow rate held constant
"""
import ctypes
import math

import numpy as np
import torch

from paratc_b200 import cases as workloads
from paratc_b200.abi import AB2, FT_CH, RK2, RK3
from paratc_b200.lib import BatchSystem, ChannelSystem, load, mesh_ycoord

DEV = "cuda"
F64 = torch.float64
SCHEMES = {"ab2": (AB2, 1), "rk2": (RK2, 2), "rk3": (RK3, 3)}
VISU = ("ux", "Q")
# transform lengths (nx / 2 and nz) met in drawn grids: powers of two and their
# multiples by 3, which a production grid takes, then lengths with factors 5
LENGTHS = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768)
ODD_LENGTHS = (18, 20, 36, 50, 54, 60, 72, 80, 90, 100, 108, 120, 144, 150, 160, 180, 200, 240, 250, 300, 320)


def _step(name, nx, ny, nz, steps, flow="channel", scheme="rk3", prec="fp64"):
    return dict(name=name, kind="step", flow=flow, nx=nx, ny=ny, nz=nz, steps=steps, scheme=scheme, prec=prec)


def listed():
    return [
        # a first run of an input deck on a small grid (tests/golden/channel_small.prm): launches and latency
        _step("channel_32x24x16", 32, 24, 16, 20),
        # the small gravity-current deck (GravityFlow.small): scalar, half channel, CFL-controlled dt
        _step("gravity_96x96x96", 96, 96, 96, 10, flow="lock"),
        # a grid whose lengths have factors 5: the transforms of any 2^a 3^b 5^c length, and RK2
        _step("channel_100x66x90_rk2", 100, 66, 90, 10, scheme="rk2"),
        # the Re_tau = 180 channel of the benchmark, FP64 and the FP32 storage form
        _step("channel_c1", 128, 96, 128, 10),
        _step("channel_c1_fp32", 128, 96, 128, 10, prec="fp32"),
        # the grid of the standard turbulent-channel deck (TurbCha0180_4th.standard)
        _step("channel_384x192x256", 384, 192, 256, 5),
        # the lock-exchange gravity current of the benchmark at full size, both storage forms
        _step("lock_c3", 1536, 160, 256, 4, flow="lock"),
        _step("lock_c3_fp32", 1536, 160, 256, 4, flow="lock", prec="fp32"),
        # pressure solves on their own: the channel's grid, and the benchmark's large grid
        dict(name="poisson_c1", kind="poisson", nx=128, ny=96, nz=128),
        dict(name="poisson_c2", kind="poisson", nx=512, ny=256, nz=512),
        # statistics, spectra and visualisation fields of the turbulent-channel deck's grid
        dict(name="output_384x192x256", kind="output", flow="channel", nx=384, ny=192, nz=256),
        # the benchmark's ensemble of uneven channels
        dict(name="ensemble_c4", kind="ensemble", members=32, seed_grids=2024, steps=5),
    ]


def _size(rng, kind, lo, hi, lengths):
    """A grid of between lo and hi cells (spread over the logarithm), ny even
    as a closed channel needs it."""
    while True:
        want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        nx, nz = 2 * rng.choice(lengths), rng.choice(lengths)
        ny = 2 * int(round(want / (nx * nz) / 2))
        if (16 if kind == "output" else 12) <= ny <= 256:
            return nx, ny, nz


def _odd(rng, flow):
    """A half channel takes any row count."""
    return 0 if flow == "channel" else rng.randint(0, 1)


def draw(rng):
    kind = rng.choices(["step", "poisson", "output", "ensemble"], [6, 2, 1, 1])[0]
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 32), seed_grids=rng.randint(1, 10 ** 6), steps=rng.randint(2, 5))
    if kind == "output":
        nx, ny, nz = _size(rng, kind, 1e5, 2e7, LENGTHS[2:])
        flow = rng.choice(["channel", "turbidity"])
        return dict(kind=kind, flow=flow, nx=nx, ny=ny - _odd(rng, flow), nz=nz)
    lengths = rng.choice([LENGTHS, LENGTHS, ODD_LENGTHS])
    if kind == "poisson":
        nx, ny, nz = _size(rng, kind, 1e4, 6e7, lengths)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz)
    nx, ny, nz = _size(rng, kind, 8e3, 4e7, lengths)
    prec = rng.choice(["fp64", "fp64", "fp32"]) if lengths is LENGTHS else "fp64"
    # about as many steps as lie between two statistics samples of the decks
    steps = 20 if nx * ny * nz < 1e5 else (10 if nx * ny * nz < 4e6 else 4)
    flow = rng.choice(["channel", "channel", "lock", "turbidity"])
    return dict(kind=kind, flow=flow, nx=nx, ny=ny - _odd(rng, flow), nz=nz,
                steps=steps, scheme=rng.choice(["rk3", "rk3", "rk3", "rk2", "ab2"]), prec=prec)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _workload(case):
    """The workload definition (parameters and mesh) of a case."""
    make = {"lock": workloads.lock_exchange_c3, "turbidity": workloads.turbidity_c5}.get(
        case.get("flow"), workloads.channel_c1)
    w = make(case["nx"], case["ny"], case["nz"])
    w.params.ischeme = SCHEMES[case.get("scheme", "rk3")][0]
    return w


def _grid(w):
    return mesh_ycoord(w.mesh, w.params.yly)


def _ptr(t):
    return ctypes.c_void_p(None if t is None else t.data_ptr())


def _initial(p, yp, seed):
    """A developing flow: a mean profile, a few large modes and noise in the
    velocity, made solenoidal; a smooth pressure; the scalar of a front."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    shape = (p.nzc, p.nyc, p.nxc)

    def noise(a):
        return (torch.rand(shape, generator=g, device=DEV, dtype=F64) * 2 - 1) * a

    x = (torch.arange(p.nxc, device=DEV, dtype=F64) / p.nxc * 2 * math.pi)[None, None, :]
    z = (torch.arange(p.nzc, device=DEV, dtype=F64) / p.nzc * 2 * math.pi)[:, None, None]
    y = torch.as_tensor(0.5 * (yp[1:] + yp[:-1]), device=DEV, dtype=F64)[None, :, None] / p.yly
    ph = torch.rand(8, generator=g, device=DEV, dtype=F64) * 2 * math.pi
    ub = p.ubulk if p.ubulk else 0.3
    eta = (2 * y - 1) if p.flow_type == FT_CH else (y - 1)
    ux = 1.5 * ub * (1 - eta * eta) + 0.1 * ub * torch.sin(2 * x + ph[0]) * torch.cos(z + ph[1]) + noise(0.1 * ub)
    uy = 0.1 * ub * torch.sin(x + ph[2]) * torch.sin(2 * z + ph[3]) + noise(0.1 * ub)
    uz = 0.1 * ub * torch.cos(x + ph[4]) * torch.sin(z + ph[5]) + noise(0.1 * ub)
    pr = 0.02 * ub * ub * torch.cos(x + ph[6]) * torch.cos(z + ph[7]) * torch.ones_like(y)
    c = None
    if p.scalar_on:
        c = (1 - y) * (0.6 + 0.3 * torch.cos(x + ph[0])) + noise(1e-3)
    m = _Torch(p, yp)
    ux, uy, uz = m.project(ux.contiguous(), uy.contiguous(), uz.contiguous())
    out = [None if t is None else t.contiguous() for t in (ux, uy, uz, pr, c)]
    # the contexts read these on streams of their own
    if DEV == "cuda":
        torch.cuda.synchronize()
    return out


def _member_loads(systems, states):
    L = load()
    for s, f in zip(systems, states):
        rc = L.paratc_set_fields_device(s.handle, *[_ptr(t) for t in f], None, None, None, None)
        if rc:
            raise RuntimeError("paratc_set_fields_device: %d" % rc)


def _member_reads(systems, outs):
    L = load()
    for s, o in zip(systems, outs):
        rc = L.paratc_get_fields_device(s.handle, *[_ptr(t) for t in o])
        if rc:
            raise RuntimeError("paratc_get_fields_device: %d" % rc)


def _out_like(p, hist=True):
    """Device arrays for u, v, w, p, c and the explicit histories."""
    shape = (p.nzc, p.nyc, p.nxc)

    def new():
        return torch.empty(shape, device=DEV, dtype=F64)

    sc = bool(p.scalar_on)
    return [new(), new(), new(), new(), new() if sc else None] + \
        ([new(), new(), new(), new() if sc else None] if hist else [None] * 4)


def _source(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    src = torch.randn((case["nz"], case["ny"], case["nx"]), generator=g, device=DEV, dtype=F64)
    src = src - src.mean()
    if DEV == "cuda":
        torch.cuda.synchronize()
    return src


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        ws = workloads.ensemble_c4(case["members"], case["seed_grids"])
        yps = [_grid(w) for w in ws]
        batch = BatchSystem([w.params for w in ws], yps)
        f = [_initial(w.params, yp, seed + i) for i, (w, yp) in enumerate(zip(ws, yps))]
        # the members' fields of one name lie in one array, member after member
        n = [w.n_cells for w in ws]
        flat = [torch.empty(sum(n), device=DEV, dtype=F64) for _ in range(4)]
        views = list(zip(*[t.split(n) for t in flat]))
        return dict(kind=kind, batch=batch, fields=f, out=[list(v) + [None] * 5 for v in views], flat=flat,
                    steps=case["steps"])
    w = workloads.poisson_c2(case["nx"], case["ny"], case["nz"]) if kind == "poisson" else _workload(case)
    yp = _grid(w)
    sys_ = ChannelSystem(w.params, yp)
    if kind == "poisson":
        src = _source(case, seed)
        return dict(kind=kind, sys=sys_, src=src, phi=torch.empty_like(src))
    f = _initial(w.params, yp, seed)
    if kind == "output":
        _member_loads([sys_], [f])
        n = case["nx"] * case["ny"] * case["nz"]
        sys_.spectra_reset()
        return dict(kind=kind, sys=sys_, fields=f, jlcs=max(1, case["ny"] // 8),
                    visu=[torch.empty(n, device=DEV, dtype=F64) for _ in VISU])
    sys_.precision = case["prec"]
    return dict(kind=kind, sys=sys_, fields=f, out=_out_like(w.params), steps=case["steps"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "ensemble":
        b = state["batch"]
        _member_loads(b.members, state["fields"])
        b.iterate(state["steps"])
        _member_reads(b.members, state["out"])
        return state["flat"]
    s = state["sys"]
    if kind == "poisson":
        s.poisson_device(state["src"].data_ptr(), state["phi"].data_ptr())
        return state["phi"]
    if kind == "output":
        s.stats_reset()
        s.spectra_reset()
        s.stats_accumulate()
        s.spectra_accumulate(state["jlcs"])
        for name, out in zip(VISU, state["visu"]):
            s.visu_quantity_device_async(name, out.data_ptr())
        stats = s.stats_get()[0]
        ex, ez = s.spectra_get()[:2]
        return [stats, ex, ez] + state["visu"]
    _member_loads([s], [state["fields"]])
    s.iterate(state["steps"])
    _member_reads([s], [state["out"]])
    return [t for t in state["out"] if t is not None]


def work(case):
    """Bytes: what has to pass through memory.  A substep reads and writes the
    state and the explicit histories once (its pressure solve couples every
    cell, so no two substeps share a pass); flops: the arithmetic of the
    stencils, sweeps and transforms."""
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(w.n_cells for w in workloads.ensemble_c4(case["members"], case["seed_grids"]))
        return {"bytes": cells * 3 * case["steps"] * 112.0, "flops": cells * 3 * case["steps"] * 500.0}
    cells = case["nx"] * case["ny"] * case["nz"]
    lg = math.log2(case["nx"]) + math.log2(case["nz"])
    if kind == "poisson":
        return {"bytes": cells * 16.0, "flops": cells * (5.0 * lg + 10)}
    if kind == "output":
        return {"bytes": cells * 8.0 * (4 + (case["flow"] != "channel") + len(VISU)), "flops": cells * (300.0 + 20 * lg)}
    sub = case["steps"] * SCHEMES[case["scheme"]][1]
    scalar = case["flow"] != "channel"
    values = 7 + 2 * scalar           # u, v, w, p, three histories (, c and its history)
    size = 8.0 if case["prec"] == "fp64" else 4.0
    per = 2 * (values * size + (8.0 - size))  # the pressure is 64-bit in every form
    return {"bytes": cells * sub * per, "flops": cells * sub * (400.0 + 150.0 * scalar + 5.0 * lg)}


# ---------------------------------------------------------------------------
# the same results by plain torch in 64 bits
# ---------------------------------------------------------------------------

class _Torch:
    """The step and the solve as whole-array expressions: periodic neighbours
    by torch.roll, the wall-normal systems of the Helmholtz solves dense, those
    of the Poisson solve by elimination over the rows.  Fields [nz, ny, nx];
    "full" arrays carry the two wall ghost rows."""

    IC = (-1 / 16, 9 / 16, 9 / 16, -1 / 16)

    def __init__(self, p, yp):
        self.p = p
        nx, ny, nz = p.nxc, p.nyc, p.nzc
        rdx, rdz = nx / p.xlx, nz / p.zlz
        self.dx = [rdx / 24, -rdx * 1.125, rdx * 1.125, -rdx / 24]
        self.dz = [rdz / 24, -rdz * 1.125, rdz * 1.125, -rdz / 24]
        self.dxx = [a * rdx * rdx for a in (-1 / 12, 4 / 3, -2.5, 4 / 3, -1 / 12)]
        self.dzz = [a * rdz * rdz for a in (-1 / 12, 4 / 3, -2.5, 4 / 3, -1 / 12)]
        self.rdx, self.rdz = rdx, rdz
        y = np.zeros(ny + 2)
        y[1:] = yp  # y[j], j = 1..ny+1
        yc = np.zeros(ny + 2)
        yc[1:ny + 1] = 0.5 * (y[1:ny + 1] + y[2:ny + 2])
        yc[0], yc[ny + 1] = 2 * y[1] - yc[1], 2 * y[ny + 1] - yc[ny]
        dyp = np.zeros(ny + 2)
        dyp[1:ny + 1] = y[2:ny + 2] - y[1:ny + 1]
        dyp[0], dyp[ny + 1] = dyp[1], dyp[ny]
        dyc = np.ones(ny + 2)
        dyc[2:ny + 1] = yc[2:ny + 1] - yc[1:ny]
        dyc[1], dyc[ny + 1] = dyp[1], dyp[ny]
        rp, rc = 1 / dyp, 1 / dyc
        self.dyc = dyc
        j = np.arange(1, ny + 1)
        am, ap = rp[j] * rc[j], rp[j] * rc[j + 1]  # cell-centred second difference

        def wall(am, ap, lo, hi):
            """Dirichlet walls half a cell away from rows 1 and ny."""
            am, ap = am.copy(), ap.copy()
            if lo:
                am[0], ap[0] = 4 * rc[1] / (dyc[1] + 2 * dyc[2]), 4 * rc[2] / (dyc[1] + 2 * dyc[2])
            if hi:
                am[-1] = 4 * rc[ny] / (dyc[ny + 1] + 2 * dyc[ny])
                ap[-1] = 4 * rc[ny + 1] / (dyc[ny + 1] + 2 * dyc[ny])
            return am, ap

        ch = p.flow_type == FT_CH
        cam, cap = wall(am, ap, True, ch)
        if not ch:
            cap[-1] = 0.0
        cac = -(cam + cap)
        self.c = (cam, cac, cap)
        nam, nac, nap = cam.copy(), cac.copy(), cap.copy()  # the implicit operator, ghosts eliminated
        nac[0] -= cam[0]
        if ch:
            nac[-1] -= cap[-1]
        self.cn = (nam, nac, nap)
        vam, vap = rc[j] * rp[j - 1], rc[j] * rp[j]  # faces
        self.v = (vam, -(vam + vap), vap)
        pam, pap = am.copy(), ap.copy()
        pam[0] = pap[-1] = 0.0
        self.ph = (pam, -(pam + pap), pap)
        if p.scalar_on:  # Robin below without flux, zero flux above
            f = p.scalar_bc_values[0]
            self.r1b = (2 + f * dyc[1]) / (2 - f * dyc[1])
            sac = -(am + ap)
            self.s = (am, sac.copy(), ap)
            sac[0] += am[0] * self.r1b
            sac[-1] += ap[-1]
            self.sn = (am, sac, ap)
        yi = dyp[1:ny + 2] / (dyp[1:ny + 2] + dyp[0:ny + 1])  # j = 1..ny+1
        self.iy1, self.iy3 = self._col(yi[:ny]), self._col(yi[1:ny + 1])
        self.rdyp, self.rdyc, self.dyp = self._col(rp[j]), self._col(rc[j]), self._col(dyp[j])

        def wave(n, r):
            w = 2 * math.pi * torch.arange(n, device=DEV, dtype=F64) / n
            return r * r / 288 * (torch.cos(3 * w) - 54 * torch.cos(2 * w) + 783 * torch.cos(w) - 730)

        self.lam = wave(nz, rdz)[:, None] + wave(nx, rdx)[None, :nx // 2 + 1]

    @staticmethod
    def _col(v):
        return torch.as_tensor(np.ascontiguousarray(v), device=DEV, dtype=F64)[None, :, None]

    @staticmethod
    def _comb(F, w, o, dim):
        """sum of w[q] * F at index + o + q along dim (periodic)."""
        out = None
        for q, a in enumerate(w):
            t = torch.roll(F, -(o + q), dims=dim) * a
            out = t if out is None else out + t
        return out

    def X(self, F, w, o):
        return self._comb(F, w, o, 2)

    def Z(self, F, w, o):
        return self._comb(F, w, o, 0)

    def _yy(self, F, co):
        am, ac, ap = (self._col(a) for a in co)
        return am * F[:, :-2] + ac * F[:, 1:-1] + ap * F[:, 2:]

    def _full(self, F, lo, hi):
        return torch.cat([lo, F, hi], dim=1)

    def vel(self, ux, uy, uz):
        """With the wall ghost rows (uy of row 1 is the lower wall's)."""
        s = -1.0 if self.p.flow_type == FT_CH else 1.0
        z = torch.zeros_like(uy[:, :1])
        uy = torch.cat([z, uy[:, 1:]], dim=1)
        return (self._full(ux, -ux[:, :1], s * ux[:, -1:]), self._full(uy, z, z),
                self._full(uz, -uz[:, :1], s * uz[:, -1:]))

    def neumann(self, F):
        return self._full(F, F[:, :1], F[:, -1:])

    def scal(self, c):
        return self._full(c, self.r1b * c[:, :1], c[:, -1:])

    def div(self, ux, uy, uz):
        """Of full arrays."""
        J = slice(1, -1)
        return self.X(ux[:, J], self.dx, -1) + (uy[:, 2:] - uy[:, J]) * self.rdyp + self.Z(uz[:, J], self.dz, -1)

    def poisson(self, src):
        nz, ny, nx = src.shape
        f = torch.fft.fft(torch.fft.rfft(src, dim=2), dim=0)
        am, ac, ap = self.ph
        x = torch.empty_like(f)
        arr = torch.empty((ny,) + self.lam.shape, device=DEV, dtype=F64)
        b = self.lam + float(ac[0])
        b[0, 0] = 1.0
        f[0, 0, 0] = 0.0
        x[:, 0] = f[:, 0] / b
        for j in range(1, ny):
            arr[j] = float(ap[j - 1]) / b
            if j == 1:
                arr[1, 0, 0] = 0.0
            b = self.lam + float(ac[j]) - float(am[j]) * arr[j]
            x[:, j] = (f[:, j] - float(am[j]) * x[:, j - 1]) / b
        for j in range(ny - 2, -1, -1):
            x[:, j] -= arr[j + 1] * x[:, j + 1]
        del f, arr
        return torch.fft.irfft(torch.fft.ifft(x, dim=0), n=nx, dim=2)

    def grad(self, phi):
        """Of a full array."""
        J = slice(1, -1)
        return self.X(phi[:, J], self.dx, -2), (phi[:, J] - phi[:, :-2]) * self.rdyc, self.Z(phi[:, J], self.dz, -2)

    def project(self, ux, uy, uz):
        f = self.vel(ux, uy, uz)
        gx, gy, gz = self.grad(self.neumann(self.poisson(self.div(*f))))
        uy = f[1][:, 1:-1] - gy
        uy[:, 0] = 0.0
        return f[0][:, 1:-1] - gx, uy, f[2][:, 1:-1] - gz

    def implicit(self, F, beta, co, first=False):
        """The solution of (I - beta L) x = F; first: row 1 is x = 0."""
        n = F.shape[1]
        am, ac, ap = co
        M = np.eye(n) - beta * (np.diag(ac) + np.diag(am[1:], -1) + np.diag(ap[:-1], 1))
        if first:
            M[0] = 0.0
            M[0, 0] = 1.0
            F = F.clone()
            F[:, 0] = 0.0
        R = F.permute(1, 0, 2).reshape(n, -1)
        S = torch.linalg.solve(torch.as_tensor(M, device=DEV, dtype=F64), R)
        return S.reshape(n, F.shape[0], F.shape[2]).permute(1, 0, 2)

    def explicit(self, U, V, W, P, C):
        """The explicit terms, -grad p and the wall-normal diffusion of full
        arrays: lists over u, v, w (, c)."""
        p, IC, dx, dz = self.p, self.IC, self.dx, self.dz
        J, JM, JP = slice(1, -1), slice(0, -2), slice(2, None)
        i1, i3 = self.iy1, self.iy3

        def lap(F):
            return self.X(F[:, J], self.dxx, -2) + self.Z(F[:, J], self.dzz, -2)

        def low(F):
            return i1 * F[:, JM] + (1 - i1) * F[:, J]

        def high(F):
            return i3 * F[:, J] + (1 - i3) * F[:, JP]

        vx, vz = self.X(V, IC, -2), self.Z(V, IC, -2)
        wx, uz = self.X(W[:, J], IC, -2), self.Z(U[:, J], IC, -2)
        ub, wb = self.X(U[:, J], IC, -1), self.Z(W[:, J], IC, -1)
        vx[:, -1] = 0.0
        vz[:, -1] = 0.0
        uw = uz * wx
        hu = self.X(ub * ub, dx, -2) + (vx[:, JP] * high(U) - vx[:, J] * low(U)) * self.rdyp + self.Z(uw, dz, -1)
        mid = (V[:, JP] + V[:, J]) ** 2 - (V[:, J] + V[:, JM]) ** 2
        hv = self.X(vx[:, J] * low(U), dx, -1) + 0.25 * mid * self.rdyc + self.Z(vz[:, J] * low(W), dz, -1)
        hw = self.X(uw, dx, -1) + (vz[:, JP] * high(W) - vz[:, J] * low(W)) * self.rdyp + self.Z(wb * wb, dz, -2)
        conv = [-hu + p.xnu * lap(U), -hv + p.xnu * lap(V), -hw + p.xnu * lap(W)]
        dyy = [self._yy(U, self.c), self._yy(V, self.v), self._yy(W, self.c)]
        if C is not None:
            fx, fy, fz = p.falling_vel_vec
            cx, cz = self.X(C[:, J], IC, -2), self.Z(C[:, J], IC, -2)
            g = p.gravity_eff_vec
            for q, t in enumerate((cx, low(C), cz)):
                conv[q] = conv[q] + g[q] * t
            hc = self.X((U[:, J] + fx) * cx, dx, -1) + self.Z((W[:, J] + fz) * cz, dz, -1) + \
                ((V[:, JP] + fy) * high(C) - (V[:, J] + fy) * low(C)) * self.rdyp
            conv.append(-hc + p.sdiff * lap(C))
            dyy.append(self._yy(C, self.s))
        total = (U[:, J] * self.dyp).sum() if C is not None else ((lap(U) + dyy[0]) * self.dyp).sum()
        return conv, [-t for t in self.grad(P)], dyy, float(total)

    def dt(self, U, V, W):
        p = self.p
        if p.icfl != 1:
            return p.dt_max
        J = slice(1, -1)
        a = (U[:, J] + torch.roll(U[:, J], -1, 2)).abs() * self.rdx + (V[:, J] + V[:, 2:]).abs() * self.rdyp + \
            (W[:, J] + torch.roll(W[:, J], -1, 0)).abs() * self.rdz
        return min(p.dt_max, p.cflc / max(0.5 * float(a.max()), 1e-300))

    GAM = {AB2: (1.5,), RK2: (0.5, 1.0), RK3: (8 / 15, 5 / 12, 3 / 4)}
    THE = {AB2: (-0.5,), RK2: (0.0, -0.5), RK3: (0.0, -17 / 60, -5 / 12)}

    def steps(self, fields, n):
        """u, v, w, p, c and the histories after n steps."""
        p = self.p
        ux, uy, uz, pr, c = fields
        nq = 4 if c is not None else 3
        hist = [torch.zeros_like(ux) for _ in range(nq)]
        for _ in range(n):
            dt = self.dt(*self.vel(ux, uy, uz))
            for gam, the in zip(self.GAM[p.ischeme], self.THE[p.ischeme]):
                U, V, W = self.vel(ux, uy, uz)
                C = None if c is None else self.scal(c)
                conv, gp, dyy, total = self.explicit(U, V, W, self.neumann(pr), C)
                a = (gam + the) * dt
                nu = [p.xnu] * 3 + ([p.sdiff] if nq > 3 else [])
                rhs = [gam * dt * conv[q] + the * dt * hist[q] + a * nu[q] * dyy[q] + (a * gp[q] if q < 3 else 0.0)
                       for q in range(nq)]
                hist = conv
                if p.is_ux_const:
                    mean = total / (p.nxc * p.nzc) / p.yly
                    rhs[0] = rhs[0] + ((gam + the) * (p.ubulk - mean) if c is not None else -a * p.xnu * mean)
                del conv, dyy, gp
                b = 0.5 * a * p.xnu
                U[:, 1:-1] += self.implicit(rhs[0], b, self.cn)
                V[:, 1:-1] += self.implicit(rhs[1], b, self.v, first=True)
                W[:, 1:-1] += self.implicit(rhs[2], b, self.cn)
                if c is not None:
                    c = c + self.implicit(rhs[3], 0.5 * a * p.sdiff, self.sn)
                phi = self.neumann(self.poisson(self.div(U, V, W) / a))
                gx, gy, gz = self.grad(phi)
                ux, uy, uz = U[:, 1:-1] - a * gx, V[:, 1:-1] - a * gy, W[:, 1:-1] - a * gz
                uy[:, 0] = 0.0
                pr = pr + phi[:, 1:-1] - b * self._yy(phi, self.ph)
        return [ux, uy, uz, pr, c] + hist

    def spectra(self, U, V, W, P, C, jlcs, dim):
        """The sums of clcStat's 1-D spectra along x (dim 2) or z (dim 0)."""
        p = self.p
        n = (p.nzc, p.nyc, p.nxc)[dim]
        J = slice(1, -1)
        ny = p.nyc
        row = np.arange(1, ny + 1)
        ref = np.where((row <= ny // 2) | (p.flow_type != FT_CH), jlcs, ny + 1 - jlcs)

        def ft(F):
            return torch.fft.rfft(F, dim=dim)

        u, v, w, q = ft(U[:, J]), ft(V[:, J]), ft(W[:, J]), ft(P)
        vc, uc = ft(0.5 * (V[:, J] + V[:, 2:])), ft(self.X(U[:, J], self.IC, -1))
        r = ft(U[:, 1:-1][:, torch.as_tensor(ref - 1, device=DEV)])
        wt = torch.full((n // 2 + 1,), 2.0, device=DEV, dtype=F64)
        wt[0] = wt[-1] = 1.0
        shp = [1, 1, 1]
        shp[dim] = -1
        wt = wt.reshape(shp)

        def ends(F):  # the two end modes keep their real parts only
            F = F.clone()
            for k in (0, n // 2):
                s = [slice(None)] * 3
                s[dim] = k
                F[tuple(s)] = F[tuple(s)].real.to(F.dtype)
            return F

        u, v, w, q, vc, uc, r = (ends(F) for F in (u, v, w, q, vc, uc, r))
        lcs = u * r.conj()
        im = lcs.imag.clone()
        for k in (0, n // 2):
            s = [slice(None)] * 3
            s[dim] = k
            im[tuple(s)] = 0.0
        parts = [wt * (F.real ** 2 + F.imag ** 2) for F in (u, v, w, q)] + \
            [wt * (u * vc.conj()).real, wt * (uc * vc.conj()).real, lcs.real, im]
        if C is not None:
            s = ends(ft(C))
            parts.append(wt * (s.real ** 2 + s.imag ** 2))
        norm = 1.0 / (float(n) * p.nxc * p.nzc)
        other = 0 if dim == 2 else 2
        out = [t.sum(dim=other) * norm for t in parts]  # [ny, modes] or [modes, ny]
        return torch.stack([t if dim == 2 else t.T for t in out])

    @staticmethod
    def visu(name, U):
        """dump_visu's ux at the cell centres (flat); None for the others."""
        if name != "ux":
            return None
        u = U[:, 1:-1]
        return (0.5 * (u + torch.roll(u, -1, 2))).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        ws = workloads.ensemble_c4(case["members"], case["seed_grids"])
        got = []
        for i, w in enumerate(ws):
            yp = _grid(w)
            got.append(_Torch(w.params, yp).steps(_initial(w.params, yp, seed + i), case["steps"])[:4])
        return [torch.cat([g[q].reshape(-1) for g in got]) for q in range(4)]
    if kind == "poisson":
        w = workloads.poisson_c2(case["nx"], case["ny"], case["nz"])
        return _Torch(w.params, _grid(w)).poisson(_source(case, seed))
    w = _workload(case)
    yp = _grid(w)
    m = _Torch(w.params, yp)
    f = _initial(w.params, yp, seed)
    if kind == "output":
        U, V, W = m.vel(*f[:3])
        sp = [m.spectra(U, V, W, f[3], f[4], max(1, case["ny"] // 8), dim) for dim in (2, 0)]
        # clcStat's 35 moments and Q have no short plain form here
        return [None] + sp + [m.visu(v, U) for v in VISU]
    return [t for t in m.steps(f, case["steps"]) if t is not None]
