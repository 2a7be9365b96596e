"""The lattice updates, ensembles and warm starts that a user of this package runs.

A pass is what a driver does between two write steps: a stretch of time steps
(or a fresh start from host fields, an ensemble's steps, a warm start) and
the read-back of the fields it writes, through ``Lattice``, ``Batch`` and
``warmstart.Network``.  Host fields live in pinned memory that the program
keeps.  FP64 runs return FP64 fields; the FP32-deviation form, whose results
are accurate to FP32, returns them as the FP32 values that a program of that
precision keeps (the field files hold FP32 as well).

``exact`` restates the model in plain torch FP64 on an explicit table of pull
sources: collide (MRT), stream, boundaries, density, heat source, temperature,
interaction force, velocity.
"""
import functools
import math
import os

import numpy as np
import torch

from multiphaselb_b200 import Batch, Lattice, abi, cases, warmstart

DEV = "cuda"

# --------------------------------------------------------------------- cases
# What each listed case stands for:
#   restart_64            one member of a parameter sweep on the smallest lattice of the ensemble: new
#                         fields from the host, start-up, steps, read-back; latency and launches count
#   bubble_256            the static D2Q9 bubble of the package's standard cases
#   column_128x512        the thermal column (liTempMRT heat, walls, gravity), the benchmark's workload
#   column_128x512_fp32   the same in the FP32-deviation form
#   column_1021x2039      a large column of odd extents, several waves of tiles, the myMRT heat model
#   column_1024x4096      the largest column of the size sweep
#   bubble_2048_fp32      a large D2Q9 lattice in the FP32-deviation form
#   bubble3d_192          the static D3Q15 bubble of the package's standard cases
#   bubble3d_192_fp32     the same in the FP32-deviation form
#   walls3d_97x61x83      a D3Q15 box of odd extents between walls, with gravity
#   cylinder_768x384      a mesh that is no box (a channel around a solid disc), one kernel per operator
#   ensemble_24           24 bubbles of uneven size advanced together
_LISTED = [
    dict(name="restart_64", kind="bubble", nx=64, ny=64, nz=1, precision="fp64", steps=200, restart=True),
    dict(name="bubble_256", kind="bubble", nx=256, ny=256, nz=1, precision="fp64", steps=200, restart=False),
    dict(name="column_128x512", kind="column", nx=128, ny=512, nz=1, precision="fp64", heat="liTempMRT", steps=200),
    dict(name="column_128x512_fp32", kind="column", nx=128, ny=512, nz=1, precision="fp32", heat="liTempMRT",
         steps=200),
    dict(name="column_1021x2039", kind="column", nx=1021, ny=2039, nz=1, precision="fp64", heat="myMRT", steps=50),
    dict(name="column_1024x4096", kind="column", nx=1024, ny=4096, nz=1, precision="fp64", heat="liTempMRT",
         steps=50),
    dict(name="bubble_2048_fp32", kind="bubble", nx=2048, ny=2048, nz=1, precision="fp32", steps=100, restart=False),
    dict(name="bubble3d_192", kind="bubble3d", nx=192, ny=192, nz=192, precision="fp64", steps=60),
    dict(name="bubble3d_192_fp32", kind="bubble3d", nx=192, ny=192, nz=192, precision="fp32", steps=60),
    dict(name="walls3d_97x61x83", kind="walls3d", nx=97, ny=61, nz=83, precision="fp64", steps=60),
    dict(name="cylinder_768x384", kind="cylinder", nx=768, ny=384, nz=1, precision="fp64", heat="liTempMRT",
         steps=60),
    dict(name="ensemble_24", kind="ensemble", lattices=24, pick=7, steps=100),
]


def listed():
    return [dict(c) for c in _LISTED]


def draw(rng):
    """One more case: kinds as often as they are used, extents log-uniform over
    each kind's range (multiples of 32 and odd values both), any precision."""
    def extent(lo, hi):
        v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return max(lo, min(hi, 32 * max(1, round(v / 32)) if rng.random() < 0.4 and v >= 48 else v))

    def steps(n):
        return int(max(20, min(200, 4e7 // n)))

    kind = rng.choice(["bubble", "bubble", "column", "column", "bubble3d", "bubble3d", "walls3d", "cylinder",
                       "ensemble", "warmstart"])
    precision = rng.choice(["fp64", "fp64", "fp32"])
    if kind == "bubble":
        nx, ny = extent(64, 2048), extent(64, 2048)
        return dict(kind=kind, nx=nx, ny=ny, nz=1, precision=precision, steps=steps(nx * ny),
                    restart=rng.random() < 0.3)
    if kind == "column":
        nx, ny = extent(32, 1024), extent(64, 4096)
        heat = "liTempMRT" if precision == "fp32" else rng.choice(["liTempMRT", "liTempMRT", "myMRT"])
        return dict(kind=kind, nx=nx, ny=ny, nz=1, precision=precision, heat=heat, steps=steps(nx * ny))
    if kind in ("bubble3d", "walls3d"):
        hi = 192 if kind == "bubble3d" else 128
        nx, ny, nz = extent(32, hi), extent(32, hi), extent(32, hi)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, steps=min(60, steps(nx * ny * nz)))
    if kind == "cylinder":
        nx, ny = extent(64, 1024), extent(64, 512)
        return dict(kind=kind, nx=nx, ny=ny, nz=1, precision="fp64", heat=rng.choice(["liTempMRT", "myMRT"]),
                    steps=min(60, steps(nx * ny)))
    if kind == "ensemble":
        return dict(kind=kind, lattices=rng.randint(6, 24), pick=rng.randint(1, 10 ** 6), steps=100)
    m = extent(48, 144)
    return dict(kind="warmstart", nx=m, ny=m, nz=m, precision="fp64", steps=20)


# ------------------------------------------------------------------- physics
CS = dict(type=abi.EOS_CS, a=1.0, b=4.0, R=1.0, G=-1.0, M=1.0, Cv=1.0, g=(0.0, 0.0, 0.0), fext=(0.0, 0.0, 0.0),
          rho_0=0.0)
# a = 9/392 keeps the pseudopotential real in the vapour (Tc = 1/14)
VDW = dict(type=abi.EOS_VDW, a=9.0 / 392.0, b=2.0 / 21.0, R=1.0, G=-1.0, M=1.0, Cv=1.0, g=(0.0, -1e-5, 0.0),
           fext=(0.0, 0.0, 0.0), rho_0=0.0)
CS_TC, VDW_TC = 0.0943287, 1.0 / 14.0
LAMBDA_LI = [1.0, 1.5, 1.4, 1.0, 1.2, 1.0, 1.2, 1.0, 1.0]
LAMBDA_XU = [1.0, 1.1, 1.1, 1.0, 1.1, 1.0, 1.1, 1.0, 1.1, 1.0, 1.0, 1.0, 1.0, 1.0, 1.2]
LAMBDA_TEMP = [1.0, 1.0, 1.0, 0.8, 1.0, 0.8, 1.0, 1.0, 1.0]
LAMBDA_MY = [0.0, 1.1, 1.1, 0.9, 1.0, 0.9, 1.0, 1.0, 1.0]
SIGMA = 0.125
ENSEMBLE_SIZES = (64, 96, 128, 192, 256, 384, 512)
V2 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]
V3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 1), (-1, 1, 1),
      (1, -1, 1), (-1, -1, 1), (1, 1, -1), (-1, 1, -1), (1, -1, -1), (-1, -1, -1)]


def _pressure(eos, rho, T):
    if eos["type"] == abi.EOS_CS:
        y = eos["b"] * rho / 4.0
        return rho * eos["R"] * T * (1 + y + y * y - y * y * y) / (1 - y) ** 3 - eos["a"] * rho * rho
    return rho * eos["R"] * T / (1 - eos["b"] * rho) - eos["a"] * rho * rho


@functools.lru_cache(maxsize=64)
def _coexistence(kind, T):
    """(vapour, liquid) densities by the equal-area rule on a fine grid of ln v."""
    eos = CS if kind == "cs" else VDW
    top = (4.0 if kind == "cs" else 1.0) / eos["b"]
    lnv = np.linspace(math.log(1.0 / (0.98 * top)), math.log(1e5), 200001)
    v = np.exp(lnv)
    p = _pressure(eos, 1.0 / v, T)
    dp = np.diff(p)
    i_lo = int(np.argmax(dp > 0))
    i_hi = i_lo + int(np.argmax(dp[i_lo:] < 0))
    lo, hi = max(p[i_lo], 0.0), p[i_hi]
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        i = int(np.argmax(p[:i_lo + 1] < mid))
        j = i_hi + int(np.argmax(p[i_hi:] < mid))
        area = float(np.sum((p[i:j] - mid) * v[i:j])) * (lnv[1] - lnv[0])
        lo, hi = (mid, hi) if area > 0 else (lo, mid)
    return 1.0 / v[j], 1.0 / v[i]


def _geometry(case):
    """(velocities, pull table [n][Q] on the GPU, points, patches): nodes in
    x-fastest order, sources at x - c, -1 where there is none."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kind = case["kind"]
    vel = V3 if kind in ("bubble3d", "walls3d", "warmstart") else V2
    per = {"column": (1, 0, 1), "cylinder": (1, 0, 1), "walls3d": (0, 1, 0)}.get(kind, (1, 1, 1))
    ids = torch.arange(nx * ny * nz, device=DEV)
    x, y, z = ids % nx, (ids // nx) % ny, ids // (nx * ny)
    index = None
    if kind == "cylinder":  # a disc of a sixth of the height, a third of the way along
        fluid = (x - 0.33 * nx) ** 2 + (y - 0.47 * ny) ** 2 >= (ny / 6.0) ** 2
        index = torch.where(fluid, torch.cumsum(fluid, 0) - 1, -1)
        x, y, z = x[fluid], y[fluid], z[fluid]
    nb = torch.empty((x.numel(), len(vel)), dtype=torch.int32, device=DEV)
    for k, c in enumerate(vel):
        s, ok = [], torch.ones_like(x, dtype=torch.bool)
        for v, d, ext, p in ((x, c[0], nx, per[0]), (y, c[1], ny, per[1]), (z, c[2], nz, per[2])):
            w = v - d
            if p:
                w = w % ext
            else:
                ok &= (w >= 0) & (w < ext)
                w = w.clamp(0, ext - 1)
            s.append(w)
        src = s[0] + nx * (s[1] + ny * s[2])
        if index is not None:
            src = index[src]
        nb[:, k] = torch.where(ok, src, -1).int()
    patches = []
    for v, ext, p in ((x, nx, per[0]), (y, ny, per[1]), (z, nz, per[2])):
        if not p:
            patches += [torch.nonzero(v == 0).flatten(), torch.nonzero(v == ext - 1).flatten()]
    if kind == "cylinder":
        wall = (y == 0) | (y == ny - 1)
        patches.append(torch.nonzero((nb == -1).any(1) & ~wall).flatten())
    return vel, nb, torch.stack([x, y, z], 1), patches


def _model(case):
    """EOS, flow and heat fields (the dicts that ``cases.Case`` takes)."""
    kind = case["kind"]
    walls = {"column": 2, "cylinder": 3, "walls3d": 4}.get(kind, 0)
    d3 = kind in ("bubble3d", "walls3d", "warmstart")
    f = dict(model=abi.XUMRT if d3 else abi.LIMRT, update=1, Lambda=LAMBDA_XU if d3 else LAMBDA_LI, sigma=SIGMA,
             bc_type=[abi.BC_BOUNCEBACK] * walls, bc_value=np.zeros((walls, 3)))
    if kind not in ("column", "cylinder"):
        return dict(CS, g=(0.0, 0.0, -1e-5)) if kind == "walls3d" else CS, f, None
    temps = [0.86, 0.84, 0.87][:walls]
    g = dict(model=abi.LITEMPMRT, update=1, Lambda=LAMBDA_TEMP)
    if case["heat"] == "myMRT":
        g = dict(model=abi.MYMRT, update=1, Lambda=LAMBDA_MY, alpha_1=1.0, alpha_2=-1.0)
    g.update(bc_type=[abi.BC_FIXEDT] * walls, bc_value=np.array([[t * VDW_TC, 0.0, 0.0] for t in temps]))
    return VDW, f, g


def _fields(case, seed, points):
    """Seeded initial rho, U, T (torch FP64): tanh bubble or liquid layer at the
    coexistence densities, a small random velocity, T noise where heat runs."""
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device=DEV).manual_seed(int(rng.integers(1 << 31)))
    p = points.double()
    n = p.shape[0]
    if case["kind"] in ("column", "cylinder"):
        T0 = 0.85 * VDW_TC
        rv, rl = _coexistence("vdw", T0)
        level = (0.4 + 0.02 * float(rng.uniform(-1, 1))) * case["ny"]
        rho = 0.5 * (rl + rv) + 0.5 * (rv - rl) * torch.tanh(2.0 * (p[:, 1] - level) / 4.0)
        T = T0 + 1e-4 * (2 * torch.rand(n, dtype=torch.float64, device=DEV, generator=gen) - 1)
    else:
        ratio = case.get("t_ratio", 0.75 if case["nz"] > 1 else 0.8)
        T0 = ratio * CS_TC
        rv, rl = _coexistence("cs", T0)
        ext = [e for e in (case["nx"], case["ny"], case["nz"]) if e > 1]
        R = case.get("radius", 0.2 * min(ext)) * (1 + 0.05 * float(rng.uniform(-1, 1)))
        r2 = sum((p[:, i] - ((e - 1) / 2.0 + float(rng.uniform(-1, 1)))) ** 2 for i, e in enumerate(ext))
        rho = 0.5 * (rv + rl) + 0.5 * (rl - rv) * torch.tanh(2.0 * (torch.sqrt(r2) - R) / 5.0)
        T = torch.full((n,), T0, dtype=torch.float64, device=DEV)
    U = torch.zeros((n, 3), dtype=torch.float64, device=DEV)
    D = 2 if case["nz"] == 1 else 3
    U[:, :D] = 1e-4 * (2 * torch.rand((n, D), dtype=torch.float64, device=DEV, generator=gen) - 1)
    return rho, U, T


def _members(case):
    """The ensemble's lattices: sizes, temperatures and radii drawn as the
    package's ensemble draws them."""
    rng = np.random.Generator(np.random.PCG64(case["pick"]))
    out = []
    for _ in range(case["lattices"]):
        L = int(rng.choice(np.array(ENSEMBLE_SIZES)))
        out.append(dict(kind="bubble", nx=L, ny=L, nz=1, precision="fp32", t_ratio=float(rng.uniform(0.7, 0.9)),
                        radius=float(rng.uniform(8.0, 0.3 * L))))
    return out


# ------------------------------------------------------------------ the user
@functools.lru_cache(maxsize=8)
def _mesh(kind, nx, ny, nz):
    """A mesh as the program has read it (host arrays); several lattices may share one."""
    _, nb, points, patches = _geometry(dict(kind=kind, nx=nx, ny=ny, nz=nz))
    return (nb.cpu().numpy(), points.int().cpu().numpy(), [q.cpu().numpy().astype(np.uint32) for q in patches])


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _lattice(case, seed):
    nb, points, patches = _mesh(case["kind"], case["nx"], case["ny"], case["nz"])
    eos, f, g = _model(case)
    rho, U, T = _fields(case, seed, torch.from_numpy(points).to(DEV))
    host = {k: _pinned(v.shape) for k, v in (("rho", rho), ("U", U), ("T", T))}
    for k, v in (("rho", rho), ("U", U), ("T", T)):
        host[k].copy_(v)
    d3 = case["nz"] > 1
    dims = (case["nx"], case["ny"], case["nz"]) if d3 else (case["nx"], case["ny"])
    c = cases.Case(case["kind"], abi.D3Q15 if d3 else abi.D2Q9, dims, (False,) * len(dims), nb, points, patches,
                   ["patch%d" % i for i in range(len(patches))], eos, f, g, host["rho"].numpy(), host["U"].numpy(),
                   host["T"].numpy())
    lat = Lattice(c, precision=abi.FP32_DEV if case["precision"] == "fp32" else abi.FP64)
    lat.upload_case()
    lat.initialize()
    names = ("rho", "U") if g is None else ("rho", "U", "T")
    out = {k: _pinned(host[k].shape) for k in names}
    kept = {k: torch.empty(v.shape, dtype=torch.float32) for k, v in out.items()} if case["precision"] == "fp32" \
        else out
    return dict(lat=lat, case=c, out=out, numpy={k: v.numpy() for k, v in out.items()}, kept=kept)


def _weights(dim):
    return os.path.join(os.path.dirname(warmstart.__file__), "data", "warmstart_d%s.npz" % dim)


def prepare(case, seed):
    if case["kind"] == "ensemble":
        members = [_lattice(m, seed + 1000 * i) for i, m in enumerate(_members(case))]
        return dict(run=_run_ensemble, members=members, batch=Batch([m["lat"] for m in members]),
                    steps=case["steps"])
    s = _lattice(case, seed)
    s["steps"] = case["steps"]
    s["run"] = _run_restart if case.get("restart") else _run_steps
    if case["kind"] == "warmstart":
        rng = np.random.Generator(np.random.PCG64(seed))
        s["net"] = warmstart.Network.load(_weights("3q15"))
        s["bubble"] = _warm(case, rng)
        s["run"] = _run_warmstart
    torch.cuda.synchronize()
    return s


def _warm(case, rng):
    """T/Tc, centre, radius and T of a warm-started bubble."""
    ratio = float(rng.uniform(0.7, 0.9))
    centre = [(case["nx"] - 1) / 2.0] * 3
    return ratio, centre, float(rng.uniform(0.12, 0.28)) * case["nx"], ratio * CS_TC


def _read(s):
    s["lat"].download(s["numpy"])
    if s["kept"] is not s["out"]:
        for k, v in s["out"].items():
            s["kept"][k].copy_(v)
    return s["kept"]


def _run_steps(s):
    s["lat"].step(s["steps"])
    return _read(s)


def _run_restart(s):
    s["lat"].upload_case()
    s["lat"].initialize()
    return _run_steps(s)


def _run_warmstart(s):
    s["net"].init_bubble(s["lat"], *s["bubble"])
    s["lat"].initialize()
    return _run_steps(s)


def _run_ensemble(s):
    s["batch"].step(s["steps"])
    return [_read(m) for m in s["members"]]


def run(state):
    return state["run"](state)


def work(case):
    """Per step: every population read once and written once, and of the fields
    those that the next step cannot rebuild (T, U and the heat source where heat
    runs, T where it does not); then the fields read back."""
    if case["kind"] == "ensemble":
        parts = [work(dict(m, steps=case["steps"])) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "cylinder":
        n -= int(math.pi * (case["ny"] / 6.0) ** 2)
    q = 15 if case["nz"] > 1 else 9
    heat = case["kind"] in ("column", "cylinder")
    size = 4 if case["precision"] == "fp32" else 8
    per_step = 2 * q * size * (2 if heat else 1) + (8 * 8 if heat else 8)
    flops = (650 if q == 15 else 330) + (230 if heat else 0)
    return {"bytes": float(n) * (case["steps"] * per_step + (40 if heat else 32)),
            "flops": float(n) * case["steps"] * flops}


# ------------------------------------------------------- the model in 64 bits
def _moments(vel):
    """Rows of the MRT basis on the velocity set (Lallemand-Luo, d'Humieres)."""
    c = np.array(vel, dtype=np.float64)
    x, y, z = c[:, 0], c[:, 1], c[:, 2]
    s = x * x + y * y + z * z
    if len(vel) == 9:
        rows = [x * 0 + 1, 3 * s - 4, (9 * s * s - 21 * s + 8) / 2, x, (3 * s - 5) * x, y, (3 * s - 5) * y,
                x * x - y * y, x * y]
    else:
        rows = [x * 0 + 1, s - 2, (15 * s * s - 55 * s + 32) / 2, x, (5 * s - 13) * x / 2, y, (5 * s - 13) * y / 2,
                z, (5 * s - 13) * z / 2, 3 * x * x - s, y * y - z * z, x * y, y * z, x * z, x * y * z]
    return torch.tensor(np.stack(rows), dtype=torch.float64, device=DEV)


class _Exact:
    """The model's state and one time step on it, [Q][n] torch FP64."""

    def __init__(self, case, rho, U, T):
        self.vel, nb, _, self.patches = _geometry(case)
        self.eos, self.ff, self.gf = _model(case)
        q = self.q = len(self.vel)
        self.D = 2 if q == 9 else 3
        nb = nb.t().long()
        here = torch.arange(nb.shape[1], device=DEV)
        self.miss = nb < 0
        self.src = torch.where(self.miss, here, nb)
        self.rev = [self.vel.index(tuple(-a for a in c)) for c in self.vel]
        self.onb = self.miss.any(0)
        c2 = [sum(a * a for a in c) for c in self.vel]
        self.w = [(4 / 9, 1 / 9, 1 / 36)[v] if q == 9 else {0: 2 / 9, 1: 1 / 9, 3: 1 / 72}[v] for v in c2]
        self.ppw = [(0, 1 / 3, 1 / 12)[v] if q == 9 else {0: 0.0, 1: 1 / 3, 3: 1 / 24}[v] for v in c2]
        self.M = _moments(self.vel)
        self.Mi = (self.M / (self.M * self.M).sum(1, keepdim=True)).t().contiguous()
        self.C = torch.tensor(self.vel, dtype=torch.float64, device=DEV)
        self.grav = torch.tensor(self.eos["g"], dtype=torch.float64, device=DEV)[:, None]
        self.rho, self.T, self.U = rho, T, U.t().contiguous()
        cu = self.C @ self.U
        self.f = self.rho * torch.tensor(self.w, dtype=torch.float64, device=DEV)[:, None] * \
            (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (self.U * self.U).sum(0))
        self._force()
        if self.gf:
            self.g = self._heat_eq(self.T, self.U)
            self.S = self._source(None)

    def _at(self, v, k):
        return v[..., self.src[k]]

    def _psi(self, rho, T):
        return torch.sqrt(2 * (_pressure(self.eos, rho, T) - rho / 3) / self.eos["G"])

    def _force(self):
        self.psi = self._psi(self.rho, self.T)
        F = torch.zeros_like(self.U)
        for k in range(1, self.q):  # psi at x + c_k
            F += self.C[k][:, None] * (self.ppw[k] * self._at(self.psi, self.rev[k]))
        self.Fi = torch.where(self.onb, 0.0, F * (-self.eos["G"] * self.psi))
        self.Ft = self.Fi + self.rho * self.grav

    def _heat_moments(self, T, U):
        z = torch.zeros_like(T)
        a1, a2 = (self.gf["alpha_1"], self.gf["alpha_2"]) if self.gf["model"] == abi.MYMRT else (-2.0, 2.0)
        return torch.stack([T, a1 * T, a2 * T, T * U[0], -T * U[0], T * U[1], -T * U[1], z, z])

    def _heat_eq(self, T, U):
        return self.Mi @ self._heat_moments(T, U)

    def _source(self, old):
        """Heat source from rho (new), T and U (of the step before)."""
        gT, gR, div, inv = [], [], 0.0, 1.0 / self.rho
        for d in range(self.D):
            up = self.vel.index(tuple(-int(i == d) for i in range(3)))  # its source is x + e_d
            dn = self.rev[up]
            two = ~self.miss[up] & ~self.miss[dn]

            def slope(v):
                return (self._at(v, up) - self._at(v, dn)) * torch.where(two, 0.5, 1.0)
            gT.append(slope(self.T))
            gR.append(slope(inv))
            div = div + slope(self.U[d])
        dot = sum(a * b for a, b in zip(gT, gR))
        L, Cv, T, rho = self.gf["Lambda"], self.eos["Cv"], self.T, self.rho
        lam = rho * Cv * (1 / L[3] - 0.5)
        if self.gf["model"] == abi.MYMRT:
            lam = lam * (4 + 3 * self.gf["alpha_1"] + 2 * self.gf["alpha_2"]) / 6
        dpdT = (_pressure(self.eos, rho, 1.1 * T) - _pressure(self.eos, rho, 0.9 * T)) / (0.2 * T)
        s = -lam * dot / Cv + div * T * (1 - dpdT / (rho * Cv))
        if self.gf["model"] == abi.MYMRT:
            return s
        return s + 0.5 * (s - (0.0 if old is None else old))

    def _bounce(self, f, ids):
        for k in range(self.q):
            r = self.rev[k]
            v, o = f[k][ids], f[r][ids]
            both = ~self.miss[k][ids] & ~self.miss[r][ids]
            if sum(map(abs, self.vel[k])) == 1:
                m = 0.5 * v + 0.5 * o
                f[r][ids] = torch.where(both, m, o)
                v = torch.where(both, m, v)
            f[k][ids] = torch.where(self.miss[k][ids], o, v)

    def _fixed(self, ids, Tw):
        for k in range(self.q):
            ok = self.miss[k][ids] & ~self.miss[self.rev[k]][ids]
            at = ids[ok]
            nbr = self.src[self.rev[k]][at]
            U, T = self.U[:, nbr], self.T[nbr]
            self.g[k][at] = (self.Mi[k] @ self._heat_moments(torch.full_like(T, Tw), U)) + \
                (self.g[k][nbr] - self.Mi[k] @ self._heat_moments(T, U))

    def _stream(self, f):
        return torch.stack([f[k][self.src[k]] for k in range(self.q)])

    def step(self):
        rho, U, psi = self.rho, self.U, self.psi
        L = torch.tensor(self.ff["Lambda"], dtype=torch.float64, device=DEV)[:, None]
        u2, z = (U * U).sum(0), torch.zeros_like(rho)
        m = self.M @ self.f
        if self.q == 9:
            F, f2 = self.Ft, (self.Fi[:2] ** 2).sum(0)
            uf = U[0] * F[0] + U[1] * F[1]
            e = 12 * SIGMA * f2 / (psi * psi)
            meq = torch.stack([rho, rho * (-2 + 3 * u2), rho * (1 - 3 * u2), rho * U[0], -rho * U[0], rho * U[1],
                               -rho * U[1], rho * (U[0] ** 2 - U[1] ** 2), rho * U[0] * U[1]])
            S = torch.stack([z, 6 * uf + e / (1 / self.ff["Lambda"][1] - 0.5),
                             -6 * uf - e / (1 / self.ff["Lambda"][2] - 0.5), F[0], -F[0], F[1], -F[1],
                             2 * (U[0] * F[0] - U[1] * F[1]), U[0] * F[1] + U[1] * F[0]])
        else:
            F = self.Fi + rho * self.grav
            uf, f2 = (U * F).sum(0), (F * F).sum(0)
            j = 7.0 / 3.0
            meq = torch.stack([rho, rho * (u2 - 1), rho * (1 - 5 * u2), rho * U[0], -j * rho * U[0], rho * U[1],
                               -j * rho * U[1], rho * U[2], -j * rho * U[2],
                               rho * (2 * U[0] ** 2 - U[1] ** 2 - U[2] ** 2), rho * (U[1] ** 2 - U[2] ** 2),
                               rho * U[0] * U[1], rho * U[1] * U[2], rho * U[0] * U[2], z])
            S = torch.stack([z, 2 * uf + 6 * SIGMA * f2 / (psi * psi * (1 / self.ff["Lambda"][1] - 0.5)), -10 * uf,
                             F[0], -j * F[0], F[1], -j * F[1], F[2], -j * F[2],
                             4 * U[0] * F[0] - 2 * U[1] * F[1] - 2 * U[2] * F[2],
                             2 * U[1] * F[1] - 2 * U[2] * F[2], U[0] * F[1] + U[1] * F[0],
                             U[1] * F[2] + U[2] * F[1], U[0] * F[2] + U[2] * F[0], z])
        self.f = self._stream(self.Mi @ (m - L * (m - meq) + (1 - 0.5 * L) * S))
        for ids in self.patches:
            self._bounce(self.f, ids)
        if self.gf:
            lam = self.gf["Lambda"]
            n, eq = self.M @ self.g, self._heat_moments(self.T, U)
            out = n - torch.tensor(lam, dtype=torch.float64, device=DEV)[:, None] * (n - eq)
            if self.gf["model"] == abi.MYMRT:
                out[3] -= lam[4] * (lam[3] / 2 - 1) * (n[4] - eq[4])
                out[5] -= lam[6] * (lam[5] / 2 - 1) * (n[6] - eq[6])
                out[0] += (1 - 0.5 * lam[0]) * self.S
            else:
                out[0] += self.S
                out[3] += (1 - lam[3] / 2) * lam[4] * n[4]
                out[5] += (1 - lam[5] / 2) * lam[6] * n[6]
            self.g = self._stream(self.Mi @ out)
            for ids, val in zip(self.patches, self.gf["bc_value"]):
                self._fixed(ids, float(val[0]))
        self.rho = self.f.sum(0)
        if self.gf:
            self.S = self._source(self.S)
            self.T = self.g.sum(0)
            if self.gf["model"] == abi.MYMRT:
                self.T = self.T + 0.5 * self.S
        self._force()
        F = self.Ft if self.q == 9 else self.Fi + self.rho * self.grav
        self.U = (self.C.t() @ self.f + 0.5 * F) / self.rho

    def out(self):
        o = dict(rho=self.rho, U=self.U.t().contiguous())
        return dict(o, T=self.T) if self.gf else o


def _network(case, seed, points):
    """The warm-start network's density: BF16 weights, inputs and activations,
    as the network is defined, everything else in 64 bits."""
    def bf16(v):
        return v.float().bfloat16().double()

    ratio, centre, R, T = _warm(case, np.random.Generator(np.random.PCG64(seed)))
    p = torch.tensor(np.load(_weights("3q15"))["params"], dtype=torch.float64, device=DEV)
    shapes = [(64, 5), (64,), (64, 64), (64,), (64, 64), (64,), (1, 64), (1,)]
    w = [t.reshape(s) for t, s in zip(torch.split(p, [int(np.prod(s)) for s in shapes]), shapes)]
    w = [bf16(t) if t.dim() == 2 else t for t in w]
    r = torch.sqrt(sum((points[:, i] - centre[i]) ** 2 for i in range(3)).double())
    one = torch.ones_like(r)
    h = bf16(torch.stack([one * (ratio - 0.775) / 0.175, one * (CS["a"] - 1), one * (CS["b"] / 4 - 1),
                          ((r - R) / 5.0).clamp(-6, 6) / 6, one * (5.0 / R - 0.3) / 0.3], 1))
    for i in range(0, 6, 2):
        h = bf16(torch.tanh(h @ w[i].t() + w[i + 1]))
    return (h @ w[6].t() + w[7]).flatten() / CS["b"], torch.zeros((r.numel(), 3), dtype=torch.float64, device=DEV), \
        torch.full_like(r, T)


def _exact_lattice(case, seed, steps):
    points = _geometry(case)[2]
    start = _network(case, seed, points) if case["kind"] == "warmstart" else _fields(case, seed, points)
    e = _Exact(case, *start)
    for _ in range(steps):
        e.step()
    if case["kind"] == "warmstart":  # U is the flow that the network's BF16 noise in rho sets off
        return dict(e.out(), U=None)
    return e.out()


def exact(case, seed):
    if case["kind"] == "ensemble":
        return [_exact_lattice(m, seed + 1000 * i, case["steps"]) for i, m in enumerate(_members(case))]
    return _exact_lattice(case, seed, case["steps"])
