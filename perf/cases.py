"""The work that users of this library have it do, as measurable cases.

Every case goes through the public entry points: `Tank` (one grid),
`Batch` (several grids solved together), `vf_step_gpu_` (the call the
Fortran time loop makes), `m1bcgs_dev` (the pressure solver on device
arrays) and `UNet` (the learned initial guess, forward and training).

A pass of a simulation is one output interval of a run: the state goes in
(cadmas_set_state, as after a restart), a few SMAC steps, and the whole state
comes out (cadmas_get_state).  Every pass starts from the same state, so a
pass costs the same however often it is repeated.

Another seed is another wave or flow on the same grid: the velocities of the
initial state scaled and disturbed, the droplets moving otherwise, another
right-hand side, other network inputs and weights.  The grids' own seeds are
part of the case.
"""
import ctypes
import functools
import importlib
import math

import numpy as np
import torch

P = importlib.import_module("multiscale-and-multiphysics-integrated-simulator-for-tsunami_b200")
warmstart = importlib.import_module(P.__name__ + ".warmstart")

REALS = ("uu", "vv", "ww", "pp", "ff")       # per cell, FP64
INTS = ("nf", "indc")                        # per cell, 32-bit
FACES = ("bcu", "bcv", "bcw", "bcp", "bcf")  # per boundary face, FP64


def listed():
    return [
        # The smallest run: the 64x8x32 dam break that the long-run test takes
        # 2000 steps through; latency and launches, one preconditioner block.
        dict(name="dam_break", kind="tank", what="dam", nx=64, ny=8, nz=32, ti=0, tj=0, solver=0, tol=1e-10, steps=4),
        # The turbulent tanks of the parity tests, grown: k-epsilon, FF-SLOPE,
        # log-law and rough walls, obstacles and porous blocks, uneven spacing,
        # odd sizes (ragged tiles), the default tolerance.
        dict(name="turbulent_tank", kind="tank", what="keps", nx=93, ny=21, nz=43, ti=16, tj=8, solver=0, tol=1e-12, steps=4),
        # Droplets in flight over a pool (the TimerDoor model), with the
        # adaptive time step asked for at every step, odd sizes.
        dict(name="droplets", kind="tank", what="drop", nx=97, ny=21, nz=45, ti=16, tj=8, solver=0, tol=1e-12, steps=4),
        # The 512x32x96 porous flume with its wave maker and sponge, FP64, in
        # the blocks its benchmark takes.
        dict(name="flume_fp64", kind="tank", what="flume", nx=512, ny=32, nz=96, ti=8, tj=16, solver=0, tol=1e-10, steps=2),
        # The same flume driven by the Fortran time loop: the whole state in and
        # out at every step, mixed solver, previous step's solution as the guess.
        dict(name="flume_mixed_host", kind="host", what="flume", nx=512, ny=32, nz=96, ti=16, tj=16, solver=1, tol=1e-10, steps=2),
        # A beach of odd size: ragged tiles on both sides, FP64.
        dict(name="beach_ragged_fp64", kind="tank", what="beach", nx=517, ny=61, nz=83, ti=16, tj=16, solver=0, tol=1e-8, steps=2),
        # The 1024x128x128 solitary-wave beach of the benchmark: the FP64 solver
        # and the mixed solver from the previous step's solution.
        dict(name="beach_fp64", kind="tank", what="beach", nx=1024, ny=128, nz=128, ti=16, tj=16, solver=0, tol=1e-8, steps=3),
        dict(name="beach_mixed", kind="tank", what="beach", nx=1024, ny=128, nz=128, ti=16, tj=16, solver=1, tol=1e-8, steps=5),
        # An ensemble of eight flumes of uneven size as one batch.
        dict(name="ensemble_batch", kind="batch", members=8, gseed=0, scale=0.5, ti=16, tj=16, solver=1, tol=1e-10, steps=2),
        # The pressure solver alone on a system that lies on the device, a mid
        # size with ragged tiles, the default tolerance.
        dict(name="solver_device", kind="solver", nx=250, ny=60, nz=70, ti=16, tj=16, tol=1e-12),
        # The learned guess: the network's forward on a 128x32x64 beach's
        # volume, and a training step on four samples of it.
        dict(name="unet_forward", kind="unet", X=132, Y=36, Z=68, batch=1),
        dict(name="unet_train", kind="train", X=132, Y=36, Z=68, batch=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dam", "keps", "drop", "flume", "flume", "beach", "beach", "batch", "solver", "unet", "train"])
    ti, tj = rng.choice([(16, 16), (16, 16), (8, 16), (16, 8), (32, 8)])
    if kind == "dam":  # up to 1024 columns: the serial factorisation, one block
        nx = _log(rng, 24, 100)
        return dict(kind="tank", what="dam", nx=nx, ny=rng.randint(3, min(16, 900 // (4 * -(-nx // 4)))), nz=rng.randint(20, 64),
                    ti=0, tj=0, solver=rng.choice([0, 1]), tol=1e-10, steps=rng.randint(1, 6))
    if kind in ("keps", "drop"):
        return dict(kind="tank", what=kind, nx=_log(rng, 40, 200), ny=rng.randint(9, 40), nz=rng.randint(24, 60), ti=ti,
                    tj=min(tj, 8), solver=0, tol=1e-12, steps=rng.randint(1, 5))
    if kind == "flume":
        return dict(kind=rng.choice(["tank", "host"]), what="flume", nx=_log(rng, 128, 768), ny=_log(rng, 8, 64),
                    nz=rng.randint(64, 110), ti=ti, tj=tj, solver=rng.choice([0, 1]), tol=1e-10, steps=rng.randint(1, 3))
    if kind == "beach":
        return dict(kind="tank", what="beach", nx=_log(rng, 256, 1024), ny=_log(rng, 16, 128), nz=rng.randint(80, 128),
                    ti=16, tj=16, solver=rng.choice([0, 1]), tol=1e-8, steps=rng.randint(1, 3))
    if kind == "batch":
        return dict(kind="batch", members=rng.randint(2, 10), gseed=rng.randint(1, 1000), scale=round(rng.uniform(0.2, 0.6), 2),
                    ti=ti, tj=tj, solver=1, tol=1e-10, steps=rng.randint(1, 2))
    if kind == "solver":
        return dict(kind="solver", nx=_log(rng, 40, 500), ny=_log(rng, 8, 100), nz=rng.randint(16, 110), ti=ti, tj=tj, tol=1e-12)
    X, Y, Z = 4 * _log(rng, 4, 48), 4 * _log(rng, 2, 12), 4 * rng.randint(4, 20)
    return dict(kind=kind, X=X, Y=Y, Z=Z, batch=1 if kind == "unet" else rng.randint(1, min(4, 1 + 600000 // (X * Y * Z))))


# ------------------------------------------------------------ simulations
@functools.lru_cache(maxsize=4)
def _grids(what, nx, ny, nz, members, gseed, scale):
    """The grids of a case with their undisturbed initial state."""
    C = P.cases
    if what == "batch":
        return C.ensemble_flumes(members, seed=gseed, scale=scale)
    if what == "dam":
        c = C.dam_break(nx=nx, ny=ny, nz=nz, column=(max(4, nx // 4), nz // 2))
    elif what == "keps":
        c = C.loglaw_tank(3, turb=True, nx=nx, ny=ny, nz=nz)
    elif what == "drop":
        c = C.droplet_tank(0, nx=nx, ny=ny, nz=nz, ndrop=max(8, nx * ny // 50))
    elif what == "flume":
        x0 = 0.6 * nx * 0.02
        c = C.porous_flume(nx=nx, ny=ny, nz=nz, block=(x0, x0 + 0.1 * nx * 0.02, 0.6), sponge_width=min(2.0, 0.2 * nx * 0.02))
        C.wave_maker(c, 0.08, 1.5, 0.5, stream=1)
        C.linear_wave_initial(c, 0.08, 1.5, 0.5, phase0=c.wave["stream"].phase0)
    else:
        c = C.solitary_beach(nx=nx, ny=ny, nz=nz, x_toe=0.5 * nx * 0.02, x0=0.25 * nx * 0.02)
    return [c]


def _grids_of(case):
    what = "batch" if case["kind"] == "batch" else case["what"]
    return _grids(what, case.get("nx", 0), case.get("ny", 0), case.get("nz", 0), case.get("members", 0),
                  case.get("gseed", 0), case.get("scale", 0.0))


class _Buffers:
    """A state's arrays in pinned host memory, as cadmas_state points to them."""

    def __init__(self, c):
        n, nb = c.ni * c.nj * c.nk, max(c.numb, 1)
        self.real = torch.zeros(len(REALS) * n, dtype=torch.float64, pin_memory=True)
        self.int = torch.zeros(len(INTS) * n, dtype=torch.int32, pin_memory=True)
        self.face = torch.zeros(len(FACES) * nb + c.nk, dtype=torch.float64, pin_memory=True)
        self.views = {f: self.real[i * n:(i + 1) * n] for i, f in enumerate(REALS)}
        self.views |= {f: self.int[i * n:(i + 1) * n] for i, f in enumerate(INTS)}
        self.views |= {f: self.face[i * nb:(i + 1) * nb] for i, f in enumerate(FACES)}
        self.views["tbub"] = self.face[len(FACES) * nb:]
        self.arrays = {k: v.numpy() for k, v in self.views.items()}
        self.struct = P.state_struct(self.arrays)

    def copy_from(self, o):
        self.real.copy_(o.real)
        self.int.copy_(o.int)
        self.face.copy_(o.face)
        self.struct.tnow, self.struct.nnow = o.struct.tnow, o.struct.nnow


class _Run:
    """One grid: its tank, the state its passes start from, and the state they end with."""

    def __init__(self, c, case, rng):
        over = dict(cgepsr=case["tol"], precond_ti=case["ti"], precond_tj=case["tj"], solver=case["solver"],
                    warm_start=case["solver"], mixed_eps_inner=1e-2)
        if case.get("what") == "keps":
            over["iscmff"] = 1
        self.case, self.tank = c, P.Tank(c, **over)
        st = P.initial_state(c)
        scale = rng.uniform(0.9, 1.1)
        amp = 1e-3 * rng.uniform(0.5, 1.0)
        ph = rng.uniform(0.0, 2.0 * np.pi, 3)
        x = np.arange(c.ni)[:, None, None] * (2 * np.pi / 37.0) + ph[0]
        y = np.arange(c.nj)[None, :, None] * (2 * np.pi / 23.0) + ph[1]
        z = np.arange(c.nk)[None, None, :] * (2 * np.pi / 31.0) + ph[2]
        wet = np.zeros(st["ff"].shape, order="F")
        wet[2:-1, 2:-1, 2:-1] = c.ff[2:-1, 2:-1, 2:-1] > 0.0
        for axis in range(3):  # faces between two cells that hold water
            wet[...] *= np.roll(c.ff > 0.0, 1, axis) & np.roll(c.nf != -1, 1, axis)
        for f, s, a in (("uu", np.sin(x), 0), ("vv", np.sin(y), 1), ("ww", np.sin(z), 2)):
            st[f] *= scale
            st[f] += amp * wet * s
        self.drop = None
        if getattr(c, "drop_state", None) is not None:
            self.drop = dict(c.drop_state)
            for f in ("dropuu", "dropvv", "dropww"):
                self.drop[f] = self.drop[f] * rng.uniform(0.5, 1.0)
        self.tank.set_state(st)
        self.tank.init_state(c.hydrostatic)
        self.turb = self.tank.get_turb() if c.params.get("leqk") else None
        self.start, self.end = _Buffers(c), _Buffers(c)
        self.get(self.start)

    def get(self, b):
        P._check(self.tank.lib, self.tank.lib.cadmas_get_state(self.tank.h, ctypes.byref(b.struct)))

    def put(self):
        P._check(self.tank.lib, self.tank.lib.cadmas_set_state(self.tank.h, ctypes.byref(self.start.struct)))
        if self.drop is not None:
            self.tank.set_drop(self.drop)
        if self.turb is not None:
            self.tank.set_turb(self.turb)

    def outputs(self):
        self.get(self.end)
        out = dict(self.end.views, fsum=self.tank.stats()["fsum"])
        if self.drop is not None:
            out.update(self.tank.get_drop())
        if self.turb is not None:
            out.update(self.tank.get_turb())
        return out

    def host_step(self):
        """One step of the Fortran time loop: VF_V1CAL and VF_F1CAL on host arrays."""
        a, t = self.end.arrays, self.tank
        dp, ip = (lambda n: P._dptr(a[n])), (lambda n: P._iptr(a[n]))
        dt, tnow, nnow = ctypes.c_double(self.case.dt), ctypes.c_double(self.end.struct.tnow), ctypes.c_int(self.end.struct.nnow)
        P._check(t.lib, t.lib.vf_step_gpu_(ctypes.byref(t.h), ctypes.byref(dt), dp("uu"), dp("vv"), dp("ww"), dp("pp"), dp("ff"),
                                           ip("nf"), ip("indc"), dp("bcu"), dp("bcv"), dp("bcw"), dp("bcp"), dp("bcf"),
                                           ctypes.byref(tnow), ctypes.byref(nnow)))
        self.end.struct.tnow, self.end.struct.nnow = tnow.value, nnow.value


# ---------------------------------------------------- the solver on its own
def _system(case, seed, device):
    """A pressure system on the device, arrays of (nk, nj, ni) in the layout's
    order: face conductances of a porous medium (0.3..1), walls around it, a
    free surface (Dirichlet) on top of the water, gas cells above it that are
    not computed (INDC = -1), and solid boxes; a right-hand side without a
    pattern."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    ni, nj, nk = case["nx"] + 2, case["ny"] + 2, case["nz"] + 2
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64).to(device)
    k = torch.arange(nk, device=device)[:, None, None]
    i = torch.arange(ni, device=device)[None, None, :]
    top = (0.7 * nk + 0.05 * nk * torch.cos(2 * np.pi * i / ni * 3 + float(torch.rand(1, generator=g)) * 6)).floor()
    live = torch.zeros(nk, nj, ni, dtype=torch.bool, device=device)
    live[1:-1, 1:-1, 1:-1] = True
    live &= k <= top
    live[1:nk // 5, nj // 3:nj // 2, ni // 2:ni // 2 + ni // 8] = False  # a solid box on the bed
    por = 0.3 + 0.7 * rnd(nk, nj, ni)
    low, up = [], []  # along i, j, k
    ad = torch.zeros(nk, nj, ni, dtype=torch.float64, device=device)
    for dim, w in ((2, 1.0), (1, 1.0), (0, 4.0)):
        f = w * torch.minimum(por, por.roll(1, dim)) * (live & live.roll(1, dim))  # face to the lower neighbour
        low.append(-f)
        up.append(-f.roll(-1, dim))
        ad += f + f.roll(-1, dim)
    surf = live & ~live.roll(-1, 0) & (k >= top - 1)
    ad += surf * 8.0 * por
    ad = torch.where(live, ad, torch.ones_like(ad))
    b = torch.where(live, rnd(nk, nj, ni) - 0.5, torch.zeros_like(ad))
    indc = torch.where(live, 0, -1).to(torch.int32)
    return [ad, *low, *up, b], indc, live


def _solver_tank(case):
    c = P.cases.dam_break(nx=case["nx"], ny=case["ny"], nz=case["nz"], column=(case["nx"] // 4, case["nz"] // 2))
    return P.Tank(c, precond_ti=case["ti"], precond_tj=case["tj"], cgepsr=case["tol"])


# ------------------------------------------------------------- the network
def _volumes(case, seed):
    """(parameters, x, t, m, a7): the features, targets, masks and systems of
    water under a free surface, FP32 host arrays as the training collects them."""
    rng = np.random.default_rng(seed)
    B, X, Y, Z = case["batch"], case["X"], case["Y"], case["Z"]
    lvl = 0.6 * Z + 0.1 * Z * np.cos(2 * np.pi * np.arange(X) / X * 3 + rng.uniform(0, 6, (B, 1)))
    f = np.clip(lvl[:, None, None, :] - np.arange(Z)[None, :, None, None], 0.0, 1.0) * np.ones((1, 1, Y, 1))
    m = np.zeros((B, Z, Y, X), np.float32)
    m[:, 1:-3, 1:-3, 1:-3] = f[:, 1:-3, 1:-3, 1:-3] > 0.0
    x = np.empty((B, Z, Y, X, 4), np.float32)
    x[..., 0] = rng.standard_normal((B, Z, Y, X), dtype=np.float32) * m
    x[..., 1] = f
    x[..., 2] = 1.0 - 0.5 * (rng.random((B, Z, 1, X), dtype=np.float32) < 0.1)
    x[..., 3] = m
    t = rng.standard_normal((B, Z, Y, X), dtype=np.float32) * m
    a7 = np.empty((B, Z, Y, X, 7), np.float32)
    a7[..., 1:] = -rng.random((B, Z, Y, X, 6), dtype=np.float32) * m[..., None]
    a7[..., 0] = 1.0 - a7[..., 1:].sum(-1)
    return warmstart.init_params(seed), x, t, m, a7


# ------------------------------------------------------------ the interface
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("tank", "host", "batch"):
        rng = np.random.default_rng(seed)
        runs = [_Run(c, case, rng) for c in _grids_of(case)]
        batch = P.Batch([r.tank for r in runs]) if kind == "batch" else None
        return dict(case=case, runs=runs, batch=batch)
    if kind == "solver":
        sysd, indc, _ = _system(case, seed, "cuda")
        return dict(case=case, tank=_solver_tank(case), sys=sysd, indc=indc, x=torch.zeros_like(sysd[0]))
    net = P.UNet(case["X"], case["Y"], case["Z"], case["batch"])
    params, x, t, m, a7 = _volumes(case, seed)
    net.set_params(params)
    return dict(case=case, net=net, x=x, t=t, m=m, a7=a7)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "tank":
        r = s["runs"][0]
        r.put()
        for _ in range(case["steps"]):
            if case["what"] == "drop":  # the adaptive step's limits, with the case's step as the largest
                r.tank.step(r.tank.cdtcal(dtinit=1e-4, dtmax=r.case.dt))
            else:
                r.tank.step(r.case.dt)
        return r.outputs()
    if kind == "host":
        r = s["runs"][0]
        r.end.copy_from(r.start)
        for _ in range(case["steps"]):
            r.host_step()
        return dict(r.end.views, fsum=r.tank.stats()["fsum"])
    if kind == "batch":
        for r in s["runs"]:
            r.put()
        for _ in range(case["steps"]):
            s["batch"].step()
        return [[v for k, v in sorted(r.outputs().items()) if k in REALS + ("nf",)] for r in s["runs"]]
    if kind == "solver":
        s["x"].zero_()
        torch.cuda.current_stream().synchronize()  # the solver runs on its tank's own stream
        P.m1bcgs_dev(s["tank"], *[a.data_ptr() for a in s["sys"]], s["x"].data_ptr(), s["indc"].data_ptr())
        return s["x"]
    if kind == "unet":
        return s["net"].forward(s["x"])
    loss, grad = s["net"].train_sys(s["x"], s["t"], s["m"], s["a7"], c=1.0, w_mse=0.1, w_res=1.0, lr=1e-3, want_grad=True)
    return loss, grad


def _conv_flops(case):
    vox = case["batch"] * case["X"] * case["Y"] * case["Z"]
    lv = (0, 0, 1, 1, 2, 2, 1, 1, 0, 0)
    return sum(2 * 27 * ci * co * vox / 8 ** l for (ci, co), l in zip(warmstart.LAYERS, lv))


def work(case):
    """Simulations: every resident field of a step once in and once out, and
    the pressure system with its solution; the solver's iterations are how it
    gets there, not what the path cannot do without."""
    kind = case["kind"]
    if kind in ("unet", "train"):
        vox = case["batch"] * case["X"] * case["Y"] * case["Z"]
        par = 4 * warmstart.init_params(0).size
        if kind == "unet":
            return dict(bytes=vox * (16 + 4) + par, flops=_conv_flops(case))
        return dict(bytes=vox * (16 + 4 + 4 + 28) + 7 * par, flops=3 * _conv_flops(case))
    if kind == "solver":
        n = (case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2)
        return dict(bytes=n * (8 * 8 + 8 + 4), flops=n * 14)
    cells = sum(c.ni * c.nj * c.nk for c in _grids_of(case))
    state = cells * (8 * len(REALS) + 4 * len(INTS))
    static = cells * (8 * 10 + 4 * 3)  # porosities, inertia, drag, viscosity; face flags
    trips = case["steps"] if kind == "host" else 1
    return dict(bytes=2 * trips * state + case["steps"] * (2 * state + static + cells * 8 * 9), flops=case["steps"] * cells * 400)


def exact(case, seed):
    """64-bit values from plain torch: the solution of the solver's system, the
    network's output, its loss and gradient.  A whole SMAC step has none here:
    it would be a second program of the library's size, and takes minutes on
    these grids."""
    kind = case["kind"]
    if kind == "solver":
        return _exact_solution(case, seed)
    if kind in ("unet", "train"):
        return _exact_net(case, seed)
    return None


def _exact_solution(case, seed):
    """Conjugate gradients with a diagonal preconditioner in 64 bits (the system is symmetric), to 1e-15."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    (ad, li, lj, lk, ui, uj, uk, b), _, live = _system(case, seed, dev)

    def mul(v):
        return (ad * v + li * v.roll(1, 2) + lj * v.roll(1, 1) + lk * v.roll(1, 0) + ui * v.roll(-1, 2) + uj * v.roll(-1, 1) +
                uk * v.roll(-1, 0)) * live

    x = torch.zeros_like(b)
    for _ in range(2):  # restarted once from the true residual
        r = b - mul(x)
        z = r / ad
        p, rz = z.clone(), (r * z).sum()
        stop = 1e-30 * (b * b / ad).sum()
        for n in range(20000):
            q = mul(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            z = r / ad
            new = (r * z).sum()
            if n % 25 == 24 and bool(new <= stop):
                break
            p = z + (new / rz) * p
            rz = new
    return x


def _exact_net(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    params, x, t, m, a7 = (torch.from_numpy(v).to(dev, torch.float64) for v in _volumes(case, seed))
    train = case["kind"] == "train"
    params.requires_grad_(train)
    at = 0

    def conv(v, n):
        """3x3x3 convolution, bias and ReLU: 27 shifted products over (B,Z,Y,X,C)."""
        nonlocal at
        ci, co = warmstart.LAYERS[n]
        w = params[at:at + 27 * ci * co].view(co, 27, ci)
        bias = params[at + 27 * ci * co:at + 27 * ci * co + co]
        at += 27 * ci * co + co
        Z, Y, X = v.shape[1:4]
        pad = torch.nn.functional.pad(v, (0, 0, 1, 1, 1, 1, 1, 1))
        out = bias
        for tap in range(27):
            dz, dy, dx = tap // 9, tap // 3 % 3, tap % 3
            out = out + pad[:, dz:dz + Z, dy:dy + Y, dx:dx + X] @ w[:, tap].T
        return torch.relu(out)

    def pool(v):
        B, Z, Y, X, C = v.shape
        return v.view(B, Z // 2, 2, Y // 2, 2, X // 2, 2, C).mean((2, 4, 6))

    def up(v):
        return v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    with torch.set_grad_enabled(train):
        v = torch.nn.functional.pad(x, (0, 12))
        s0 = conv(conv(v, 0), 1)
        s1 = conv(conv(pool(s0), 2), 3)
        v = conv(conv(pool(s1), 4), 5)
        v = conv(conv(torch.cat([up(v), s1], -1), 6), 7)
        v = conv(conv(torch.cat([up(v), s0], -1), 8), 9)
        y = v @ params[at:at + 16] + params[at + 16]
        if not train:
            return y.cpu().numpy()
        n = m.sum()
        my = torch.nn.functional.pad(m * y, (1, 1, 1, 1, 1, 1))
        Z, Y, X = y.shape[1:]
        ay = 0.0
        for c, (dz, dy, dx) in enumerate(((1, 1, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 2), (1, 2, 1), (2, 1, 1))):
            ay = ay + a7[..., c] * my[:, dz:dz + Z, dy:dy + Y, dx:dx + X]
        loss = 0.1 * (m * (y - t) ** 2).sum() / n + (m * (x[..., 0] - ay) ** 2).sum() / n
        loss.backward()
    return float(loss), params.grad.cpu().numpy()
