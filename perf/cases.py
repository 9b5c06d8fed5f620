"""What the engine's speed is measured on: the calls a user's program makes, over their range of sizes.

Four kinds of case, each through the package's public entry points:
  ramsey   a whole interferometry run: ground states from host memory, the first pi/2 pulse, split steps with
           samples of the moments (and axial profiles, and the states of a small ensemble) back to the host
  ground   the ground state of one ensemble (FP64), as a run starts from
  batch    ground states of many parameter sets at once (FP32), as the warm start's training data and evaluation
  mlp      the warm-start network: inference, gradients, training
`exact` gives the same outputs in 64 bits from the definitions, with torch alone.
"""
import math

import numpy as np
import torch

from bec_b200 import warmstart
from bec_b200._abi import (BEC_GS_FIXED_STEPS, BEC_GS_MU, BEC_GS_MU_RESIDUAL, BEC_LR_COSINE, BEC_PATH_FP32_BATCHED,
                           BEC_PATH_FP64_PLAIN)
from bec_b200.configs import A11, A12, A22, FX, FZ, GAMMA12, GAMMA22, GAMMA111, RB87_MASS, rb87_params
from bec_b200.engine import MLP, Engine

DT_EVO, DT_STEADY = 4e-5, 1e-5


def _ramsey(name, grids, groups, ne, steps, every, noise=True, pi=-1, axial=False, states=False, path="fp32"):
    """`groups` ensembles of `ne` trajectories each, their grids taken in turn from `grids`."""
    return dict(name=name, kind="ramsey", grids=grids, groups=groups, ne=ne, steps=steps, every=every, noise=noise,
                pi=pi, axial=axial, states=states, path=path)


def listed():
    return [
        # the 2D x-z slice: one noise-free trajectory, the smallest run; every launch counts
        _ramsey("slice_32x128", "32x1x128", 1, 1, 500, 100, noise=False, states=True),
        # the reference's own ensemble size: four noisy trajectories, still bound by latency
        _ramsey("ensemble_16x16x128", "16x16x128", 1, 4, 500, 50, states=True),
        # the uneven batch of the benchmark: 1024 ensembles of one trajectory, three grid classes, e2e from host memory
        _ramsey("uneven_1024", "8x8x64 16x16x128 32x32x256", 1024, 1, 40, 10),
        # the spin echo: the largest ensemble, a pi pulse half way
        _ramsey("spin_echo_1024", "32x32x256", 1, 1024, 16, 8, pi=8),
        # grids that are not square, or long and short in z, in one context, sampled with axial profiles as the
        # experiment front-end does
        _ramsey("mixed_grids_axial", "16x8x64 8x8x32 4x4x512 64x32x16 128x1x32", 10, 5, 100, 10, axial=True),
        # double precision, where a run is checked against single
        _ramsey("ensemble_fp64", "16x16x128", 1, 4, 20, 10, states=True, path="fp64"),
        # the ground state that a run starts from
        dict(name="ground_16x16x128", kind="ground", grid="16x16x128", steps=500, check=0),
        # training data of the warm start: cold ground states, coefficients back
        dict(name="batch_cold_256", kind="batch", grid="32x32x256", n=256, steps=200, check=20, warm=False, rows=50),
        # held-out sets started from predicted coefficients: few steps, so what surrounds the loop counts
        dict(name="batch_warm_96", kind="batch", grid="32x32x256", n=96, steps=60, check=20, warm=True, rows=50),
        # the network: inference for the held-out sets (the smallest call), gradients at odd sizes, training
        dict(name="mlp_forward_256", kind="mlp", do="forward", widths="6-256-256-256-64", batch=256, n=256, steps=0),
        dict(name="mlp_gradients_odd", kind="mlp", do="gradients", widths="5-70-130-3", batch=100, n=100, steps=0),
        dict(name="mlp_train", kind="mlp", do="train", widths="6-256-256-256-64", batch=256, n=4096, steps=400),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ramsey", "ramsey", "ramsey", "ground", "batch", "mlp"])
    if kind == "ramsey":
        fp64 = rng.random() < 0.15
        grid = rng.choice(["32x1x128", "64x1x64", "16x1x256", "8x8x64", "8x8x256", "16x16x64", "16x16x128", "16x16x256",
                           "32x32x64", "32x32x128", "32x32x256", "16x8x64", "8x8x32", "4x4x512", "64x32x16"])
        nx, ny, nz = _dims(grid)
        cells = nx * ny * nz
        ne = _log_int(rng, 1, max(1, min(300, (1 << 19 if fp64 else 1 << 26) // cells)))
        steps = _log_int(rng, 20, 400)
        while steps > 20 and ne * cells * steps > (1 << 23 if fp64 else 1 << 31):
            steps = max(20, steps // 2)
        axial, states = rng.random() < 0.4, ne * cells <= 1 << 18
        return dict(kind="ramsey", grids=grid, groups=rng.randint(1, 2) if ne > 1 else 1, ne=ne, steps=steps,
                    every=max(1, steps // rng.randint(1, 8)), noise=rng.random() < 0.8,
                    pi=rng.choice([-1, steps // 2]), axial=axial, states=states, path="fp64" if fp64 else "fp32")
    if kind == "ground":
        return dict(kind="ground", grid=rng.choice(["32x1x128", "8x8x64", "16x16x128", "32x32x256", "16x8x64", "64x32x16"]),
                    steps=_log_int(rng, 50, 400), check=rng.choice([0, 0, 10]))
    if kind == "batch":
        return dict(kind="batch", grid=rng.choice(["8x8x64", "16x16x128", "32x32x256", "16x16x64", "32x32x128"]),
                    n=_log_int(rng, 3, 200), steps=_log_int(rng, 30, 150), check=rng.choice([7, 20]),
                    warm=rng.random() < 0.5, rows=rng.choice([17, 50, 64]))
    widths = rng.choice(["6-256-256-256-64", "6-512-512-512-64", "5-70-130-3", "3-40-40-40-1", "6-256-64"])
    do = rng.choice(["forward", "gradients", "train"])
    batch = _log_int(rng, 20, 2000) if do != "train" else _log_int(rng, 60, 512)
    return dict(kind="mlp", do=do, widths=widths, batch=batch, n=4 * batch if do == "train" else batch,
                steps=_log_int(rng, 40, 200) if do == "train" else 0)


# ---------------------------------------------------------------- inputs
def _dims(grid):
    return tuple(int(v) for v in grid.split("x"))


def _sets(case, seed):
    """The parameter sets of a case, as plain dicts: trap frequencies, atom number, scattering lengths, Philox seed."""
    rng = np.random.default_rng([seed, 11])
    grids = [_dims(g) for g in case.get("grids", case.get("grid")).split()]
    n = case["n"] if case["kind"] == "batch" else case.get("groups", 1)
    out = []
    for i in range(n):
        lo, hi = ((5e3, 1e5) if case["kind"] == "batch" else (5e3, 7e4))
        sx, sz = rng.uniform(0.9, 1.1, 2)
        s = rng.uniform(0.98, 1.02, 3) if case["kind"] == "batch" else np.ones(3)
        out.append(dict(grid=grids[i % len(grids)], N=float(rng.uniform(lo, hi)), fx=FX * sx, fz=FZ * sz, a11=A11 * s[0],
                        a12=A12 * s[1], a22=A22 * s[2], seed=int(1000003 * (seed % 1000003) + i)))
    return out


def _params(case, seed):
    return [rb87_params(N=s["N"], grid=s["grid"], ne=case.get("ne", 1), noise=bool(case.get("noise", False)), fx=s["fx"],
                        fy=s["fx"], fz=s["fz"], a11=s["a11"], a12=s["a12"], a22=s["a22"], seed=s["seed"])
            for s in _sets(case, seed)]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _starts(case, seed):
    """Host ground states (Thomas-Fermi): complex128 for one ensemble; for many, real FP32 back to back in pinned
    memory, as a program that hands many arrays over keeps them."""
    sets = _sets(case, seed)
    if len(sets) == 1:
        return [_States(sets, case).thomas_fermi().reshape(-1).cpu().numpy().astype(np.complex128)]
    sizes = [math.prod(s["grid"]) for s in sets]
    flat = torch.empty(sum(sizes), dtype=torch.float32, pin_memory=torch.cuda.is_available())
    views = flat.split(sizes)
    for grid in dict.fromkeys(s["grid"] for s in sets):
        for part in _chunks([i for i, s in enumerate(sets) if s["grid"] == grid], math.prod(grid)):
            for i, v in zip(part, _States([sets[i] for i in part], case).thomas_fermi().float().cpu()):
                views[i].copy_(v.reshape(-1))
    return [v.numpy() for v in views]


def _basis(grid, rows):
    """Orthonormal smooth rows (rows x cells, float32) in the scaled coordinates, as a learned basis has them."""
    nx, ny, nz = grid
    ax = [torch.linspace(-1.2, 1.2, n, dtype=torch.float64, device=_device()) if n > 1 else
          torch.zeros(1, dtype=torch.float64, device=_device()) for n in (nz, ny, nx)]
    Z, Y, X = torch.meshgrid(*ax, indexing="ij")
    rho2, z2 = (X * X + Y * Y).reshape(-1), (Z * Z).reshape(-1)
    env = torch.exp(-(rho2 + z2) ** 2)
    cols = [env * torch.cos(1.3 * i * rho2) * torch.cos(1.7 * j * z2) for i in range(8) for j in range(8)]
    return torch.linalg.qr(torch.stack(cols[:rows], 1))[0].T.contiguous().float()


def _mlp_inputs(case, seed):
    w = [int(v) for v in case["widths"].split("-")]
    rng = np.random.default_rng([seed, 12])
    x = rng.uniform(-1.0, 1.0, (case["n"], w[0])).astype(np.float32)
    mix = rng.normal(0.0, 1.0, (w[0], w[-1]))
    t = np.sin(x @ mix + rng.uniform(0, 6, w[-1])).astype(np.float32)
    p = []
    for a, b in zip(w[:-1], w[1:]):
        lim = math.sqrt(6.0 / (a + b))
        p += [rng.uniform(-lim, lim, a * b), rng.normal(0.0, 0.05, b)]
    return w, x, t, np.concatenate(p).astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "ramsey":
        eng = Engine(_params(case, seed), path=BEC_PATH_FP64_PLAIN if case["path"] == "fp64" else BEC_PATH_FP32_BATCHED)
        return dict(case=case, eng=eng, gs=_starts(case, seed))
    if case["kind"] == "ground":
        return dict(case=case, eng=Engine(_params(case, seed), path=BEC_PATH_FP32_BATCHED))
    if case["kind"] == "batch":
        grid, params = _dims(case["grid"]), _params(case, seed)
        state = dict(case=case, params=params, grid=grid, basis=_basis(grid, case["rows"]).cpu().numpy())
        if case["warm"]:
            state["eng"] = Engine(params, path=BEC_PATH_FP32_BATCHED)
            state["eng"].set_warmstart_basis(grid, state["basis"])
            state["coef"] = _coef_in(case, seed)
        return state
    w, x, t, p = _mlp_inputs(case, seed)
    state = dict(case=case, widths=w, x=x, t=t, seed=seed)
    if case["do"] != "train":
        state["net"] = MLP(w, seed=seed)
        state["net"].set_params(p)
    return state


def _coef_in(case, seed):
    rng = np.random.default_rng([seed, 13])
    cells = math.prod(_dims(case["grid"]))
    c = np.zeros((case["n"], 64))
    c[:, :case["rows"]] = rng.normal(0.0, 0.01 * math.sqrt(cells), (case["n"], case["rows"])) * 0.85 ** np.arange(case["rows"])
    return c


def run(state):
    case = state["case"]
    if case["kind"] == "ramsey":
        eng = state["eng"]
        eng.set_step_index(0, 0)
        if len(state["gs"]) == 1:
            eng.init_group(0, state["gs"][0])
        else:
            eng.init_groups(range(eng.n_groups), state["gs"])
        eng.start_evolution()
        got = eng.run(case["steps"], sample_every=case["every"], pi_pulse_step=case["pi"], axial=case["axial"])
        out = {"moments": got[0] if case["axial"] else got}
        if case["axial"]:
            out["axial"] = list(got[1])
        if case["states"]:
            out["states"] = np.concatenate([eng.get_state(g, t).reshape(-1) for g in range(eng.n_groups)
                                            for t in range(case["ne"])])
        return out
    if case["kind"] == "ground":
        psi, rep = state["eng"].ground_state(0, mode=BEC_GS_MU if case["check"] else BEC_GS_FIXED_STEPS, max_steps=case["steps"],
                                             tol=0.0, check_every=max(1, case["check"]))
        return {"psi": psi, "steps": rep.steps, "report": [rep.mu, rep.energy, rep.N, rep.residual]}
    if case["kind"] == "batch":
        kw = dict(mode=BEC_GS_MU_RESIDUAL, max_steps=case["steps"], tol=1e-13, check_every=case["check"])
        if case["warm"]:
            coef, _, reps = state["eng"].ground_state_coeffs(coef_in=state["coef"], **kw)
            get = lambda k: np.array([getattr(r, k) for r in reps])  # noqa: E731
            return {"coef": coef, "steps": get("steps"), "mu": get("mu"), "energy": get("energy"), "N": get("N"),
                    "residual": get("residual"), "step_residual": get("step_residual")}
        got = warmstart.ground_states(state["params"], basis=state["basis"], **kw)
        return {k: got[k] for k in ("coef", "steps", "mu", "residual", "step_residual")}
    if case["do"] == "forward":
        return state["net"].forward(state["x"])
    if case["do"] == "gradients":
        loss, grads = state["net"].gradients(state["x"], state["t"])
        return {"loss": loss, "grads": grads}
    net = MLP(state["widths"], seed=state["seed"])
    hist = net.train(state["x"], state["t"], case["steps"], batch=case["batch"], lr=1e-3, seed=state["seed"],
                     schedule=BEC_LR_COSINE)
    params = net.get_params()
    net.close()
    return {"params": params, "history": hist}


# ---------------------------------------------------------------- work
def work(case):
    if case["kind"] == "mlp":
        w = [int(v) for v in case["widths"].split("-")]
        pars = sum(a * b + b for a, b in zip(w[:-1], w[1:]))
        macs = sum(a * b for a, b in zip(w[:-1], w[1:]))
        rows, passes, steps = case["batch"], {"forward": 1, "gradients": 3, "train": 3}[case["do"]], max(1, case["steps"])
        io = 4 * rows * (w[0] + w[-1])
        per = {"forward": 4 * pars + io, "gradients": 8 * pars + io, "train": 24 * pars + io}[case["do"]]
        return {"bytes": steps * per, "flops": steps * passes * 2 * rows * macs}
    if case["kind"] == "ramsey":
        per, el = 1, (64 if case["path"] == "fp64" else 32)
        sets, comps = _plain_grids(case), 2
        per = case["ne"]
        steps, cell_flops = case["steps"] + 1, 200 if case["noise"] else 80
    else:
        sets, comps, per, steps, cell_flops = _plain_grids(case), 1, 1, case["steps"], 30
        el = 32 if case["kind"] == "ground" else 16
    total, flops = 0.0, 0.0
    for nx, ny, nz in sets:
        cells = nx * ny * nz * per
        total += cells
        flops += steps * cells * (comps * 10 * math.log2(nx * ny * nz) + cell_flops)
    # each step reads and writes the state once; the start comes from the host or is made on the device
    return {"bytes": total * el * steps, "flops": flops}


def _plain_grids(case):
    grids = [_dims(g) for g in case.get("grids", case.get("grid")).split()]
    n = case["n"] if case["kind"] == "batch" else case.get("groups", 1)
    return [grids[i % len(grids)] for i in range(n)]


# ---------------------------------------------------------------- the same in 64 bits
_M32 = 0xFFFFFFFF


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 on int64 tensors that hold 32-bit words (products wrap modulo 2^64)."""
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & _M32) ^ c1 ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c3 ^ k1, p0 & _M32)
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c0, c1, c2, c3


class _States:
    """States of parameter sets that share one grid, in natural units and 64 bits; axes (state, z, y, x)."""

    def __init__(self, sets, case):
        self.case = case
        self.dev = dev = _device()
        self.nx, self.ny, self.nz = nx, ny, nz = sets[0]["grid"]
        self.cells = nx * ny * nz

        def col(v):
            return torch.tensor(v, dtype=torch.float64, device=dev).reshape(-1, 1, 1, 1)

        hbar, bohr = 1.054571628e-34, 5.2917720859e-11
        w = 2.0 * math.pi * col([s["fx"] for s in sets])
        l = torch.sqrt(hbar / (RB87_MASS * w))
        self.lam = col([s["fx"] / s["fz"] for s in sets])
        self.l111, self.l12, self.l22 = GAMMA111 / (l ** 6 * w), GAMMA12 / (l ** 3 * w), GAMMA22 / (l ** 3 * w)
        self.g11, self.g12, self.g22 = (4.0 * math.pi * col([s[k] for s in sets]) * bohr / l for k in ("a11", "a12", "a22"))
        self.N = col([s["N"] for s in sets])
        if ny > 1:
            self.mu = (15.0 * self.N * self.g11 / (16.0 * math.pi * self.lam * math.sqrt(2.0))) ** 0.4
        else:   # the transverse width is 1 (fy = fx)
            s2, s3 = 1.0 / math.sqrt(2.0 * math.pi), 1.0 / (math.sqrt(3.0) * math.pi)
            self.g11, self.g12, self.g22 = self.g11 * s2, self.g12 * s2, self.g22 * s2
            self.l12, self.l22, self.l111 = self.l12 * s2, self.l22 * s2, self.l111 * s3
            self.mu = torch.sqrt(self.N * self.g11 / (math.pi * self.lam))
        self.dt, self.dts = DT_EVO * w, DT_STEADY * w
        self.amp = torch.sqrt(self.mu / self.g11)
        half = 1.2 * torch.sqrt(2.0 * self.mu)
        self.dV, self.V, self.K = torch.ones_like(w), 0.0, 0.0
        for n, axis, h in ((nx, 3, half), (ny, 2, half), (nz, 1, half * self.lam)):
            if n == 1:
                continue
            shape = [1, 1, 1, 1]
            shape[axis] = n
            i = torch.arange(n, dtype=torch.float64, device=dev).reshape(shape)
            d = 2.0 * h / (n - 1)
            self.dV = self.dV * d
            self.V = self.V + (-h + d * i) ** 2 / (2.0 * (self.lam ** 2 if axis == 1 else 1.0))
            self.K = self.K + (torch.where(2 * i > n, i - n, i) * math.pi / h) ** 2 / 2.0

    def thomas_fermi(self):
        return torch.sqrt(torch.clamp(self.mu - self.V, min=0.0) / self.g11)

    @staticmethod
    def to_k(v):
        return torch.fft.ifftn(v, dim=(-3, -2, -1))

    @staticmethod
    def to_x(v):
        return torch.fft.fftn(v, dim=(-3, -2, -1))

    # ---- real time
    def init(self, traj, seeds, single):
        """x-space start of trajectory traj[i] of the ensemble with Philox seed seeds[i] on every state; single: the
        ground state is handed over in 32 bits."""
        gs = self.thomas_fermi()
        gs = gs.float().double() if single else gs
        words = torch.tensor([[t, s & _M32, s >> 32] for t, s in zip(traj, seeds)], dtype=torch.int64, device=self.dev)
        self.traj, *self.keys = words.T.reshape(3, -1, 1, 1, 1)
        self.cell = torch.arange(self.cells, dtype=torch.int64, device=self.dev).reshape(1, self.nz, self.ny, self.nx)
        self.a, self.b = gs.to(torch.complex128), torch.zeros_like(gs, dtype=torch.complex128)
        self.philox_step = 0
        if self.case["noise"]:
            w, n = self.draw(0, 0), []
            for u, v in ((w[0], w[1]), (w[2], w[3])):
                nl = torch.where(u < 0x80000000, -torch.log((u.double() + 1.0) * 2.0 ** -32),
                                 -torch.log1p(-((_M32 - u).double()) * 2.0 ** -32))
                n.append(torch.polar(torch.sqrt(2.0 * nl), v.double() * (2.0 * math.pi * 2.0 ** -32)) * 0.5 / torch.sqrt(self.dV))
            self.a, self.b = self.a + n[0], n[1]

    def draw(self, step, tag):
        zero = torch.zeros_like(self.cell)
        return _philox(self.cell + 0 * self.traj, zero + step, self.traj, zero + tag, *self.keys)

    def kick(self, v):
        return self.to_x(self.to_k(v) * torch.polar(torch.ones_like(self.K), self.K * self.dt / 2.0))

    def advance(self):
        a, b = self.kick(self.a), self.kick(self.b)
        na, nb, h = a.real ** 2 + a.imag ** 2, b.real ** 2 + b.imag ** 2, self.dt / 2.0
        da = torch.polar(torch.exp(-(self.l111 * na * na + self.l12 * nb) / 2.0 * h), (self.V + self.g11 * na + self.g12 * nb) * h)
        db = torch.polar(torch.exp(-(self.l22 * nb + self.l12 * na) / 2.0 * h), (self.V + self.g22 * nb + self.g12 * na) * h)
        ao, bo = a * da * da, b * db * db
        if self.case["noise"]:
            w = self.draw(self.philox_step, 1)
            f = (w[0] & 0x1FFFFF, (w[0] >> 21) | ((w[1] & 0x3FF) << 11), (w[1] >> 10) & 0x1FFFFF,
                 (w[1] >> 31) | ((w[2] & 0xFFFFF) << 1), (w[2] >> 20) | ((w[3] & 0x1FF) << 12), (w[3] >> 9) & 0x1FFFFF)
            amp = torch.sqrt(self.dt / (2.0 * self.dV))
            w1, w2, w3 = (torch.polar(amp * torch.sqrt(-2.0 * torch.log((f[i].double() + 0.5) * 2.0 ** -21)),
                                      f[i + 1].double() * (2.0 * math.pi * 2.0 ** -21)) for i in (0, 2, 4))
            ca, cb = a.conj(), b.conj()
            c1, c2, c3 = 3.0 * torch.sqrt(self.l111 / 6.0), torch.sqrt(self.l12 / 2.0), torch.sqrt(self.l22)
            ao = ao + c1 * ca * ca * w1 + c2 * cb * w2
            bo = bo + c2 * ca * w2 + c3 * cb * w3
        self.a, self.b = self.kick(ao), self.kick(bo)
        self.philox_step += 1

    def pulse(self, theta):
        c, s = math.cos(theta / 2.0), math.sin(theta / 2.0)
        self.a, self.b = c * self.a - 1j * s * self.b, -1j * s * self.a + c * self.b

    def sums(self):
        """(state, z, 4): |a|^2, |b|^2 and conj(a) b, summed over y and x."""
        ab = self.a.conj() * self.b
        v = (self.a.real ** 2 + self.a.imag ** 2, self.b.real ** 2 + self.b.imag ** 2, ab.real, ab.imag)
        return (torch.stack([q.sum(dim=(2, 3)) for q in v], 2) * self.dV[:, :, 0]).cpu().numpy()

    # ---- imaginary time
    @staticmethod
    def norm2(x):
        return (x.real ** 2 + x.imag ** 2).sum(dim=(1, 2, 3), keepdim=True)

    def renorm(self, x):
        return x * torch.sqrt(self.N / (self.norm2(x) * self.dV))

    def imaginary_step(self, x):
        f = torch.exp(-self.dts / 2.0 * self.K)
        x = self.to_x(self.to_k(x) * f)
        x = x * torch.exp(self.dts / 2.0 * (-self.V - self.g11 * (x.real ** 2 + x.imag ** 2))) ** 2
        return self.renorm(self.to_x(self.to_k(x) * f))

    def measures(self, x):
        """mu, energy per particle, norm and residual of every state."""
        n, xk = x.real ** 2 + x.imag ** 2, self.to_k(x)
        total = lambda v: v.sum(dim=(1, 2, 3), keepdim=True) * self.dV  # noqa: E731
        ekin = total((xk.real ** 2 + xk.imag ** 2) * self.K) * self.cells
        epot, eint, N = total(n * self.V), self.g11 * total(n * n), total(n)
        mu = (ekin + epot + eint) / N
        h = self.to_x(xk * self.K) + x * (self.V + self.g11 * n - mu)
        res = torch.sqrt(self.norm2(h) * self.dV / N)
        return mu, (ekin + epot + 0.5 * eint) / N, N, res


def _chunks(items, cells):
    size = max(1, (1 << 25) // cells)
    return [items[i:i + size] for i in range(0, len(items), size)]


def _exact_ramsey(case, seed):
    sets = _sets(case, seed)
    n_samples, ne = case["steps"] // case["every"], case["ne"]
    moments = np.zeros((n_samples, len(sets), 5))
    axial = [np.zeros((n_samples, s["grid"][2], 4)) for s in sets]
    states = {}
    for grid in dict.fromkeys(s["grid"] for s in sets):
        mine = [(g, t) for g, s in enumerate(sets) if s["grid"] == grid for t in range(ne)]
        for part in _chunks(mine, math.prod(grid)):
            st = _States([sets[g] for g, _ in part], case)
            st.init([t for _, t in part], [sets[g]["seed"] for g, _ in part], len(sets) > 1)
            st.advance()
            st.pulse(math.pi / 2.0)
            for i in range(1, case["steps"] + 1):
                st.advance()
                if i % case["every"] == 0:
                    for (g, _), v in zip(part, st.sums()):
                        axial[g][i // case["every"] - 1] += v
                        moments[i // case["every"] - 1, g, 1:] += v.sum(axis=0)
                if i == case["pi"]:
                    st.pulse(math.pi)
            if case["states"]:
                both = torch.stack([st.a, st.b], 1).reshape(len(part), 2, -1).cpu().numpy()
                states.update(zip(part, both))
            del st
    moments[:, :, 0] = (np.arange(1, n_samples + 1) * case["every"] * DT_EVO)[:, None]
    out = {"moments": moments}
    if case["axial"]:
        out["axial"] = axial
    if case["states"]:
        out["states"] = np.concatenate([states[g, t].reshape(-1) for g in range(len(sets)) for t in range(ne)])
    return out


def _exact_batch(case, seed):
    grid, rows = _dims(case["grid"]), case["rows"]
    B = _basis(grid, rows).double()
    gram = B @ B.T
    gram = gram + 1e-10 * gram[0, 0] * torch.eye(rows, dtype=torch.float64, device=B.device)
    out = {k: [] for k in ("coef", "mu", "energy", "N", "residual", "step_residual")}
    sets = _sets(case, seed)
    for part in _chunks(list(range(len(sets))), math.prod(grid)):
        st = _States([sets[i] for i in part], case)
        scaled = torch.sqrt(torch.clamp(1.0 - st.V / st.mu, min=0.0))
        x = st.amp * scaled
        if case["warm"]:
            c = torch.tensor(_coef_in(case, seed)[part][:, :rows], device=B.device)
            x = st.amp * torch.clamp(scaled + (c @ B).reshape(scaled.shape), min=0.0)
        x = st.renorm(x.to(torch.complex128))
        prev, change, checks = None, torch.zeros_like(st.mu), 0
        for k in range(1, case["steps"] + 1):
            x = st.imaginary_step(x)
            if k % case["check"] == 0 and k < case["steps"]:
                if checks:
                    change = torch.sqrt(st.norm2(x - prev) / st.norm2(x)) / (case["check"] * st.dts * st.measures(x)[0].abs())
                prev, checks = x, checks + 1
        d = (x.abs() / st.amp - scaled).reshape(len(part), -1)
        c = torch.zeros(len(part), 64, dtype=torch.float64, device=B.device)
        c[:, :rows] = torch.linalg.solve(gram, B @ d.T).T
        for k, v in zip(out, (c, *st.measures(x), change)):
            out[k].append((v if k == "coef" else v.reshape(-1)).cpu().numpy())
    keep = ("coef", "steps", "mu", "energy", "N", "residual", "step_residual") if case["warm"] else \
        ("coef", "steps", "mu", "residual", "step_residual")
    return {k: None if k == "steps" else np.concatenate(out[k]) for k in keep}


def _exact_mlp(case, seed):
    w, x, t, p = _mlp_inputs(case, seed)
    dev, o, layers = _device(), 0, []
    p = torch.tensor(p, dtype=torch.float64, device=dev)
    for a, b in zip(w[:-1], w[1:]):
        layers.append((p[o:o + a * b].reshape(b, a).clone().requires_grad_(), p[o + a * b:o + a * b + b].clone().requires_grad_()))
        o += a * b + b
    y = torch.tensor(x, dtype=torch.float64, device=dev)
    for i, (W, bias) in enumerate(layers):
        y = y @ W.T + bias
        if i + 1 < len(layers):
            y = torch.tanh(y)
    if case["do"] == "forward":
        return y.detach().cpu().numpy()
    loss = ((y - torch.tensor(t, dtype=torch.float64, device=dev)) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grads": torch.cat([q.grad.reshape(-1) for l in layers for q in l]).cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "ramsey":
        return _exact_ramsey(case, seed)
    if case["kind"] == "batch":
        return _exact_batch(case, seed)
    if case["kind"] == "mlp":
        # a training run's minibatch order comes from the library's own shuffle
        return None if case["do"] == "train" else _exact_mlp(case, seed)
    st = _States(_sets(case, seed), case)
    x = st.renorm(st.thomas_fermi().to(torch.complex128))
    for _ in range(case["steps"]):
        x = st.imaginary_step(x)
    return {"psi": x.reshape(-1).cpu().numpy(), "steps": None, "report": [float(v) for v in st.measures(x)]}
