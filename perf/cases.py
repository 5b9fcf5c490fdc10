"""The work that programs have this framework do, as cases that can be timed.

Four kinds of call, each through its public entry point:

* ``projection``: one compatibility projection of a field that is already on the GPU
  (``ssfft_apply_projection_device`` of a solver handle, planar (6, V) in and out);
* ``solve``: a run of load increments on a handle that is kept
  (``SolverHandle.solve_constant_rates``), stress and strain read back into GPU buffers
  (``ssfft_get_field``);
* ``material``: the drop-in call ``SmallStrainFFT(...)(material)``, host fields in and out;
* ``serve``: a batch of requests through a running ``RVEServer``.

Grid points are numbered in C order of (x, y, z); symmetric tensors are Mandel 6-vectors.
"""

import ctypes
import math

import numpy as np
import torch

import materialite_b200 as mb
from materialite_b200 import _native as nat
from materialite_b200 import serving
from materialite_b200.engine import PhaseSpec, SolverHandle
from materialite_b200.small_strain_fft import (Elastic, ElasticViscoplastic, LoadSchedule,
                                               SmallStrainFFT, voce)

# ---- the cases ---------------------------------------------------------------------------


def _projection(nx, ny, nz, precision):
    return {"kind": "projection", "nx": nx, "ny": ny, "nz": nz, "precision": precision}


def _solve(nx, ny, nz, precision, model, grains, steps, biaxial=False):
    return {"kind": "solve", "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "model": model, "grains": grains, "steps": steps, "biaxial": biaxial}


def listed():
    return [
        # a single projection at the reference's default grid, where launches are the cost
        dict(_projection(16, 16, 16, "fp64"), name="projection fp64 16"),
        # ragged grid with an odd axis (radix 3, 5 and 7 factors)
        dict(_projection(42, 45, 75, "fp64"), name="projection fp64 42x45x75"),
        # the grid of the large plain solve, in the precision of its Krylov iterations
        dict(_projection(128, 128, 128, "mixed"), name="projection mixed 128"),
        # the grid of the largest workload, in the precision of its residuals
        dict(_projection(256, 256, 256, "fp64"), name="projection fp64 256"),
        # elastic homogenisation at the smallest grid of the serving mix
        dict(_solve(32, 32, 32, "fp64", "elastic", 50, 4), name="elastic fp64 32"),
        # the first increments of the plain 128^3 workload
        dict(_solve(128, 128, 128, "mixed", "elastic", 500, 2), name="elastic mixed 128"),
        # crystal plasticity at the middle size of the serving mix, through yield
        dict(_solve(64, 64, 64, "mixed", "evp", 200, 10), name="evp mixed 64"),
        # the same physics in double on a non-cubic grid
        dict(_solve(48, 40, 36, "fp64", "evp", 100, 8), name="evp fp64 48x40x36"),
        # crystal-plastic and stiff elastic grains together (contrast 10)
        dict(_solve(96, 96, 96, "mixed", "twophase", 200, 1), name="twophase mixed 96"),
        # J2 matrix with elastic grains, odd sizes, biaxial load
        dict(_solve(45, 50, 63, "fp64", "j2", 80, 3, True), name="j2 fp64 45x50x63"),
        # the drop-in call of a reference user: its defaults (double, tolerance 1e-3)
        {"name": "material fp64 32", "kind": "material", "nx": 32, "ny": 32, "nz": 32,
         "precision": "fp64", "model": "evp", "grains": 60, "steps": 8, "biaxial": False},
        # a burst of requests of the serving mix on a warm server
        {"name": "serve mixed 8", "kind": "serve", "precision": "mixed", "requests": 8,
         "largest": 64, "steps": 10},
    ]


def _size(rng, lo, hi):
    """A grid axis, spread over the logarithm of the range: the next length whose prime
    factors are at most 7 (odd ones among them)."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while n <= hi:
        m = n
        for f in (2, 3, 5, 7):
            while m % f == 0:
                m //= f
        if m == 1:
            return n
        n += 1
    return hi


def draw(rng):
    kind = rng.choice(["projection", "projection", "solve", "solve", "solve", "solve",
                       "material", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "projection":
        return _projection(*(_size(rng, 16, 256) for _ in range(3)), precision)
    if kind == "serve":
        return {"kind": "serve", "precision": precision, "requests": rng.randint(1, 10),
                "largest": rng.choice([32, 48, 64]), "steps": rng.randint(2, 10)}
    model = rng.choice(["elastic", "evp", "twophase", "j2"])
    if kind == "material":
        n = [_size(rng, 16, 40) for _ in range(3)]
        return {"kind": "material", "nx": n[0], "ny": n[1], "nz": n[2], "precision": precision,
                "model": rng.choice(["elastic", "evp"]), "grains": rng.randint(20, 80),
                "steps": rng.randint(1, 8), "biaxial": rng.random() < 0.5}
    top = 128 if model == "elastic" and precision == "mixed" else 80
    n = [_size(rng, 16, top) for _ in range(3)]
    steps = rng.randint(1, 10) if model == "evp" else rng.randint(1, 3)
    if model == "twophase":
        steps = 1
    return _solve(*n, precision, model, rng.randint(20, 400), steps, rng.random() < 0.5)


# ---- what one pass cannot do without -------------------------------------------------------

# Matrix-vector products of one load increment (linear solves times their iterations):
# counts seen with these models at contrast 1-10 and the tolerances used here.
_MATVECS = {"elastic": 15, "evp": 100, "twophase": 250, "j2": 80}


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _projection_flops(V):
    """Six real transforms there and back (2.5 V log2 V each) and the operator on half of
    the frequencies."""
    return 12 * 2.5 * V * math.log2(max(V, 2)) + 60 * V / 2


def _solve_work(V, precision, model, steps):
    """Per product: the direction and its tangent read, the result written."""
    w = 4 if precision == "mixed" else 8
    tangent = 4 if model == "elastic" else 21 * w
    n = steps * _MATVECS[model]
    return V * n * (12 * w + tangent) + 2 * 48 * V, n * (_projection_flops(V) + 66 * V)


def work(case):
    if case["kind"] == "projection":
        V = math.prod(_dims(case))
        return {"bytes": 2 * 6 * V * (4 if case["precision"] == "mixed" else 8),
                "flops": _projection_flops(V)}
    if case["kind"] == "serve":
        parts = [_solve_work(n ** 3, case["precision"], model, case["steps"])
                 for n, model, _ in _serve_mix(case)]
    else:
        parts = [_solve_work(math.prod(_dims(case)), case["precision"], case["model"],
                             case["steps"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ---- inputs --------------------------------------------------------------------------------

_DEVICE = "cuda"
_MODELS = {  # strain rate and time increment of a load step
    "elastic": (1e-3, 1.0), "evp": (1e-3, 0.2), "twophase": (1e-3, 0.2), "j2": (1.0, 5e-4),
}
_CUBIC = (250.0, 150.0, 120.0)
_EVP = {"rate": 1e-3, "exponent": 20.0, "resistance": 0.1,
        "voce": {"tau_1": 0.2, "theta_0": 1.0, "theta_1": 0.0}}
_J2 = {"modulus": 150000.0, "shear": 60000.0, "yield": 150.0, "hardening": 1000.0}
_GTOL, _LTOL = 1e-6, 1e-5


def _voronoi(dims, count, gen):
    """Grain of each point: the nearest of `count` seeds, periodic."""
    seeds = torch.rand(count, 3, dtype=torch.float64, generator=gen)
    seeds = seeds.to(_DEVICE) * torch.tensor(dims, dtype=torch.float64, device=_DEVICE)
    axes = []
    for a in range(3):
        d = (torch.arange(dims[a], dtype=torch.float64, device=_DEVICE)[:, None] - seeds[None, :, a]).abs()
        axes.append(torch.minimum(d, dims[a] - d).square())
    yz = axes[1][:, None, :] + axes[2][None, :, :]
    ids = torch.stack([(axes[0][x] + yz).argmin(-1) for x in range(dims[0])])
    return ids.reshape(-1).to(torch.int32).cpu().numpy()


def _microstructure(dims, grains, model, seed):
    """(rotations (G, 3, 3), grain of point, phase of point or None)."""
    gen = torch.Generator().manual_seed(int(seed))
    grain = _voronoi(dims, grains, gen)
    rng = np.random.default_rng(int(seed))
    rotations = mb.microstructure.quaternion_random_rotations(grains, rng)
    phase = None
    if model in ("twophase", "j2"):
        phase = (rng.random(grains) < 0.5).astype(np.int32)[grain]
    return rotations, grain, phase


def _cubic(scale=1.0):
    return serving.cubic(*_CUBIC, scale)


def _phases(model):
    if model == "elastic":
        return [PhaseSpec("elastic", _cubic())]
    if model == "j2":
        return [PhaseSpec("j2", _isotropic(), slip_resistance=_J2["yield"], hardening="linear",
                          hardening_props={"hardening_rate": _J2["hardening"]},
                          modulus=_J2["modulus"], shear_modulus=_J2["shear"]),
                PhaseSpec("elastic", _cubic(1000.0))]
    evp = serving.evp_phase()
    return [evp] if model == "evp" else [evp, PhaseSpec("elastic", _cubic(10.0))]


def _load(model, biaxial):
    """Stress mask and strain rate: stretched along x (and y), free of stress otherwise."""
    mask, rate = np.ones(6), np.zeros(6)
    for a in range(2 if biaxial else 1):
        mask[a], rate[a] = 0.0, _MODELS[model][0]
    return mask, rate


def _serve_mix(case):
    """(size, model, biaxial) of each request: the serving mix's sizes up to the largest."""
    sizes = [n for n in (32, 48, 64) if n <= case["largest"]]
    return [(sizes[(i + 1) % len(sizes)], "evp" if i % 2 else "elastic", i % 3 == 0)
            for i in range(case["requests"])]


def _serve_seed(seed, i):
    return 1000 * int(seed) + i


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        reqs = []
        for i, (n, model, biaxial) in enumerate(_serve_mix(case)):
            rotations, grain, _ = _microstructure((n, n, n), 20 + 40 * i, model,
                                                  _serve_seed(seed, i))
            mask, rate = _load(model, biaxial)
            reqs.append(serving.RVERequest(
                tag=i, dims=(n, n, n), phases=_phases(model), rotations=rotations, grain=grain,
                stress_mask=mask, strain_rate=rate, stress_rate=np.zeros(6),
                dt=_MODELS[model][1], steps=case["steps"], keep_stress=True))
        server = serving.RVEServer(max_slots=16, precision=case["precision"])
        return {"case": case, "server": server, "requests": reqs}
    dims = _dims(case)
    V = math.prod(dims)
    if kind == "projection":
        gen = torch.Generator(_DEVICE).manual_seed(int(seed))
        dtype = torch.float32 if case["precision"] == "mixed" else torch.float64
        tau = torch.randn(6, V, dtype=dtype, device=_DEVICE, generator=gen)
        mask, _ = _load("elastic", False)
        return {"case": case, "handle": SolverHandle(dims, mask, case["precision"]),
                "tau": tau, "out": torch.empty_like(tau)}
    model = case["model"]
    rotations, grain, phase = _microstructure(dims, case["grains"], model, seed)
    mask, rate = _load(model, case["biaxial"])
    if kind == "material":
        material = mb.Material(dimensions=list(dims)).create_fields(
            {"grain": grain, "orientation": mb.Orientation(rotations[grain], "p")})
        C = mb.Order4SymmetricTensor.from_cubic_constants(*_CUBIC)
        law = Elastic(C) if model == "elastic" else ElasticViscoplastic(
            C, mb.SlipSystem.octahedral(), _EVP["rate"], _EVP["exponent"], _EVP["resistance"],
            voce, _EVP["voce"])
        zero = mb.Order2SymmetricTensor.zero()
        dt = _MODELS[model][1]
        solver = SmallStrainFFT(
            LoadSchedule.from_constant_rates(mb.Order2SymmetricTensor(rate), zero, mask),
            end_time=dt * case["steps"], initial_time_increment=dt, constitutive_model=law,
            precision=case["precision"])
        return {"case": case, "solver": solver, "material": material}
    handle = SolverHandle(dims, mask, case["precision"], global_tolerance=_GTOL,
                          linear_solver_tolerance=_LTOL)
    handle.set_phases(_phases(model))
    handle.set_microstructure(rotations, grain, phase)
    return {"case": case, "handle": handle, "rate": rate, "V": V}


# ---- one pass ------------------------------------------------------------------------------


def _kept(x, precision):
    """Mixed-precision solves are single-precision results in double buffers; a program
    keeps them as such."""
    return x if precision == "fp64" else x.float()


def run(state):
    case = state["case"]
    kind, precision = case["kind"], case["precision"]
    if kind == "projection":
        h = state["handle"]
        nat.check(h.lib.ssfft_apply_projection_device(h.h, state["tau"].data_ptr(),
                                                      state["out"].data_ptr()))
        return state["out"]
    if kind == "solve":
        h = state["handle"]
        # the handle works on its own stream: earlier work on the buffers has to be done
        torch.cuda.current_stream().synchronize()
        dt = _MODELS[case["model"]][1]
        h.solve_constant_rates(state["rate"], np.zeros(6), dt * case["steps"], dt)
        outs = {}
        for name in ("stress", "strain"):
            buf = torch.empty(state["V"], 6, dtype=torch.float64, device=_DEVICE)
            ptr = ctypes.cast(buf.data_ptr(), ctypes.POINTER(ctypes.c_double))
            nat.check(h.lib.ssfft_get_field(h.h, nat.FIELD_IDS[name], ptr, 0))
            outs[name] = _kept(buf, precision)
        return outs
    if kind == "material":
        new = state["solver"](state["material"])
        return {name: _kept(torch.from_numpy(new.extract(name).components), precision)
                for name in ("stress", "strain")}
    serving.run_stream(state["server"], state["requests"])
    return [_kept(torch.from_numpy(r.stress), precision) for r in state["requests"]]


# ---- the same in 64 bits, in plain torch ---------------------------------------------------

_R2 = math.sqrt(2.0)
_PAIRS = ((1, 2), (0, 2), (0, 1))


class _Projector:
    """Gamma-hat : tau-hat with t = normalised tan(pi f): t(x)u + u(x)t - (t.u) t(x)t,
    u = tau-hat t; Nyquist planes zero, the zero frequency masked."""

    def __init__(self, dims, mask):
        self.dims = dims
        f = [torch.fft.fftfreq(n, dtype=torch.float64, device=_DEVICE) for n in dims]
        t = torch.stack(torch.meshgrid(*(torch.tan(math.pi * x) for x in f), indexing="ij"))
        keep = torch.ones(dims, dtype=torch.bool, device=_DEVICE)
        for a, n in enumerate(dims):
            if n % 2 == 0:
                keep.select(a, n // 2).zero_()
        keep[0, 0, 0] = False
        half = dims[2] // 2 + 1
        t = torch.where(keep, t, torch.zeros_like(t))[..., :half]
        norm = t.square().sum(0).sqrt()
        self.t = torch.where(norm > 0, t / torch.where(norm > 0, norm, torch.ones_like(norm)),
                             torch.zeros_like(t))
        self.mask = torch.as_tensor(mask, dtype=torch.float64, device=_DEVICE)

    def __call__(self, tau):
        t = self.t
        s = torch.fft.rfftn(tau.reshape(6, *self.dims), dim=(1, 2, 3))
        mean = s[:, 0, 0, 0] * self.mask
        T = {(i, i): s[i] for i in range(3)}
        for k, (i, j) in enumerate(_PAIRS):
            T[i, j] = T[j, i] = s[3 + k] / _R2
        u = [sum(T[i, j] * t[j] for j in range(3)) for i in range(3)]
        tu = sum(t[i] * u[i] for i in range(3))
        o = [2 * t[i] * u[i] - tu * t[i] * t[i] for i in range(3)]
        o += [_R2 * (t[i] * u[j] + u[i] * t[j] - tu * t[i] * t[j]) for i, j in _PAIRS]
        o = torch.stack(o)
        o[:, 0, 0, 0] = mean
        return torch.fft.irfftn(o, s=self.dims, dim=(1, 2, 3)).reshape(6, -1)


def _isotropic():
    E, G = _J2["modulus"], _J2["shear"]
    lam = G * (E - 2 * G) / (3 * G - E)
    C = np.diag([2 * G] * 6)
    C[:3, :3] += lam
    return C


def _rotation_mandel(R):
    """Mandel form of rotations (G, 3, 3) from specimen to crystal components."""
    M = np.empty((len(R), 6, 6))
    basis = []
    for i in range(3):
        b = np.zeros((3, 3))
        b[i, i] = 1.0
        basis.append(b)
    for i, j in _PAIRS:
        b = np.zeros((3, 3))
        b[i, j] = b[j, i] = 1 / _R2
        basis.append(b)
    for a, A in enumerate(basis):
        for c, B in enumerate(basis):
            M[:, a, c] = np.einsum("ij,gik,gjl,kl->g", A, R, R, B)
    return torch.as_tensor(M, device=_DEVICE)


def _schmid():
    """Mandel Schmid tensors of the twelve {111}<110> systems."""
    out = []
    for n in ((1, 1, 1), (-1, 1, 1), (1, -1, 1), (1, 1, -1)):
        for d in ((0, 1, -1), (1, 0, -1), (1, -1, 0), (0, 1, 1), (1, 0, 1), (1, 1, 0)):
            if np.dot(n, d) == 0:
                P = np.outer(d, n) / (_R2 * math.sqrt(3.0))
                P = (P + P.T) / 2
                out.append([P[0, 0], P[1, 1], P[2, 2], _R2 * P[1, 2], _R2 * P[0, 2], _R2 * P[0, 1]])
    return torch.tensor(out, dtype=torch.float64, device=_DEVICE)


class _Plain:
    """Point-wise material response: backward Euler to full convergence."""

    def __init__(self, model, rotations, grain, phase):
        index = torch.as_tensor(grain.astype(np.int64), device=_DEVICE)
        V = len(grain)
        self.model = model
        self.R = _rotation_mandel(rotations)[index]
        soft = torch.ones(V, dtype=torch.bool, device=_DEVICE)
        if phase is not None:
            soft = torch.as_tensor(phase, device=_DEVICE) == 0
        if model == "elastic":
            soft = ~soft
        scale = {"twophase": 10.0, "j2": 1000.0}.get(model, 1.0)
        C = torch.as_tensor(_cubic(), device=_DEVICE)
        turn = lambda A: self.R.mT @ A @ self.R
        self.K0 = turn(torch.where(soft[:, None, None], C, scale * C))
        if model == "j2":
            self.K0[soft] = torch.as_tensor(_isotropic(), device=_DEVICE)
        self.soft, self.C = soft.nonzero()[:, 0], C
        self.ep = torch.zeros(V, 6, dtype=torch.float64, device=_DEVICE)
        self.G = torch.zeros(V, dtype=torch.float64, device=_DEVICE)
        self.g = torch.full((V,), _EVP["resistance"] if model != "j2" else _J2["yield"],
                            dtype=torch.float64, device=_DEVICE)

    def __call__(self, eps, guess, dt):
        """Stress (6, V), tangent (V, 6, 6); the trial state is kept for commit()."""
        K = self.K0.clone()
        sig = (K @ eps.T[..., None])[..., 0]
        v = self.soft
        self.trial = None
        if len(v) and self.model == "j2":
            sig[v], K[v] = self._j2(eps.T[v])
        elif len(v):
            R = self.R[v]
            s, k = self._crystal((R @ eps.T[v][..., None])[..., 0],
                                 (R @ guess.T[v][..., None])[..., 0], dt)
            sig[v] = (R.mT @ s[..., None])[..., 0]
            K[v] = R.mT @ k @ R
        return sig.T.contiguous(), K

    def commit(self):
        if self.trial is not None:
            v = self.soft
            self.ep[v], self.G[v], self.g[v] = self.trial

    def _j2(self, eps):
        v, G, H = self.soft, _J2["shear"], _J2["hardening"]
        bulk = G * _J2["modulus"] / (3 * (3 * G - _J2["modulus"]))
        one = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=torch.float64, device=_DEVICE)
        e = eps - self.ep[v]
        tr = e[:, :3].sum(1)
        s = 2 * G * (e - tr[:, None] / 3 * one)
        q = math.sqrt(1.5) * s.norm(dim=1)
        # the return mapping's first update, whose residual is clipped at zero from then on
        # (the hardening raises the yield stress past it), so it stands
        dp = ((q - self.g[v]) / (3 * G)).clamp(min=0.0)
        safe = torch.where(q > 0, q, torch.ones_like(q))
        self.trial = (self.ep[v] + 1.5 * dp[:, None] * s / safe[:, None], self.G[v] + dp,
                      self.g[v] + H * dp)
        ratio = 3 * G / safe
        dev = torch.eye(6, dtype=torch.float64, device=_DEVICE) - torch.outer(one, one) / 3
        t1 = (2 * G * ratio * dp)[:, None, None]
        t2 = torch.where(dp > 0, ratio ** 2 * (dp / safe - 1 / (3 * G)), 0.0)[:, None, None]
        K = torch.as_tensor(_isotropic(), device=_DEVICE) - t1 * dev + t2 * s[:, :, None] * s[:, None, :]
        return (1 - ratio * dp)[:, None] * s + (bulk * tr)[:, None] * one, K

    def _crystal(self, eps, sig, dt):
        """Newton on the stress; the slip resistance follows the last iterate."""
        v, P, n = self.soft, _schmid(), _EVP["exponent"]
        Ci = torch.linalg.inv(self.C)
        tau1, th0 = _EVP["voce"]["tau_1"], _EVP["voce"]["theta_0"]
        g = self.g[v].clone()
        PP = (P[:, :, None] * P[:, None, :]).reshape(12, 36)
        for _ in range(100):
            tau = sig @ P.T
            pref = _EVP["rate"] * (tau.abs() / g[:, None]) ** (n - 1) / g[:, None]
            rate = pref * tau
            ep = self.ep[v] + dt * rate @ P
            M = Ci + (dt * n * pref @ PP).reshape(-1, 6, 6)
            L = torch.linalg.cholesky(M)
            z = torch.cholesky_solve((sig @ Ci - (eps - ep))[..., None], L)[..., 0]
            sig = sig - z
            inc = dt * rate.abs().sum(1)
            g_new = self.g[v] - tau1 * torch.exp(-th0 / tau1 * self.G[v]) * torch.expm1(-th0 / tau1 * inc)
            done = float((z.norm(dim=1) / sig.norm(dim=1).clamp(min=1e-12)).max()) < 1e-12 and \
                float((g_new - g).abs().max()) < 1e-13
            g = g_new
            if done:
                break
        self.trial = (ep, self.G[v] + inc, g)
        return sig, torch.cholesky_inverse(L)


def _plain_solve(dims, mask, rate, model, micro, dt, steps):
    """Total strain and stress after the increments, (V, 6) each: Newton with conjugate
    gradients on compatible strains, both to round-off."""
    project, law = _Projector(dims, mask), _Plain(model, *micro)
    V = math.prod(dims)
    d = torch.as_tensor(rate * dt, device=_DEVICE)[:, None]
    eps = torch.zeros(6, V, dtype=torch.float64, device=_DEVICE)
    fluct, sig = torch.zeros_like(eps), None
    apply = lambda K, x: (K @ x.T[..., None])[..., 0].T
    for _ in range(steps):
        eps = eps + d + fluct
        fluct_now = fluct.clone()
        if sig is None:
            sig = apply(law.K0, d.expand(6, V))
        for _ in range(40):
            sig, K = law(eps, sig, dt)
            r = -project(sig)
            size = float(r.square().sum().sqrt())
            if size < 1e-11 * float(sig.square().sum().sqrt()):
                break
            x, p, rr = torch.zeros_like(r), r.clone(), size ** 2
            r0 = rr
            for _ in range(400):
                Kp = project(apply(K, p))
                a = rr / float((p * Kp).sum())
                x += a * p
                r -= a * Kp
                new = float(r.square().sum())
                if new < 1e-20 * r0:
                    break
                p = r + new / rr * p
                rr = new
            eps = eps + x
            fluct_now = fluct_now + x
        law.commit()
        fluct = fluct_now
    return {"stress": sig.T.contiguous(), "strain": eps.T.contiguous()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        outs = []
        for i, (n, model, biaxial) in enumerate(_serve_mix(case)):
            if model != "elastic":  # a minute or more for each
                outs.append(None)
                continue
            mask, rate = _load(model, biaxial)
            micro = _microstructure((n, n, n), 20 + 40 * i, model, _serve_seed(seed, i))
            outs.append(_plain_solve((n, n, n), mask, rate, model, micro, _MODELS[model][1],
                                     case["steps"])["stress"])
        return outs
    dims = _dims(case)
    if kind == "projection":
        gen = torch.Generator(_DEVICE).manual_seed(int(seed))
        dtype = torch.float32 if case["precision"] == "mixed" else torch.float64
        tau = torch.randn(6, math.prod(dims), dtype=dtype, device=_DEVICE, generator=gen)
        return _Projector(dims, _load("elastic", False)[0])(tau.double())
    model = case["model"]
    if model == "twophase" or (model == "evp" and case["biaxial"]):
        return None  # increments may be cut back: no fixed sequence of them to restate
    if model == "evp" and math.prod(dims) * case["steps"] > 600_000:
        return None  # over about 20 seconds
    mask, rate = _load(model, case["biaxial"])
    return _plain_solve(dims, mask, rate, model,
                        _microstructure(dims, case["grains"], model, seed), _MODELS[model][1],
                        case["steps"])
