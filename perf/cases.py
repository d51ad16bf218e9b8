"""The work that users of this framework have it do, as measurable cases.

A case is one call, or the few calls of one turn of a user's loop, through the
public Python surface of the library (spooky_b200):

  mainloop  Supervisor.executeMainLoop: steps with the host reading the time
            after each, as the command line runs them
  steps     Context.advance: steps without host synchronisation, then the state
  rhs       Context.compute_dfield: the right-hand side of a caller's state
  outputs   real fields, energies and shell spectra of a state (an output time)
  ensemble  Ensemble.advance of independent boxes of mixed sizes
  closure   Context.advance with the learned tensor-network closure
  train     one loss and gradient of that network over a set of samples

physics: "hd", "mhd" (incompressible, 2/3 dealiasing, low-storage RK3, CFL dt)
or "mti" (Boussinesq MHD, anisotropic conduction of theta by RKL2 cycles
before odd and after even steps).  form: "plain" (FP64 passes) or "fp32" (FP32
passes, FP64 state).  outside: the state carries content outside the 2/3 mask.

exact() restates the equations in 64-bit torch on the same inputs.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spooky-git_b200"))
import spooky_b200 as S  # noqa: E402
from spooky_b200.closure import init_params3  # noqa: E402
from spooky_b200.params import SPK_FORM_FP32, SPK_FORM_PLAIN, default_params  # noqa: E402

BOX_SIZES = (16, 24, 32, 48, 64)             # boxes of an ensemble
LENGTHS = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)


def _case(call, nx, ny, nz, physics="mhd", form="fp32", steps=1, outside=False, count=0):
    return {"call": call, "nx": nx, "ny": ny, "nz": nz, "physics": physics, "form": form, "steps": steps,
            "outside": outside, "count": count}


def listed():
    def named(name, *a, **k):
        return {"name": name, **_case(*a, **k)}
    return [
        # a small decaying-turbulence run from the command line: launch latency and host reads
        named("mainloop_hd32_plain", "mainloop", 32, 32, 32, "hd", "plain", steps=10),
        # a long, thin box with mixed lengths whose state fills the whole spectrum
        named("steps_mhd96x48x192_fp32", "steps", 96, 48, 192, "mhd", "fp32", steps=4, outside=True),
        # the convergence runs at 128^3 in the reference's precision
        named("steps_mhd128_plain", "steps", 128, 128, 128, "mhd", "plain", steps=4),
        # an embedding code that has its own integrator
        named("rhs_mhd128_fp32", "rhs", 128, 128, 128, "mhd", "fp32"),
        # the headline turbulence run, in both forms
        named("steps_mhd256_fp32", "steps", 256, 256, 256, "mhd", "fp32", steps=4),
        named("steps_mhd256_plain", "steps", 256, 256, 256, "mhd", "plain", steps=2),
        # the largest production box here: hydrodynamic turbulence
        named("steps_hd512_fp32", "steps", 512, 512, 512, "hd", "fp32", steps=2),
        # stratified plasma with field-aligned conduction by super-time-stepping
        named("steps_mti256_fp32", "steps", 256, 256, 256, "mti", "fp32", steps=2, outside=True),
        # a parameter study: many small boxes, mixed sizes, HD and MHD
        named("ensemble512_fp32", "ensemble", 16, 16, 16, "mhd", "fp32", steps=4, count=512),
        # a coarse run with the trained closure in its right-hand side
        named("closure_mhd64_fp32", "closure", 64, 64, 64, "mhd", "fp32", steps=4),
        # fitting that closure: forward and backward over the samples of one 64^3 snapshot
        named("train_262144", "train", 64, 64, 64, "mhd", "fp32", count=262144),
        # an output time of the headline run
        named("outputs_mhd256_fp32", "outputs", 256, 256, 256, "mhd", "fp32"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choice(["mainloop", "steps", "steps", "steps", "steps", "rhs", "rhs", "outputs", "ensemble", "closure",
                       "train", "mti"])
    form = rng.choice(["plain", "fp32"])
    if call == "train":
        return _case("train", 64, 64, 64, "mhd", "fp32", count=int(_log_uniform(rng, 2000, 400000)))
    if call == "ensemble":
        return _case("ensemble", 16, 16, 16, "mhd", form, steps=rng.randint(2, 4),
                     count=int(_log_uniform(rng, 10, 300)))
    top = {"mainloop": 64, "closure": 96, "mti": 192}.get(call, 512)
    low = 32 if call in ("closure", "mti") else 16
    while True:
        n = [min(LENGTHS, key=lambda v: abs(math.log(v) - x)) for x in
             (math.log(_log_uniform(rng, low, top)) for _ in range(3))]
        if n[0] * n[1] * n[2] <= 2 ** 24:
            break
    if call == "mti":
        return _case("steps", *n, "mti", form, steps=2, outside=True)
    physics = "mhd" if call == "closure" else rng.choice(["hd", "mhd"])
    steps = {"mainloop": 10, "steps": rng.randint(2, 5), "closure": 4}.get(call, 1)
    return _case(call, *n, physics, form, steps=steps, outside=call in ("steps", "rhs") and rng.random() < 0.3)


# ---------------------------------------------------------------------------
# parameters and inputs
# ---------------------------------------------------------------------------
L = 2 * math.pi


def _params(case, n=None, physics=None, nu=1e-3, eta=1e-3):
    physics = physics or case["physics"]
    kw = dict(incompressible=1, mhd=int(physics != "hd"), gridsize=n or (case["nx"], case["ny"], case["nz"]),
              boxsize=(L, L, L), reynolds=1.0 / nu, reynolds_magnetic=1.0 / eta, cfl=1.5, t_final=1e30,
              toutput_flow=1e30, form=SPK_FORM_FP32 if case["form"] == "fp32" else SPK_FORM_PLAIN)
    if physics == "mti":
        kw.update(boussinesq=1, stratification=1, strat_direction=2, anisotropic_diffusion=1, supertimestepping=1,
                  sts_variables=["th"], safety_sts=95, reynolds_ani=20.0, N2=1.0, OmegaT2=1.0, reynolds=1e4,
                  reynolds_magnetic=1e4)
    if case["call"] == "closure":
        kw.update(closure=3, reynolds=5e3, reynolds_magnetic=5e3)
    if case["call"] == "mainloop":
        kw.update(reynolds=100.0, reynolds_magnetic=100.0, fixed_dt=1e-3)
    return default_params(**kw)


def _axis(n, length, half):
    k = torch.arange(n // 2 + 1) if half else torch.fft.fftfreq(n, 1.0 / n)
    k = (k.to(torch.float64) * (2 * math.pi / length)).cuda()
    return k, (k.abs() <= (2.0 / 3.0) * (2 * math.pi / length * (n // 2 - 1))).to(torch.float64)


class _Grid:
    """Wavevectors (i, j, k < nz/2 + 1) and the 2/3 mask of a box."""

    def __init__(self, p):
        (kx, mx), (ky, my), (kz, mz) = _axis(p.nx, p.lx, 0), _axis(p.ny, p.ly, 0), _axis(p.nz, p.lz, 1)
        self.k = [kx[:, None, None], ky[None, :, None], kz[None, None, :]]
        self.k2 = sum(k * k for k in self.k)
        self.ik2 = torch.where(self.k2 > 0, 1.0 / self.k2.clamp_min(1e-300), torch.ones_like(self.k2))
        self.mask = mx[:, None, None] * my[None, :, None] * mz[None, None, :]
        self.n = (p.nx, p.ny, p.nz)
        self.kmax = [2.0 / 3.0 * 2 * math.pi / a * (n // 2 - 1) for a, n in zip((p.lx, p.ly, p.lz), self.n)]

    def project(self, V):
        """V [..., 3, modes] made divergence-free, in place."""
        s = sum(self.k[c] * V[..., c, :, :, :] for c in range(3)) * self.ik2
        for c in range(3):
            V[..., c, :, :, :] -= self.k[c] * s
        return V

    def real(self, X):
        X = torch.fft.ifftn(X, dim=(-3, -2))
        X[..., 0].imag = 0              # a line's mean and Nyquist mode are real
        X[..., self.n[2] // 2].imag = 0
        return torch.fft.irfft(X, n=self.n[2], dim=-1)

    def spec(self, R):
        return torch.fft.rfftn(R, dim=(-3, -2, -1))


def _solenoidal(g, gen, nb=1, kpeak=4.0):
    """Random solenoidal fields [nb, 3, modes] inside the mask, E(k) ~ k^4 exp(-2 (k/kpeak)^2), rms 1 a component."""
    k = g.k2.sqrt()
    V = g.spec(torch.randn((nb, 3) + g.n, generator=gen, device="cuda", dtype=torch.float64))
    V *= k * torch.exp(-(k / kpeak) ** 2) * g.mask
    g.project(V)
    for b in range(nb):
        V[b] /= math.sqrt(sum(float(g.real(V[b, c]).square().mean()) for c in range(3)) / 3)
    return V


def _state(case, p, seed, nb=1):
    """Initial spectral states [nb, fields, modes]."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    g = _Grid(p)
    N = p.nx * p.ny * p.nz
    if p.boussinesq:   # white noise in u and theta on a weak uniform field along x
        U = torch.zeros((nb, 7) + tuple(g.mask.shape), dtype=torch.complex128, device="cuda")
        for f in (0, 1, 2, 6):
            U[:, f] = g.spec(1e-4 * torch.randn((nb,) + g.n, generator=gen, device="cuda", dtype=torch.float64))
        U[:, 3, 0, 0, 0] = 1e-3 * N
        return U
    U = _solenoidal(g, gen, nb)
    if p.mhd:
        B = _solenoidal(g, gen, nb)
        B[:, 2, 0, 0, 0] += 0.1 * N
        U = torch.cat([U, B], dim=1)
        del B
    if case["outside"]:
        for f in range(0, U.shape[1], 3):
            W = g.spec(torch.randn((nb, 3) + g.n, generator=gen, device="cuda", dtype=torch.float64)) * (1 - g.mask)
            g.project(W)
            U[:, f:f + 3] += W * (1e-3 * U[:, f:f + 3].norm() / W.norm())
    return U


def _boxes(case):
    """(params, size, physics) of each box of an ensemble; sizes and modules interleaved."""
    out = []
    for i in range(case["count"]):
        n, physics = BOX_SIZES[i % 5], "mhd" if (i // 5) % 2 else "hd"
        u = (i * 0.6180339887498949) % 1.0   # nu, eta spread over [1e-4, 1e-2]
        out.append((_params(case, (n, n, n), physics, 10 ** (-4 + 2 * u), 10 ** (-2 - 2 * u)), n, physics))
    return out


def _groups(case):
    """{(size, physics): box indices}"""
    got = {}
    for i, (_, n, physics) in enumerate(_boxes(case)):
        got.setdefault((n, physics), []).append(i)
    return got


def _ensemble_states(case, seed):
    boxes, states = _boxes(case), {}
    for q, (_, ids) in enumerate(sorted(_groups(case).items())):
        U = _state(case, boxes[ids[0]][0], seed * 64 + q, len(ids))
        states.update({i: U[b] for b, i in enumerate(ids)})
    return [states[i] for i in range(len(boxes))]


def _samples(case, seed):
    """Closure training samples [51, count]: random gradients, a noisy eddy stress and EMF as targets."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    n = case["count"]
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=torch.float32)  # noqa: E731
    A, G = rnd(3, 3, n), rnd(3, 3, n)
    for M in (A, G):
        M -= torch.eye(3, device="cuda")[:, :, None] * (M[0, 0] + M[1, 1] + M[2, 2]) / 3
    norm, S5, J = _strain(A.double(), G.double())
    sc = (0.01 * norm).float()
    X = torch.empty((51, n), dtype=torch.float32, device="cuda")
    X[0:8] = 0.0
    X[8:13], X[13:16], X[16] = S5.float(), J.float(), sc
    X[17:22] = -0.02 * sc * X[8:13] + 0.02 * sc * norm.float() * rnd(5, n)
    X[22:25] = -0.02 * sc * X[13:16] + 0.02 * sc * norm.float() * rnd(3, n)
    X[25:30], X[30:33] = X[8:13], X[13:16]
    X[33:42], X[42:51] = A.reshape(9, n), G.reshape(9, n)
    return X


def prepare(case, seed):
    call = case["call"]
    if call == "train":
        tr = S.Trainer(init_params3(seed=seed % 1000, out=0.5), variant=3)
        tr.set_samples(_samples(case, seed), (1e4, 1e4, 1e4))
        return {"case": case, "trainer": tr}
    if call == "ensemble":
        ens = S.Ensemble([p for p, _, _ in _boxes(case)])
        states = _ensemble_states(case, seed)
        for b, U in zip(ens.boxes, states):
            b.set_state(U)
        out = torch.empty(sum(U.numel() for U in states), dtype=torch.complex128, device="cuda")
        at, views = 0, []
        for U in states:
            views.append(out[at:at + U.numel()])
            at += U.numel()
        torch.cuda.synchronize()   # the states may be freed
        return {"case": case, "ens": ens, "out": out, "views": views}
    p = _params(case)
    U = _state(case, p, seed)[0]
    if call == "rhs":
        return {"case": case, "ctx": S.Context(p), "U": U, "dU": torch.empty_like(U)}
    st = {"case": case}
    if call == "mainloop":
        st["sup"] = S.Supervisor(p, toutput_time=1e30)
        ctx = st["ctx"] = st["sup"].ctx
    else:
        ctx = st["ctx"] = S.Context(p)
    if call == "closure":
        ctx.closure_set(init_params3(seed=seed % 1000, out=1.0))
    ctx.set_state(U)
    if call == "outputs":
        ctx.clean_divergence()
        st["R"] = torch.empty(ctx.shape_r, dtype=torch.float64, device="cuda")
    else:
        st["out"] = torch.empty_like(U)
    ctx.synchronize()              # U may be freed
    return st


def run(st):
    case = st["case"]
    call = case["call"]
    if call == "train":
        loss, grad = st["trainer"].loss_grad()
        return {"loss": loss, "grad": grad}
    if call == "ensemble":
        ens = st["ens"]
        ens.advance(case["steps"])
        for i, v in enumerate(st["views"]):
            ens._check(S.lib().spk_ensemble_get_state(ens._h, i, v.data_ptr(), 0))
        return st["out"]
    ctx = st["ctx"]
    if call == "rhs":
        ctx.compute_dfield(st["U"], st["dU"])
        return st["dU"]
    if call == "outputs":
        ctx.to_real(st["R"])
        energy, dissipation = ctx.budgets()
        return {"R": st["R"], "energy": energy, "dissipation": dissipation,
                "spectra": np.stack([ctx.spectrum(f)[0] for f in range(ctx.F)])}
    if call == "mainloop":
        st["sup"].executeMainLoop(max_steps=case["steps"])
    else:
        ctx.advance(case["steps"])
    return ctx.get_state(st["out"])


def _fields(physics):
    return {"hd": 3, "mhd": 6, "mti": 7}[physics]


def work(case):
    def box(n, physics):
        nr, nc, F = n[0] * n[1] * n[2], n[0] * n[1] * (n[2] // 2 + 1), _fields(physics)
        nfft = {"hd": 8, "mhd": 14, "mti": 18}[physics]        # transforms of one right-hand side
        fft = 2.5 * nr * math.log2(nr)
        return nc, F, fft, nfft
    if case["call"] == "train":
        n = case["count"]
        return {"bytes": 4.0 * (51 - 8) * n, "flops": 6.0 * n * (18 * 64 + 2 * 64 * 64 + 64 * 12)}
    if case["call"] == "ensemble":
        got = [box((n, n, n), physics) for _, n, physics in _boxes(case)]
        return {"bytes": case["steps"] * sum(2 * 16.0 * F * nc for nc, F, _, _ in got),
                "flops": case["steps"] * sum(3 * nfft * fft for _, _, fft, nfft in got)}
    nc, F, fft, nfft = box((case["nx"], case["ny"], case["nz"]), case["physics"])
    if case["call"] == "outputs":
        return {"bytes": 16.0 * F * nc + 8.0 * F * case["nx"] * case["ny"] * case["nz"], "flops": F * fft}
    if case["call"] == "rhs":
        return {"bytes": 32.0 * F * nc, "flops": nfft * fft}
    flops = 3 * nfft * fft
    if case["physics"] == "mti":
        flops += 19 * 6 * fft       # the conduction stages of a cycle
    if case["call"] == "closure":
        flops += 3 * 2.0 * case["nx"] * case["ny"] * case["nz"] * (18 * 64 + 2 * 64 * 64 + 64 * 12)
    return {"bytes": case["steps"] * 32.0 * F * nc, "flops": case["steps"] * flops}


def tolerance(case):
    # about four times the difference from exact() over the ranges above
    if case["call"] == "train":
        return {"rel": 1.5e-3, "max": 2e-2}
    if case["call"] == "closure":
        return {"rel": 2.5e-4, "max": 4e-3}
    if case["form"] == "plain":
        if case["call"] in ("rhs", "outputs"):
            return {"rel": 3e-14, "max": 5e-12}
        return {"rel": 8e-16, "max": 4e-14}
    if case["call"] == "rhs":
        return {"rel": 2e-5, "max": 2.5e-3}
    if case["call"] == "outputs":
        return {"rel": 7e-7, "max": 4e-6}
    return {"rel": 1.2e-7, "max": 2.5e-5}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _strain(A, G):
    """n, strain (xx xy xz yy yz) and current of gradients A = grad u, G = grad B ([3, 3, ...])."""
    S5 = torch.stack([A[0, 0], (A[0, 1] + A[1, 0]) / 2, (A[0, 2] + A[2, 0]) / 2, A[1, 1], (A[1, 2] + A[2, 1]) / 2])
    J = torch.stack([G[2, 1] - G[1, 2], G[0, 2] - G[2, 0], G[1, 0] - G[0, 1]])
    n2 = A.square().sum((0, 1)) + G.square().sum((0, 1))   # S:S + |w|^2/2, and the same of B
    return (n2 + 1e-30).sqrt(), S5, J


def _bf16(x):
    """x rounded to BF16; the gradient passes as if it were not."""
    return x + (x.detach().to(torch.bfloat16).to(x.dtype) - x.detach())


def _network(w, x):
    """The tensor network's 12 outputs for inputs x [18, points]; w: flat parameters."""
    at, h = 0, x
    for n_out, n_in in ((64, 18), (64, 64), (64, 64), (12, 64)):
        W = w[at:at + n_out * n_in].reshape(n_out, n_in)
        b = w[at + n_out * n_in:at + n_out * n_in + n_out]
        at += n_out * n_in + n_out
        h = _bf16(W) @ _bf16(h) + b[:, None]
        if n_out == 64:
            h = torch.tanh(h)
    return h


def _stress_emf(s):
    tr = (s[0] + s[3] + s[5]) / 3
    return (torch.stack([s[0] - tr, s[1], s[2], s[3] - tr, s[4]]),
            torch.stack([(s[9] - s[11]) / 2, (s[10] - s[7]) / 2, (s[6] - s[8]) / 2]))


def _dot5(a, b):
    """The full contraction of two traceless symmetric tensors given as xx xy xz yy yz."""
    return a[0] * b[0] + a[3] * b[3] + (a[0] + a[3]) * (b[0] + b[3]) + 2 * (a[1] * b[1] + a[2] * b[2] + a[4] * b[4])


class _Run:
    """Steps of a batch of boxes U [nb, F, modes] in 64 bits; nu, eta: one value a box."""

    def __init__(self, p, U, nu, eta, weights=None):
        self.p, self.g, self.U, self.weights = p, _Grid(p), U, weights
        self.nu, self.eta = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (nu, eta))
        self.step_no = 0
        self.clean(self.U)

    def clean(self, U):
        self.g.project(U[:, 0:3])
        if self.p.mhd:
            self.g.project(U[:, 3:6])

    def rhs(self, U, want_dt=False, theta=None):
        """theta: real values that u theta takes in place of the state's."""
        p, g = self.p, self.g
        nb = U.shape[0]
        bc = lambda v: v.reshape(nb, 1, 1, 1)  # noqa: E731
        R = torch.stack([g.real(U[:, f]) for f in range(U.shape[1])], 1)
        u = [R[:, c] for c in range(3)]
        b = [R[:, 3 + c] for c in range(3)] if p.mhd else None
        if want_dt:
            self.rates = [R[:, c].abs().flatten(1).amax(1) for c in range(min(6, U.shape[1]))]
        T = {}
        for i in range(3):
            for j in range(i, 3):
                T[i, j] = u[i] * u[j] - (b[i] * b[j] if p.mhd else 0.0)
        tr = (T[0, 0] + T[1, 1] + T[2, 2]) / 3
        for i in range(3):
            T[i, i] = T[i, i] - tr
        E = [u[(i + 1) % 3] * b[(i + 2) % 3] - u[(i + 2) % 3] * b[(i + 1) % 3] for i in range(3)] if p.mhd else None
        if self.weights is not None:
            grad = lambda f0: torch.stack([torch.stack([g.real(1j * g.k[j] * U[0, f0 + i]) for j in range(3)])  # noqa: E731
                                           for i in range(3)])
            A, G = grad(0), grad(3)
            n, S5, J = _strain(A, G)
            pts = (3, 3, -1)
            x = torch.cat([A.reshape(9, -1), G.reshape(9, -1)]) / n.reshape(1, -1)
            d2 = (math.pi ** 3 / (g.kmax[0] * g.kmax[1] * g.kmax[2])) ** (2.0 / 3.0)
            with torch.no_grad():
                o = _network(self.weights, x).reshape((12,) + n.shape)
            dT, dE = _stress_emf(d2 * n * n * o)
            P = -_dot5(dT, S5) - (dE * J).sum(0)
            Pm = (_dot5(dT, dT) * _dot5(S5, S5)).sqrt() + ((dE * dE).sum(0) * (J * J).sum(0)).sqrt()
            r = (P / (0.1 * Pm + 1e-30)).clamp(0, 1)
            dT, dE = r * dT, r * dE
            for c, ij in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2))):
                T[ij] = T[ij] + dT[c]
            T[2, 2] = -(T[0, 0] + T[1, 1])
            E = [E[c] + dE[c] for c in range(3)]
            if want_dt:
                self.eddy = float((_dot5(dT, dT).sqrt() / (2 * n)).max()) + float(((dE * dE).sum(0).sqrt() / n).max())
        T = {ij: g.spec(t) for ij, t in T.items()}
        D = torch.empty_like(U)
        for i in range(3):
            D[:, i] = -1j * g.mask * sum(g.k[j] * T[min(i, j), max(i, j)] for j in range(3))
        if p.boussinesq:
            D[:, 2] -= U[:, 6]
        for i in range(3):
            D[:, i] -= bc(self.nu) * g.k2 * U[:, i]
        g.project(D[:, 0:3])
        if p.mhd:
            E = [g.spec(e) for e in E]
            for i in range(3):
                j, k = (i + 1) % 3, (i + 2) % 3
                D[:, 3 + i] = 1j * g.mask * (g.k[j] * E[k] - g.k[k] * E[j]) - bc(self.eta) * g.k2 * U[:, 3 + i]
        if p.boussinesq:
            th = R[:, 6] if theta is None else theta
            D[:, 6] = -1j * g.mask * sum(g.k[j] * g.spec(u[j] * th) for j in range(3)) + p.N2 * U[:, 2]
        return D

    def dt(self):
        """The CFL step (one a box) from the maxima of the first stage."""
        p, g = self.p, self.g
        rate = sum(g.kmax[c % 3] * m for c, m in enumerate(self.rates))
        par = sum(k * k for k in g.kmax) * (self.nu + (self.eta if p.mhd else 0.0))
        if self.weights is not None:
            par = par + sum(k * k for k in g.kmax) * self.eddy
        if p.boussinesq:
            rate = rate + (math.sqrt(p.N2) + math.sqrt(p.OmegaT2)) / p.safety_source
        dt = torch.minimum(p.cfl / rate, p.cfl_par / par)
        if p.boussinesq:
            self.dt_sts = p.cfl_sts / (sum(k * k for k in g.kmax) / p.reynolds_ani)
            dt = dt.clamp_max(self.dt_sts * p.safety_sts)
        if p.fixed_dt > 0:
            dt = torch.full_like(dt, p.fixed_dt)
        return dt.reshape(-1, 1, 1, 1, 1)

    def conduct(self, dt):
        """One RKL2 cycle of theta."""
        g, p = self.g, self.p
        B = [g.real(self.U[0, 3 + c]) for c in range(3)]
        b2 = sum(v * v for v in B)
        dt_sts = min(self.dt_sts, dt)
        r = dt / dt_sts
        s = 1 + int(4.0 * (1.0 + 2.0 * r) / (1.0 + math.sqrt(9.0 + 16.0 * r)))

        def d(th):
            q = (sum(B[c] * g.real(1j * g.k[c] * th) for c in range(3)) + p.OmegaT2 * B[2]) / (b2 * p.reynolds_ani)
            return 1j * g.mask * sum(g.k[c] * g.spec(q * B[c]) for c in range(3))
        w1 = 4.0 / (s * s + s - 2.0)
        bj = lambda j: 1.0 / 3.0 if j < 3 else 0.5 * (j * j + j - 2.0) / (j * (j + 1.0))  # noqa: E731
        Y0 = self.U[0, 6].clone()
        D0 = d(Y0)
        Ym, Y = Y0, Y0 + dt * w1 / 3.0 * D0
        for j in range(2, s + 1):
            mu = (2.0 * j - 1.0) / j * bj(j) / bj(j - 1)
            nu = -(j - 1.0) / j * bj(j) / bj(j - 2)
            mt = w1 * mu
            Ym, Y = Y, mu * Y + nu * Ym + (1 - mu - nu) * Y0 + dt * mt * d(Y) - dt * (1.0 - bj(j - 1)) * mt * D0
        self.U[0, 6] = Y

    def step(self):
        U, p = self.U, self.p
        D = self.rhs(U, True)
        dt = self.dt()
        if p.boussinesq and self.step_no & 1:
            theta = self.g.real(U[:, 6])   # the first stage keeps the real fields of the dt rule
            self.conduct(float(dt))
            D = self.rhs(U, theta=theta)
        U += 8.0 / 15.0 * dt * D
        W = U - 17.0 / 60.0 * dt * D
        D = self.rhs(U)
        U.copy_(W + 5.0 / 12.0 * dt * D)
        W = U - 5.0 / 12.0 * dt * D
        U.copy_(W + 0.75 * dt * self.rhs(U))
        self.clean(U)
        if p.boussinesq and not self.step_no & 1:
            self.conduct(float(dt))
        self.step_no += 1


def exact(case, seed):
    call = case["call"]
    if call == "train":
        X = _samples(case, seed).double()
        w = torch.from_numpy(init_params3(seed=seed % 1000, out=0.5)).double().cuda().requires_grad_()
        loss = 0.0
        for at in range(0, X.shape[1], 65536):
            x = X[:, at:at + 65536]
            A, G = x[33:42].reshape(3, 3, -1), x[42:51].reshape(3, 3, -1)
            n, _, _ = _strain(A, G)
            dT, dE = _stress_emf(x[16] * n * _network(w, torch.cat([x[33:42], x[42:51]]) / n))
            T, E, Sf, Jf = x[17:22], x[22:25], x[25:30], x[30:33]
            dP = -_dot5(dT - T, Sf) - ((dE - E) * Jf).sum(0)
            part = 1e4 * (_dot5(dT - T, dT - T) + (dE - E).square().sum(0) + dP.square()).sum() / X.shape[1]
            part.backward()
            loss += float(part.detach())
        return {"loss": loss, "grad": w.grad.cpu().numpy()}
    if call == "ensemble":
        boxes, states, done = _boxes(case), _ensemble_states(case, seed), {}
        for (n, physics), ids in _groups(case).items():
            r = _Run(boxes[ids[0]][0], torch.stack([states[i] for i in ids]), [boxes[i][0].nu for i in ids],
                     [boxes[i][0].nu_m for i in ids])
            for _ in range(case["steps"]):
                r.step()
            done.update({i: r.U[b].reshape(-1) for b, i in enumerate(ids)})
        return torch.cat([done[i] for i in range(len(boxes))])
    p = _params(case)
    U = _state(case, p, seed)
    g = _Grid(p)
    if call == "outputs":
        g.project(U[:, 0:3])
        if p.mhd:
            g.project(U[:, 3:6])
        U = U[0]
        N = float(p.nx * p.ny * p.nz)
        a2 = U.real.square() + U.imag.square()
        a2[..., 1:] *= 2
        shell = ((g.k2.sqrt() / (2 * math.pi / min(p.lx, p.ly, p.lz))) + 0.5).to(torch.int64)
        nb = int(math.sqrt(sum(k * k for k in g.kmax)) / (2 * math.pi / min(p.lx, p.ly, p.lz)) + 0.5)
        spectra = torch.stack([torch.bincount(shell.reshape(-1), a.reshape(-1))[:nb] for a in a2 / N ** 2])
        return {"R": torch.stack([g.real(u) for u in U]), "energy": 0.5 * a2.sum((1, 2, 3)) / N ** 2,
                "dissipation": (a2 * g.k2).sum((1, 2, 3)) / N ** 2, "spectra": spectra}
    weights = None
    if call == "closure":
        weights = torch.from_numpy(init_params3(seed=seed % 1000, out=1.0)).double().cuda()
    if call == "rhs":
        r = _Run.__new__(_Run)
        r.p, r.g, r.weights = p, g, None
        r.nu, r.eta = (torch.tensor([v], dtype=torch.float64, device="cuda") for v in (p.nu, p.nu_m))
        return r.rhs(U)[0]
    r = _Run(p, U, [p.nu], [p.nu_m], weights)
    for _ in range(case["steps"]):
        r.step()
    return r.U[0]
