"""The framework's work as its users call it, as cases that can be timed and compared.

A case is one call pattern of the public interface (``Spectral2D``,
``Ensemble``, ``ClosureNet``) at one size and precision:

  rhs       ``compute_rhs``: one right-hand side into a host array
  host      ``integrate_one_step_host`` on page-locked arrays: a host program
            that keeps wC and psiC itself and calls once per step
  run       ``integrate_steps`` then ``get_state``: a run between two outputs
  ensemble  ``Ensemble.integrate_steps``, then every run's state
  les       ``les_integrate_steps`` with the learned closure, then the state
  lesbatch  an ``Ensemble`` with the closure, then every run's state
  grad      ``ClosureNet.grad``: loss and gradient of one training batch

Flows are decaying (or Kolmogorov-forced) turbulence: random phases, E(k) ~
k^4 exp(-2 (k / k0)^2), kinetic energy 0.5, dt at a CFL number of about 0.5.
``exact`` restates the same path with torch in 64 bits.
"""

import math
import os

import numpy as np
import torch

import spectral2d_gb300 as S
from spectral2d_gb300 import closure
from spectral2d_gb300.solver import pinned_array

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(S.__file__)), "data", "closure_les128.npz")
CHANNELS = (2, 32, 32, 32, 32, 32, 1)

# every grid the 3/2 rule supports is nx = 2^a 3^b, a >= 3
SIZES = (24, 32, 48, 64, 72, 96, 128, 144, 192, 216, 256, 288, 384, 432, 512, 576, 648, 768, 864, 1024, 1152, 1296,
         1536, 1728, 2048, 2304, 2592, 3072, 3456, 4096)


def listed():
    return [
        # the smallest call: one right-hand side of a small grid (a user's own time loop or a check); latency
        dict(name="rhs_64_fp64", kind="rhs", n=64, precision="fp64", nu=2e-3),
        # the Taylor-Green-sized grid between two outputs
        dict(name="run_256_fp64", kind="run", n=256, precision="fp64", nu=5e-4, steps=50),
        # the reference's conservative form of the nonlinear term
        dict(name="run_512_fp64_conservative", kind="run", n=512, precision="fp64", nu=2.5e-4, steps=20,
             form="conservative"),
        # a grid that is no power of two (M = 1728 = 2^6 3^3)
        dict(name="host_1152_fp64", kind="host", n=1152, precision="fp64", nu=1e-4),
        # the headline: 2048^2 decaying turbulence, a host program's step
        dict(name="host_2048_fp64", kind="host", n=2048, precision="fp64", nu=1e-4),
        dict(name="host_2048_fp32", kind="host", n=2048, precision="fp32", nu=1e-4),
        # Kolmogorov flow with drag at the largest grid
        dict(name="host_4096_fp64_forced", kind="host", n=4096, precision="fp64", nu=1e-5, alpha=0.1, amp=4.0, kf=4),
        # uneven runs in one batch, both precisions
        dict(name="ensemble_24_fp64", kind="ensemble", n=128, runs=24, precision="fp64", nu=1e-3, steps=20),
        dict(name="ensemble_24_fp32", kind="ensemble", n=128, runs=24, precision="fp32", nu=1e-3, steps=20),
        # the LES with the learned closure, one run (latency) and a batch of runs (throughput)
        dict(name="les_128_fp32", kind="les", n=128, precision="fp32", nu=1e-4, steps=20),
        dict(name="lesbatch_32x256_fp32", kind="lesbatch", n=256, runs=32, precision="fp32", nu=1e-4, steps=8),
        # one training batch of the closure
        dict(name="grad_192_batch64", kind="grad", n=128, batch=64),
    ]


def draw(rng):
    def size(lo, hi):
        t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min((s for s in SIZES if lo <= s <= hi), key=lambda s: abs(math.log(s / t)))

    kind = rng.choice(["rhs", "host", "host", "run", "run", "ensemble", "les", "lesbatch", "grad"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "rhs":
        n = size(24, 512)
        return dict(kind=kind, n=n, precision=prec, nu=round(0.128 / n * rng.uniform(0.8, 1.2), 7))
    if kind == "host":
        n = size(48, 4096)
        c = dict(kind=kind, n=n, precision=prec, nu=round(0.2 / n * rng.uniform(0.8, 1.2), 7))
        if rng.random() < 0.3:
            c.update(alpha=0.1, amp=rng.choice([1.0, 4.0]), kf=rng.choice([2, 4, 6]))
        return c
    if kind == "run":
        n = size(32, 1152)
        c = dict(kind=kind, n=n, precision=prec, nu=round(0.128 / n * rng.uniform(0.8, 1.2), 7),
                 steps=rng.randint(3, 40 if n <= 512 else 10))
        if rng.random() < 0.25:
            c["form"] = "conservative"
        return c
    if kind == "ensemble":
        n = rng.choice([16, 32, 64, 128])
        return dict(kind=kind, n=n, runs=rng.randint(4, 24), precision=prec,
                    nu=round(0.128 / n * rng.uniform(0.8, 1.2), 7), steps=rng.randint(2, 20))
    if kind == "les":
        n = rng.choice([32, 48, 64, 96, 128, 192, 256])
        return dict(kind=kind, n=n, precision=prec, nu=round(rng.uniform(0.8, 1.5) * 1e-4, 7), steps=rng.randint(2, 20))
    if kind == "lesbatch":
        return dict(kind=kind, n=rng.choice([64, 128, 256]), runs=rng.randint(4, 32), precision=prec,
                    nu=round(rng.uniform(0.8, 1.5) * 1e-4, 7), steps=rng.randint(2, 6))
    return dict(kind=kind, n=rng.choice([32, 64, 96, 128]), batch=rng.randint(4, 64))


# ---- inputs ---------------------------------------------------------------
def waves(n, device="cuda"):
    """(kx, ky) of the reference layout (nyG, cISize), int64."""
    M = 3 * n // 2
    kx = torch.arange(M // 2 + 1, device=device)[None, :]
    ky = torch.arange(M, device=device)
    ky = torch.where(ky <= M // 2, ky, ky - M)[:, None]
    return kx, ky


def vorticity(n, seed, tke=0.5):
    """Random-phase vorticity in the reference layout on the GPU, Hermitian on kx = 0, truncated to |k| <= n/2."""
    kx, ky = waves(n)
    k2 = (kx * kx + ky * ky).double()
    k = k2.sqrt()
    k0 = min(10.0, n / 8)
    g = torch.Generator(device="cuda").manual_seed(seed)
    ph = torch.rand(k.shape, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    # |w^|^2 = k^2 |u^|^2 and E(k) is spread over about pi k modes
    amp = k * torch.sqrt(k ** 4 * torch.exp(-2 * (k / k0) ** 2) / k.clamp(min=1.0))
    amp = torch.where((k2 > 0) & (k2 <= (n // 2) ** 2), amp, torch.zeros_like(amp))
    w = torch.polar(amp, ph)
    M = 3 * n // 2
    w[M - torch.arange(1, n // 2 + 1, device="cuda"), 0] = w[1:n // 2 + 1, 0].conj()
    e = (w.abs() ** 2 / k2.clamp(min=1.0))
    e = e[:, 1:].sum() + 0.5 * e[:, 0].sum()
    return w * math.sqrt(tke / float(e))


def step_size(n):
    """About CFL 0.5: max(|u| + |v|) is near 5 at kinetic energy 0.5."""
    return 0.1 * 2 * math.pi / (3 * n // 2)


def ensemble_sizes(case):
    """A third each of n, 2 n and 4 n (n alone for the closure's batches)."""
    if case["kind"] == "lesbatch":
        return [case["n"]] * case["runs"]
    return [case["n"] << (i % 3) for i in range(case["runs"])]


def random_params(rng):
    """Parameters of the closure network in its logical order (W[co, tap, ci] and b per layer)."""
    out = []
    for ci, co in zip(CHANNELS[:-1], CHANNELS[1:]):
        out += [rng.standard_normal(co * 9 * ci) * math.sqrt(2.0 / (9 * ci)), 0.05 * rng.standard_normal(co)]
    return np.concatenate(out).astype(np.float32)


def physical(w, n):
    """(omega, psi) on the collocation grid, in 64 bits."""
    kx, ky = waves(n)
    k2 = (kx * kx + ky * ky).double()
    psi = w / k2.clamp(min=1.0)
    return to_phys(w, n), to_phys(psi, n)


def training_batch(case, seed):
    n, B = case["n"], case["batch"]
    M = 3 * n // 2
    x = torch.empty((B, M, M, 2), dtype=torch.float32)
    t = torch.empty((B, M, M), dtype=torch.float32)
    for b in range(B):
        w, p = physical(vorticity(n, seed * 1000 + 2 * b), n)
        q, _ = physical(vorticity(n, seed * 1000 + 2 * b + 1), n)
        x[b, :, :, 0], x[b, :, :, 1] = (w / w.std()).cpu(), (p / p.std()).cpu()
        t[b] = (0.5 * w / w.std() * p / p.std() + 0.5 * q / q.std()).cpu()
    return x.numpy(), t.numpy(), random_params(np.random.default_rng(seed))


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    st = {"case": case, "dt": step_size(n)}
    if kind == "grad":
        x, t, p = training_batch(case, seed)
        net = S.ClosureNet(3 * n // 2, max_batch=case["batch"], seed=0)
        net.set_params(p)
        st.update(net=net, x=x, t=t)
        return st
    if kind in ("ensemble", "lesbatch"):
        nxs = ensemble_sizes(case)
        nus = [case["nu"] * n / m for m in nxs]
        ens = S.Ensemble(nxs, nus, precision=case["precision"])
        for i, r in enumerate(ens.runs):
            r.set_state(vorticity(nxs[i], seed * 1000 + i).cpu().numpy())
        ens.set_dt([step_size(m) for m in nxs])
        if kind == "lesbatch":
            st["net"] = net = S.ClosureNet(3 * n // 2, max_batch=len(nxs), seed=0)
            closure.load_weights(net, WEIGHTS)
            ens.set_closure(net)
        st["ens"] = ens
        return st
    sim = S.Spectral2D(n, nu=case["nu"], precision=case["precision"], alpha=case.get("alpha", 0.0),
                       forcing_amp=case.get("amp", 0.0), forcing_k=case.get("kf", 0),
                       nonlinear_form=case.get("form", "basdevant"))
    st["sim"] = sim
    w = vorticity(n, seed)
    if kind == "host":
        st["w"], st["psi"] = pinned_array(sim.shape), pinned_array(sim.shape)
        torch.from_numpy(st["w"]).copy_(w)
        return st
    sim.set_state(w.cpu().numpy())
    if kind == "les":
        st["net"] = net = S.ClosureNet(3 * n // 2, max_batch=1, seed=0)
        closure.load_weights(net, WEIGHTS)
        S.les_set_closure(sim, net)
    return st


def run(state):
    case, dt = state["case"], state["dt"]
    kind = case["kind"]
    if kind == "rhs":
        return state["sim"].compute_rhs()
    if kind == "host":
        return state["sim"].integrate_one_step_host(state["w"], dt, state["psi"], inplace=True)
    if kind == "run":
        state["sim"].integrate_steps(case["steps"], dt)
        return state["sim"].get_state()
    if kind == "les":
        S.les_integrate_steps(state["sim"], case["steps"], dt)
        return state["sim"].get_state()
    if kind in ("ensemble", "lesbatch"):
        state["ens"].integrate_steps(case["steps"])
        return [r.get_state() for r in state["ens"].runs]
    return state["net"].grad(state["x"], state["t"])


# ---- what a pass cannot do without ---------------------------------------
def step_work(n, precision, rhs=3):
    """A step reads and writes the retained modes once; each right-hand side is 4 real 2-D FFTs of the padded grid."""
    M, K = 3 * n // 2, n // 2
    return {"bytes": 2.0 * (K + 1) * (2 * K + 1) * (16 if precision == "fp64" else 8),
            "flops": rhs * 4 * 2.5 * M * M * math.log2(float(M) * M)}


def net_flops(pixels):
    return 2.0 * 9 * sum(a * b for a, b in zip(CHANNELS[:-1], CHANNELS[1:])) * pixels


def work(case):
    kind, n = case["kind"], case["n"]
    M = 3 * n // 2
    ref = 16.0 * M * (M // 2 + 1)   # one array of the reference layout
    if kind == "grad":
        px = case["batch"] * float(M) * M
        return {"bytes": 12.0 * px + 8.0 * 37889, "flops": 3 * net_flops(px)}
    if kind == "rhs":
        s = step_work(n, case["precision"], rhs=1)
        return {"bytes": s["bytes"] / 2 + ref, "flops": s["flops"]}
    if kind == "host":
        s = step_work(n, case["precision"])
        K = n // 2
        return {"bytes": 16.0 * (K + 1) * (2 * K + 1) + 2 * ref, "flops": s["flops"]}
    total = {"bytes": 0.0, "flops": 0.0}
    for m in (ensemble_sizes(case) if kind in ("ensemble", "lesbatch") else [n]):
        s = step_work(m, case["precision"])
        Mm = 3 * m // 2
        total["bytes"] += case["steps"] * s["bytes"] + 32.0 * Mm * (Mm // 2 + 1)
        total["flops"] += case["steps"] * s["flops"]
        if kind in ("les", "lesbatch"):
            total["flops"] += case["steps"] * net_flops(float(Mm) * Mm)
    return total


# ---- the same results in 64 bits -----------------------------------------
def to_phys(f, n):
    """Unnormalised inverse transform (y, then x) of a half spectrum."""
    return torch.fft.irfft(torch.fft.ifft(f, dim=0, norm="forward"), n=3 * n // 2, dim=1, norm="forward")


def to_spec(p):
    return torch.fft.fft(torch.fft.rfft(p, dim=1, norm="forward"), dim=0, norm="forward")


class Flow:
    """The equations of one run: dW = -i kx F[u w] - i ky F[v w] - nu k^2 w - alpha w + F."""

    def __init__(self, n, nu, alpha=0.0, amp=0.0, kf=0):
        self.n, self.nu, self.alpha = n, nu, alpha
        kx, ky = waves(n)
        self.kx, self.ky = kx.double(), ky.double()
        self.k2 = self.kx ** 2 + self.ky ** 2
        self.keep = kx * kx + ky * ky <= (n // 2) ** 2
        self.force = None
        if amp:
            M = 3 * n // 2
            c = 0.5 * amp * complex(math.cos(kf * 2 * math.pi / M), math.sin(kf * 2 * math.pi / M))
            self.force = torch.zeros(self.k2.shape, dtype=torch.complex128, device="cuda")
            self.force[kf, 0], self.force[M - kf, 0] = c, c.conjugate()

    def cut(self, f):
        return torch.where(self.keep, f, torch.zeros((), dtype=f.dtype, device=f.device))

    def psi(self, w):
        return w / self.k2.clamp(min=1.0)

    def rhs(self, w, source=None):
        p = self.psi(w)
        wp = to_phys(w, self.n)
        fu = to_spec(to_phys(1j * self.ky * p, self.n) * wp)
        fv = to_spec(to_phys(-1j * self.kx * p, self.n) * wp)
        d = -1j * self.kx * fu - 1j * self.ky * fv - (self.nu * self.k2 + self.alpha) * w
        for extra in (self.force, source):
            if extra is not None:
                d = d + extra
        return self.cut(d)

    def step(self, w, dt, source=None):
        a = self.cut(w + dt * self.rhs(w, source))
        b = self.cut(0.75 * w + 0.25 * a + 0.25 * dt * self.rhs(a, source))
        return self.cut(w / 3 + 2.0 / 3 * b + 2.0 / 3 * dt * self.rhs(b, source))


class Net:
    """The closure network in 64 bits; its weights are BF16 by definition, nothing else is rounded."""

    def __init__(self, p, grad=False):
        self.layers, o = [], 0
        for ci, co in zip(CHANNELS[:-1], CHANNELS[1:]):
            W = torch.from_numpy(p[o:o + co * 9 * ci].copy()).reshape(co, 3, 3, ci)
            W = W.bfloat16().double().permute(0, 3, 1, 2).contiguous().cuda()
            b = torch.from_numpy(p[o + co * 9 * ci:o + co * 9 * ci + co].copy()).double().cuda()
            o += co * 9 * ci + co
            self.layers.append((W.requires_grad_(grad), b.requires_grad_(grad)))

    def __call__(self, x):
        F = torch.nn.functional
        for i, (W, b) in enumerate(self.layers):
            x = F.conv2d(F.pad(x, (1, 1, 1, 1), mode="circular"), W, b)
            if i < len(self.layers) - 1:
                x = F.gelu(x)
        return x[:, 0]


def closure_source(flow, net, scale, band, w):
    """-Pi^ of the state: inputs over the flow's rms vorticity, output times its square, only modes |k| >= band."""
    wp, pp = to_phys(w, flow.n), to_phys(flow.psi(w), flow.n)
    a = wp.square().mean().sqrt()
    y = net(torch.stack([wp / (a * scale[0]), pp / (a * scale[1])])[None])[0]
    s = to_spec(-scale[2] * a * a * y)
    return flow.cut(torch.where(flow.k2 >= band * band, s, torch.zeros_like(s)))


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "grad":
        x, t, p = training_batch(case, seed)
        net = Net(p, grad=True)
        loss = 0.0
        for b in range(0, case["batch"], 4):   # a few images at a time
            xb = torch.from_numpy(x[b:b + 4]).cuda().double().permute(0, 3, 1, 2)
            e = (net(xb) - torch.from_numpy(t[b:b + 4]).cuda().double()).square().sum() / t.size
            e.backward()
            loss += float(e)
        g = [v.grad.permute(0, 2, 3, 1) if v.dim() == 4 else v.grad for W, c in net.layers for v in (W, c)]
        return loss, torch.cat([v.reshape(-1) for v in g]).float().cpu().numpy()
    with torch.no_grad():
        net = scale = band = None
        if kind in ("les", "lesbatch"):
            d = np.load(WEIGHTS)
            net, scale, band = Net(d["params"]), [float(v) for v in d["scales"]], float(d["band"])
        outs = []
        batch = kind in ("ensemble", "lesbatch")
        for i, m in enumerate(ensemble_sizes(case) if batch else [n]):
            flow = Flow(m, case["nu"] * n / m, case.get("alpha", 0.0), case.get("amp", 0.0), case.get("kf", 0))
            w = vorticity(m, seed * 1000 + i if batch else seed)
            if kind == "rhs":
                return flow.rhs(w).cpu().numpy()
            for _ in range(case.get("steps", 1)):
                w = flow.step(w, step_size(m), closure_source(flow, net, scale, band, w) if net else None)
            outs.append((w.cpu().numpy(), flow.psi(w).cpu().numpy()))
        return outs if batch else outs[0]
