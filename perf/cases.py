"""Performance cases of the model: what a user has it do, through its public entry points.

A case is a dict of plain values; ``prepare`` makes what a user's program holds before the call
(a model context, an ensemble or a network, and its inputs, from a seed), ``run`` makes one pass
through the public API, ``exact`` evaluates the same pass in plain 64-bit torch.

Kinds of cases:

* ``model``: ``steps`` TimeStep calls on a host ``q_hat`` (``time_step`` for one step, ``advance``
  for more), as the Fortran driver and the Python module make them.  The step size is held at
  ``dt_max`` (TOL = 1e30, as in the named Phillips workload), so that a pass does a fixed amount
  of work and its result does not hinge on the roundoff of an error estimate; every kernel of an
  adaptive step still runs.  Models whose right-hand sides run in single precision
  (``precision="mixed"``, an attached network) hand out single-precision snapshots on the GPU.
* ``ensemble``: ``steps`` BSRK3 steps of independent members, one launch per pass.
* ``cnn``: the closure network's inference (``forward``) or its loss and gradients
  (``gradients``), which is a training step up to the optimiser.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from qgn_fortran_b200 import QGNModule
from qgn_fortran_b200.closure import ClosureNet, attach
from qgn_fortran_b200.inputs import exponential_stratification, notebook_profiles, phillips_two_layer
from qgn_fortran_b200.model import QGNEnsemble

LEITH_13 = float(np.float32(1.3))   # the reference's single-precision literal


def listed():
    m = dict(kind="model", scheme="ark43_qgleith", precision="fp64", profile="exponential", drag=False, net=0)
    return [
        # the drop-in TimeStep on the closure's coarse grid: host array in and out, launch-bound
        dict(m, name="timestep_128x4", nx=128, ny=128, nz=4, steps=1),
        # the two-layer Phillips workload, fixed hyperviscosity
        dict(m, name="phillips_256x2", nx=256, ny=256, nz=2, steps=40, scheme="ark43", profile="phillips"),
        # a rectangular domain with an odd number of layers, explicit dissipation and quadratic drag
        dict(m, name="bsrk3_512x256x5", nx=512, ny=256, nz=5, steps=20, scheme="bsrk3", drag=True),
        # the reference's default configuration (32 layers of its notebook, quadratic drag) on 512^2
        dict(m, name="notebook_512x32", nx=512, ny=512, nz=32, steps=8, profile="notebook", drag=True),
        # the drop-in TimeStep of the headline workload, one call per step
        dict(m, name="timestep_1024x8", nx=1024, ny=1024, nz=8, steps=1),
        # the headline workload between two outputs
        dict(m, name="advance_1024x8", nx=1024, ny=1024, nz=8, steps=20),
        # the same in mixed precision
        dict(m, name="mixed_1024x8", nx=1024, ny=1024, nz=8, steps=20, precision="mixed"),
        # the largest workload, which is what the mixed precision is for
        dict(m, name="mixed_2048x16", nx=2048, ny=2048, nz=16, steps=10, precision="mixed"),
        # an ensemble of mixed grid sizes and layer counts
        dict(name="ensemble_32_mixed", kind="ensemble", members=32, steps=20, precision="mixed", pick=0),
        # the coarse model under the learned closure
        dict(m, name="closure_128x4", nx=128, ny=128, nz=4, steps=40, net=6),
        # the closure network: offline inference and training at the experiment's batch
        dict(name="cnn_forward_32", kind="cnn", call="forward", nz=4, H=128, W=128, layers=6, batch=32),
        dict(name="cnn_gradients_32", kind="cnn", call="gradients", nz=4, H=128, W=128, layers=6, batch=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "model", "model", "model", "ensemble", "cnn"])
    if kind == "cnn":
        H, W = rng.choice([64, 96, 128, 200, 256]), rng.choice([128, 256])
        most = max(1, 32 * 128 * 128 // (H * W))
        return dict(kind="cnn", call=rng.choice(["forward", "gradients"]), nz=rng.randint(2, 8), H=H, W=W,
                    layers=rng.randint(3, 6), batch=_log_int(rng, 1, most))
    if kind == "ensemble":
        return dict(kind="ensemble", members=_log_int(rng, 2, 32), steps=rng.randint(4, 20),
                    precision=rng.choice(["mixed", "fp64"]), pick=rng.randint(1, 1 << 20))
    nx = 1 << rng.randint(6, 11)
    ny = min(2048, max(64, nx * rng.choice([1, 1, 1, 2]) // rng.choice([1, 1, 2])))
    scheme = rng.choice(["ark43_qgleith", "ark43_qgleith", "ark43", "bsrk3", "rk4", "ab3"])
    profile = "exponential"
    nz = _log_int(rng, 2, 16)
    if rng.random() < 0.2:
        nz, profile = 32, "notebook"
    precision = rng.choice(["fp64", "mixed"]) if scheme.startswith("ark43") else "fp64"
    net = 0
    if nx == ny == 128 and nz <= 8 and scheme == "ark43_qgleith" and precision == "fp64":
        net = rng.choice([0, 6])
    # at most the largest listed case: 10 mixed steps of 2048^2 x 16, an FP64 step costing twice as much
    room = 2048 * 2048 * 16 * 10 * (1.0 if precision == "mixed" else 0.5) * 0.8
    while nx * ny * nz > min(room, 2048 * 2048 * 16):
        nz -= 1
    steps = _log_int(rng, 1, max(1, min(40, int(room / (nx * ny * nz)))))
    return dict(kind="model", nx=nx, ny=ny, nz=nz, scheme=scheme, precision=precision, profile=profile,
                drag=rng.random() < 0.4, net=net, steps=steps)


# ------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _notebook(nz):
    return notebook_profiles(nz)[:3]


def _dt(nx, ny):
    return 900.0 if max(nx, ny) <= 1024 else 450.0


def _configuration(c):
    """Run parameters and background profiles of a model case."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    Lx, beta, Htot = 2.0e6, 2.0e-11, 4000.0
    if c["profile"] == "phillips":
        (H, S, U), Lx, beta = phillips_two_layer(), 1.0e6, 1.6e-11
    elif c["profile"] == "notebook":
        (H, S, U), Lx, Htot = _notebook(nz), 1.3824e6, 4800.0
    else:
        H, S, U = exponential_stratification(nz)
    explicit = c["scheme"] in ("bsrk3", "rk4", "ab3")
    one_day = 1.0 / (86400.0 * (math.pi * nx / Lx) ** 8)   # grid-scale e-folding
    p = dict(nx=nx, ny=ny, nz=nz, Lx=Lx, Ly=Lx * ny / nx, Htot=Htot, f0=1.0e-4, beta=beta, A2=0.0, A8=one_day,
             r0=1.0e-7, C_d=1.0e-5 if c["drag"] else 0.0, TOL=1.0e30, is_explicit=explicit, dt_max=_dt(nx, ny))
    return p, H, S, U


def _random_pv(p, seed, k0=16.0, rms=1.0e-6):
    """Spectrum (on the GPU) of a random PV field of peak wavenumber k0 and the given rms per layer."""
    nx, ny, nz = p["nx"], p["ny"], p["nz"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    i = torch.arange(nx // 2 + 1, dtype=torch.float64, device="cuda")
    j = torch.fft.fftfreq(ny, d=1.0 / ny, dtype=torch.float64, device="cuda") * (p["Lx"] / p["Ly"])
    k = torch.sqrt(i[None, :] ** 2 + j[:, None] ** 2) / min(k0, nx / 8.0)
    amp = k * torch.exp(-0.5 * k * k)
    keep = _kept(nx, ny)
    q = torch.empty((nz, ny, nx // 2 + 1), dtype=torch.complex128, device="cuda")
    for l in range(nz):
        f = torch.randn((ny, nx), dtype=torch.float64, device="cuda", generator=g)
        s = torch.fft.rfft2(f) * amp * keep
        f = torch.fft.irfft2(s, s=(ny, nx))
        q[l] = s * (rms / f.square().mean().sqrt())
    return q


def _kept(nx, ny):
    keep = torch.ones((ny, nx // 2 + 1), dtype=torch.float64, device="cuda")
    keep[:, nx // 3:] = 0.0
    keep[ny // 3:2 * (ny // 3) + 1] = 0.0
    keep[0, 0] = 0.0
    return keep


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _weights(shapes, cin, cout, seed, damping):
    """Weights of the network; with ``damping`` its output is about minus its PV inputs, as of a
    closure that removes enstrophy (GELU(x) - GELU(-x) = x carries the PV through the layers)."""
    g = torch.Generator().manual_seed(seed)
    out = []
    for l, (co, ci) in enumerate(shapes):
        ri, ro = (cin if l == 0 else ci), (cout if l == len(shapes) - 1 else co)
        w, b = torch.zeros((9, co, ci)), torch.zeros(co)
        std = 0.01 if damping else math.sqrt(2.0 / (9 * ri))
        w[:, :ro, :ri] = std * torch.randn((9, ro, ri), generator=g)
        b[:ro] = 0.01 * torch.randn(ro, generator=g)
        if damping:
            for k in range(cout):
                a, n = 2 * k, 2 * k + 1
                if l == 0:
                    w[4, a, k] += 1.0
                    w[4, n, k] -= 1.0
                elif l < len(shapes) - 1:
                    w[4, a, a] += 1.0
                    w[4, a, n] -= 1.0
                    w[4, n, a] -= 1.0
                    w[4, n, n] += 1.0
                else:
                    w[4, k, a] -= 1.0
                    w[4, k, n] += 1.0
        out.append((w.numpy(), b.numpy()))
    return out


def _scales(q, p, H, S):
    """Input scales 1/std of q and psi, and the output scale of a tendency of about q per 20 days."""
    ref = _Reference(p, H, S, np.zeros(len(H)))
    sq = ref.phys(q).std(dim=(1, 2)).cpu().numpy()
    sp = ref.phys(ref.psi(q)).std(dim=(1, 2)).cpu().numpy()
    return np.concatenate([1.0 / sq, 1.0 / sp]).astype(np.float32), (20 * 86400.0 / sq).astype(np.float32)


def _net_shapes(nz, layers):
    return [(16 if l == layers - 1 else 64, 16 if l == 0 else 64) for l in range(layers)]


def _background(p):
    return 1.0 / (3 * 86400.0 * (math.pi * p["nx"] / p["Lx"]) ** 8)


def _members(c):
    """Grids and flows of the ensemble's members: they are the case's, the states are the seed's."""
    out = []
    for m in range(c["members"]):
        rng = np.random.default_rng(1000 + 7919 * c["pick"] + m)
        n, nz = int(rng.choice((128, 256, 512))), int(rng.choice((2, 4, 8)))
        efold, U0 = float(rng.uniform(500.0, 1500.0)), float(rng.uniform(0.02, 0.15))
        H, S, U = exponential_stratification(nz, N_efold=efold, U0=U0, U_efold=efold)
        p = dict(nx=n, ny=n, nz=nz, Lx=2.0e6, Ly=2.0e6, Htot=4000.0, f0=1.0e-4, beta=2.0e-11, A2=0.0,
                 A8=1.0 / (86400.0 * (math.pi * n / 2.0e6) ** 8), r0=1.0e-7, C_d=0.0, TOL=1.0e30,
                 is_explicit=True, dt_max=900.0)
        out.append((p, H, S, U))
    return out


def _member_states(members, seed):
    return [_random_pv(p, 100003 * seed + m, 8.0) for m, (p, _, _, _) in enumerate(members)]


def _samples(c, seed):
    """Network inputs (q and psi of unit variance, smooth on the grid) and targets."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, W, nz = c["batch"], c["H"], c["W"], c["nz"]
    i = torch.arange(W // 2 + 1, device="cuda") / 12.0
    j = torch.fft.fftfreq(H, d=1.0 / H, device="cuda") / 12.0
    amp = torch.exp(-0.5 * (i[None, :] ** 2 + j[:, None] ** 2))

    def fields(n):
        f = torch.fft.irfft2(torch.fft.rfft2(torch.randn((B, n, H, W), device="cuda", generator=g)) * amp, s=(H, W))
        return (f / f.std()).permute(0, 2, 3, 1)

    x = torch.zeros((B, H, W, 16), dtype=torch.bfloat16, device="cuda")
    y = torch.zeros((B, H, W, 16), dtype=torch.float32, device="cuda")
    x[..., :2 * nz] = fields(2 * nz).to(torch.bfloat16)
    y[..., :nz] = fields(nz)
    return x, y


# ------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------
def prepare(case, seed):
    c = case
    if c["kind"] == "cnn":
        net = ClosureNet(nz=c["nz"], H=c["H"], W=c["W"], layers=c["layers"], max_batch=c["batch"], seed=0)
        net.set_weights(_weights(_net_shapes(c["nz"], c["layers"]), 2 * c["nz"], c["nz"], seed, False))
        x, y = _samples(c, seed)
        return {"case": c, "net": net, "x": x, "y": y, "out": torch.empty_like(y)}
    if c["kind"] == "ensemble":
        specs = _members(c)
        members, size = [], 0
        states = _member_states(specs, seed)
        flat = torch.empty(sum(q.numel() for q in states), dtype=torch.complex128, pin_memory=True)
        views = []
        for (p, H, S, U), q in zip(specs, states):
            v = flat[size:size + q.numel()].view(q.shape)
            size += q.numel()
            v.copy_(q)
            m = QGNModule(p, H, S, U, scheme="bsrk3")
            m.set_state(v.numpy(), 0.0, p["dt_max"])
            members.append(m)
            views.append(v.numpy())
        return {"case": c, "ens": QGNEnsemble(members, precision=c["precision"]), "members": members,
                "views": views, "flat": flat}
    p, H, S, U = _configuration(c)
    q = _random_pv(p, seed)
    g = QGNModule(p, H, S, U, scheme=c["scheme"], precision=c["precision"])
    state = {"case": c, "model": g, "host": _pinned(q), "t": 0.0, "dt": p["dt_max"]}
    if c["net"]:
        net = ClosureNet(nz=c["nz"], H=c["ny"], W=c["nx"], layers=c["net"], max_batch=1, seed=0)
        net.set_weights(_weights(_net_shapes(c["nz"], c["net"]), 2 * c["nz"], c["nz"], seed, True))
        in_scale, out_scale = _scales(q, p, H, S)
        attach(g, net, in_scale, out_scale, A8_background=_background(p))
        state["net"] = net
    state["q"] = state["host"].numpy()
    return state


def _single(q):
    """Single-precision snapshot on the GPU of a host state (16 of its digits are not there to keep)."""
    return q.to("cuda", non_blocking=True).to(torch.complex64)


def run(state):
    c = state["case"]
    if c["kind"] == "cnn":
        if c["call"] == "forward":
            state["net"].forward(state["x"], state["out"], c["batch"])
            return state["out"]
        loss, grads = state["net"].gradients(state["x"], state["y"], c["batch"])
        return {"loss": loss, "weights": [w for w, _ in grads], "biases": [b for _, b in grads]}
    if c["kind"] == "ensemble":
        state["ens"].advance(c["steps"])
        for m, v in zip(state["members"], state["views"]):
            m.get_state(v)
        return _single(state["flat"]) if c["precision"] == "mixed" else state["flat"]
    g = state["model"]
    if c["steps"] == 1:
        state["t"], state["dt"] = g.time_step(state["q"], state["t"], state["dt"])
    else:
        state["t"], state["dt"] = g.advance(state["q"], state["t"], state["dt"], c["steps"])
    single = c["precision"] == "mixed" or c["net"]
    return {"q": _single(state["host"]) if single else state["q"], "t": state["t"], "dt": state["dt"]}


# ------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------
RHS_PER_STEP = {"ark43_qgleith": 6, "ark43": 6, "bsrk3": 3, "rk4": 4, "ab3": 1}


def _step_work(p, scheme, steps):
    """State in and out once per step; FLOPs of the five 2-D transforms of a layer's right-hand
    side (5/2 n log2 n each) and of the mode inversion."""
    n, nz = p["nx"] * p["ny"], p["nz"]
    kept = (p["nx"] // 3) * (p["ny"] - p["ny"] // 3 - 1)
    rhs = 5 * nz * 2.5 * n * math.log2(n) + 8.0 * nz * nz * kept
    return 2 * 16.0 * kept * nz * steps, rhs * RHS_PER_STEP[scheme] * steps


def work(case):
    c = case
    if c["kind"] == "cnn":
        flops = sum(2.0 * 9 * co * ci for co, ci in _net_shapes(c["nz"], c["layers"])) * c["batch"] * c["H"] * c["W"]
        pixels = c["batch"] * c["H"] * c["W"]
        if c["call"] == "forward":
            return {"bytes": pixels * 16 * (2 + 4.0), "flops": flops}
        first = 2.0 * 9 * 64 * 16 * pixels      # the first layer's input needs no gradient
        return {"bytes": pixels * 16 * (2 + 4.0), "flops": 3 * flops - first}
    if c["kind"] == "ensemble":
        parts = [_step_work(p, "bsrk3", c["steps"]) for p, _, _, _ in _members(c)]
    else:
        p = _configuration(c)[0]
        parts = [_step_work(p, c["scheme"], c["steps"])]
        if c["net"]:
            flops = sum(2.0 * 9 * co * ci for co, ci in _net_shapes(c["nz"], c["net"]))
            parts.append((0.0, flops * c["nx"] * c["ny"] * c["steps"]))
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


# ------------------------------------------------------------------------------------
# The same in plain 64-bit torch
# ------------------------------------------------------------------------------------
def _tableau():
    """ARK4(3)6L[2]SA (Kennedy and Carpenter, 2003)."""
    ae = np.zeros((6, 6))
    ai = np.zeros((6, 6))
    ae[1, 0] = 0.5
    ae[2, :2] = 13861 / 62500, 6889 / 62500
    ae[3, :3] = -116923316275 / 2393684061468, -2731218467317 / 15368042101831, 9408046702089 / 11113171139209
    ae[4, :4] = (-451086348788 / 2902428689909, -2682348792572 / 7519795681897, 12662868775082 / 11960479115383,
                 3355817975965 / 11060851509271)
    ae[5, :5] = (647845179188 / 3216320057751, 73281519250 / 8382639484533, 552539513391 / 3454668386233,
                 3354512671639 / 8306763924573, 4040 / 17871)
    b = np.array([82889 / 524892, 0, 15625 / 83664, 69875 / 102672, -2260 / 8211, 0.25])
    ai[1, :2] = 0.25, 0.25
    ai[2, :3] = 8611 / 62500, -1743 / 31250, 0.25
    ai[3, :4] = 5012029 / 34652500, -654441 / 2922500, 174375 / 388108, 0.25
    ai[4, :5] = (15267082809 / 155376265600, -71443401 / 120774400, 730878875 / 902184768, 2285395 / 8070912, 0.25)
    ai[5] = b
    return ae, ai, b


class _Reference:
    """The model's right-hand side on full spectra in 64-bit torch."""

    def __init__(self, p, H, S, U):
        self.p = p
        nz, nx, ny = p["nz"], p["nx"], p["ny"]
        H = p["Htot"] * np.asarray(H) / np.sum(H)
        L = np.zeros((nz, nz))
        for k in range(nz):
            if k > 0:
                L[k, k - 1] = 2.0 * S[k] / (H[k] * (H[k] + H[k - 1]))
            if k < nz - 1:
                L[k, k + 1] = 2.0 * S[k + 1] / (H[k] * (H[k] + H[k + 1]))
            L[k, k] = -L[k].sum()
        r = np.sqrt(H)                         # L is symmetric in the thickness-weighted layers
        ev, V = np.linalg.eigh(0.5 * ((L * (r[:, None] / r[None, :])) + (L * (r[:, None] / r[None, :])).T))

        def dev(a):
            return torch.tensor(np.asarray(a), dtype=torch.float64, device="cuda")

        self.ev, self.back, self.proj = dev(ev), dev(V / r[:, None]), dev(V.T * r[None, :])
        self.U, self.Qy = dev(U)[:, None, None], dev(L @ -np.asarray(U))[:, None, None] + p["beta"]
        self.kx = (2 * math.pi / p["Lx"]) * torch.arange(nx // 2 + 1, dtype=torch.float64, device="cuda")[None, :]
        j = torch.arange(ny, device="cuda")
        self.ky = (2 * math.pi / p["Ly"]) * torch.where(j <= ny // 2, j, j - ny).to(torch.float64)[:, None]
        self.k2 = self.kx ** 2 + self.ky ** 2
        self.k8 = self.k2 ** 4
        self.keep = _kept(nx, ny)
        self.Hw = dev(H / p["Htot"])

    def phys(self, f):
        """y transform, then the real x transform of each row."""
        f = torch.fft.ifft(f, dim=-2)
        f[..., 0] = f[..., 0].real.to(f.dtype)
        return torch.fft.irfft(f, n=self.p["nx"], dim=-1)

    def psi(self, q):
        out = torch.zeros_like(q)
        for m in range(self.p["nz"]):
            den = -self.k2 + self.ev[m]
            den[0, 0] = 1.0
            a = torch.zeros_like(q[0])
            for l in range(self.p["nz"]):
                a += self.proj[m, l] * q[l]
            a = a / den * self.keep
            for l in range(self.p["nz"]):
                out[l] += self.back[l, m] * a
        return out

    def rhs(self, q):
        p, out = self.p, torch.empty_like(q)
        psi = self.psi(q)
        ikx, iky = 1j * self.kx, 1j * self.ky
        for l in range(p["nz"]):
            v_hat = ikx * psi[l]
            ql, u, v = self.phys(q[l].clone()), self.phys(-iky * psi[l]), self.phys(v_hat.clone())
            r = -(ikx * torch.fft.rfft2(u * ql) + iky * torch.fft.rfft2(v * ql))
            r = r - self.U[l] * ikx * q[l] - self.Qy[l] * v_hat
            if p["is_explicit"]:
                r = r - (p["A2"] * self.k2 + p["A8"] * self.k8) * q[l]
            if l == p["nz"] - 1:
                r = r + (p["r0"] / self.Hw[l]) * self.k2 * psi[l]
                if p["C_d"]:
                    s = torch.sqrt(u * u + v * v)
                    r = r + (p["C_d"] / self.Hw[l]) * (iky * torch.fft.rfft2(s * u) - ikx * torch.fft.rfft2(s * v))
            out[l] = r * self.keep
        return out

    def leith(self, q):
        fac = (LEITH_13 * self.p["Lx"] / (self.p["nx"] * math.pi)) ** 12
        return torch.stack([fac * torch.sqrt((self.phys(f.clone()) * self.phys(self.k8 * f)).mean()) for f in q])


def _exact_network(layers, x):
    """Periodic 3x3 convolutions, GELU between them; x [B, C, H, W], weights [(w [9, co, ci], b)]."""
    for l, (w, b) in enumerate(layers):
        w4 = w.reshape(3, 3, w.shape[1], w.shape[2]).permute(2, 3, 0, 1)
        x = torch.nn.functional.conv2d(torch.nn.functional.pad(x, (1, 1, 1, 1), mode="circular"), w4, b)
        if l < len(layers) - 1:
            x = torch.nn.functional.gelu(x)
    return x


def _exact_weights(weights):
    return [tuple(torch.tensor(a, dtype=torch.float64, device="cuda") for a in wb) for wb in weights]


def _exact_closure(ref, c, q0, seed, H, S):
    """The closure's tendency and its energy-budget check."""
    nz, p = c["nz"], ref.p
    isc, osc = (torch.tensor(a, dtype=torch.float64, device="cuda")[:, None, None] for a in _scales(q0, p, H, S))
    layers = _exact_weights(_weights(_net_shapes(nz, c["net"]), 2 * nz, nz, seed, True))

    def tendency(q):
        psi = ref.psi(q)
        qp, pp = ref.phys(q.clone()), ref.phys(psi.clone())
        x = torch.zeros((1, 16, p["ny"], p["nx"]), dtype=torch.float64, device="cuda")
        x[0, :2 * nz] = torch.cat([qp, pp]) * isc
        s = torch.fft.rfft2(_exact_network(layers, x)[0, :nz] / osc) * ref.keep
        sp, w = ref.phys(s.clone()), ref.Hw
        dZ = float((w * (qp * sp).mean(dim=(1, 2))).sum())
        dE = -float((w * (pp * sp).mean(dim=(1, 2))).sum())
        E = -0.5 * float((w * (pp * qp).mean(dim=(1, 2))).sum())
        return s if dZ <= 0.0 and dE <= E / 86400.0 else None

    return tendency


def _exact_steps(ref, scheme, q, dt, steps, tendency=None, background=0.0):
    p, rhs = ref.p, ref.rhs
    if scheme.startswith("ark43"):
        ae, ai, b = _tableau()
        for _ in range(steps):
            s = tendency(q) if tendency else None
            A8 = ref.leith(q) if scheme == "ark43_qgleith" else torch.full((p["nz"],), p["A8"], device="cuda", dtype=torch.float64)
            if s is not None:
                A8 = torch.full_like(A8, background)
            f = rhs if s is None else (lambda a: rhs(a) + s)
            D = [p["A2"] * ref.k2 + a * ref.k8 for a in A8]
            N, Qs = [f(q)], [q]
            for i in range(1, 6):
                qi = torch.empty_like(q)
                for l in range(p["nz"]):
                    a = sum(ae[i, j] * N[j][l] for j in range(i)) - D[l] * sum(ai[i, j] * Qs[j][l] for j in range(i))
                    qi[l] = (q[l] + dt * a) / (1.0 + 0.25 * dt * D[l])
                N.append(f(qi))
                Qs.append(qi)
            q = q.clone()
            for l in range(p["nz"]):
                q[l] += dt * sum(b[i] * (N[i][l] - D[l] * Qs[i][l]) for i in (0, 2, 3, 4, 5))
            q *= ref.keep
        return q
    R0 = R1 = None
    for n in range(steps):
        if scheme == "bsrk3":
            R0 = rhs(q) if R0 is None else R0
            R1 = rhs(q + 0.5 * dt * R0)
            R2 = rhs(q + 0.75 * dt * R1)
            q = q + dt * (2.0 / 9.0 * R0 + 1.0 / 3.0 * R1 + 4.0 / 9.0 * R2)
            R0 = rhs(q)
        elif scheme == "rk4":
            a = rhs(q)
            b2 = rhs(q + 0.5 * dt * a)
            c3 = rhs(q + 0.5 * dt * b2)
            q = q + (dt / 6.0) * (a + 2.0 * b2 + 2.0 * c3 + rhs(q + dt * c3))
        else:
            R2 = rhs(q)
            inc = R2 if n == 0 else 1.5 * R2 - 0.5 * R1 if n == 1 else (23.0 * R2 - 16.0 * R1 + 5.0 * R0) / 12.0
            q, R0, R1 = q + dt * inc, R1, R2
    return q


def exact(case, seed):
    c = case
    if c["kind"] == "cnn":
        x, y = _samples(c, seed)
        layers = _exact_weights(_weights(_net_shapes(c["nz"], c["layers"]), 2 * c["nz"], c["nz"], seed, False))
        for w, b in layers:
            w.requires_grad_(c["call"] == "gradients")
            b.requires_grad_(c["call"] == "gradients")
        B, nz = c["batch"], c["nz"]
        with torch.set_grad_enabled(c["call"] == "gradients"):
            if c["call"] == "forward":
                out = torch.cat([_exact_network(layers, x[i:i + 1].double().permute(0, 3, 1, 2)) for i in range(B)])
                return out.permute(0, 2, 3, 1).contiguous()
            total = 0.0
            for i in range(B):        # one sample's graph at a time
                out = _exact_network(layers, x[i:i + 1].double().permute(0, 3, 1, 2))[:, :nz]
                d = out - y[i:i + 1, ..., :nz].double().permute(0, 3, 1, 2)
                part = d.square().sum() / (B * c["H"] * c["W"] * nz)
                part.backward()
                total += float(part.detach())
        return {"loss": total, "weights": [w.grad for w, _ in layers], "biases": [b.grad for _, b in layers]}
    if c["kind"] == "ensemble":
        specs = _members(c)
        done = [_exact_steps(_Reference(p, H, S, U), "bsrk3", q, p["dt_max"], c["steps"]).reshape(-1)
                for (p, H, S, U), q in zip(specs, _member_states(specs, seed))]
        return torch.cat(done)
    p, H, S, U = _configuration(c)
    ref, q = _Reference(p, H, S, U), _random_pv(p, seed)
    tendency = _exact_closure(ref, c, q, seed, H, S) if c["net"] else None
    q = _exact_steps(ref, c["scheme"], q, p["dt_max"], c["steps"], tendency, _background(p))
    return {"q": q, "t": c["steps"] * p["dt_max"], "dt": p["dt_max"]}
