"""What a user of this package has the GPU do, for timing: time steps of the
channel, perturbation and linearised equations, their gradients, and batches of
runs, through the package's public calls.

``exact`` restates the step from its definition in plain torch (64 bits): real
2-D FFTs on the 3/2 grid, dense Chebyshev matrices, one dense inverse per
wavenumber, and autograd for the gradient of the linearised gain.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jax-spectral-dns_b200"))

# box and flow of each equation: (Lx, Lz, Re or Re_tau, dt, largest populated |mode index|)
FLOWS = {
    "channel": (4 * math.pi, 4 * math.pi / 3, 180.0, 0.002, 16),  # turbulent channel, Reichardt mean, fixed flow rate
    "perturbation": (2 * math.pi, math.pi, 5000.0, 0.005, 8),     # nonlinear, about U = 1 - y^2
    "linear": (2 * math.pi, math.pi, 3000.0, 0.01, 8),            # linearised about U = 1 - y^2
}
E0 = 1e-3           # kinetic energy of a perturbation
GRADIENT_E0 = 1e-4  # of the start field of a nonlinear gradient
ALPHA = (29 / 96, -3 / 40, 1 / 6)
BETA = (37 / 160, 5 / 24, 1 / 6)
GAMMA = (8 / 15, 5 / 12, 3 / 4)
XI = (0.0, -17 / 60, -5 / 12)


def _case(call, flow, nx, ny, nz, steps, precision="fp64", runs=1, **more):
    return dict(call=call, flow=flow, nx=nx, ny=ny, nz=nz, steps=steps, precision=precision, runs=runs, **more)


def listed():
    return [
        # one step of a small linearised run and its energy, as a monitored time loop makes them: launches and latency
        _case("step", "linear", 8, 65, 4, 1, energy=True, name="linear step 9x65x5"),
        # a stretch of an optimal-perturbation forward run, captured once and replayed
        _case("graph", "perturbation", 32, 65, 32, 10, name="perturbation 10 steps replayed 33x65x33"),
        # the reference's own call: reference layout in and out, one step
        _case("timestep", "perturbation", 48, 65, 48, 1, name="perform_time_step 49x65x49"),
        # the mixed-precision form of the same run
        _case("step", "perturbation", 48, 65, 48, 2, "mixed", name="perturbation mixed 49x65x49"),
        # uneven box with an even number of Chebyshev points: no mid-plane, mode counts far from each other
        _case("step", "channel", 40, 82, 24, 2, name="channel 41x82x25"),
        # an ensemble's box group: runs with their own Reynolds numbers side by side
        _case("step", "perturbation", 32, 97, 32, 1, runs=8, name="8 runs 33x97x33"),
        # transient growth: gain of the linearised equations and its exact gradient
        _case("gradient", "linear", 32, 65, 32, 20, name="linear gain and gradient 33x65x33"),
        # the same for the nonlinear equations: forward run, recompute, dual run
        _case("gradient", "perturbation", 32, 65, 32, 20, name="nonlinear gain and dual gradient 33x65x33"),
        # the turbulent channel at its usual resolution: plain, and mixed with the kernels its plan timed
        _case("step", "channel", 128, 129, 128, 2, name="channel 129x129x129"),
        _case("step", "channel", 128, 129, 128, 2, "mixed", tuned=True, name="channel mixed 129x129x129"),
        # a finer grid of the same channel
        _case("step", "channel", 160, 145, 160, 2, name="channel 161x145x161"),
    ]


def _spread(rng, low, high, step=1):
    """A multiple of `step` in [low, high], even over its logarithm."""
    return max(low, min(high, step * round(math.exp(rng.uniform(math.log(low), math.log(high))) / step)))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "graph", "timestep", "gradient", "batch"))
    if kind == "gradient":
        return _case("gradient", rng.choice(("linear", "perturbation")), _spread(rng, 8, 40, 4), _spread(rng, 25, 97),
                     _spread(rng, 4, 40, 4), rng.randint(4, 24))
    if kind == "batch":
        return _case("step", rng.choice(("linear", "perturbation")), _spread(rng, 8, 48, 4), _spread(rng, 25, 97),
                     _spread(rng, 8, 48, 4), 1, runs=rng.randint(2, 12))
    flow = rng.choice(("channel", "channel", "perturbation", "linear"))
    top = 160 if kind == "step" and flow == "channel" else 64
    return _case(kind, flow, _spread(rng, 8, top, 4), _spread(rng, 17, 145 if top > 64 else 97), _spread(rng, 4, top, 4),
                 1 if kind == "timestep" else rng.randint(1, 2),
                 "fp64" if kind == "timestep" or flow == "linear" else rng.choice(("fp64", "mixed")))


# ---------------------------------------------------------------------------
# discretisation (plain torch)
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class Box:
    """Grid of a case: Mx = nx + 1 and Mz = nz + 1 modes, ny Chebyshev points."""

    def __init__(self, case):
        dev = _device()
        self.lx, self.lz, self.re, self.dt, self.kmax = FLOWS[case["flow"]]
        self.mx, self.ny, self.mz = case["nx"] + 1, case["ny"], case["nz"] + 1
        self.modes = (self.mx, self.ny, self.mz)

        def physical(m):  # points of the dealiased grid: ceil(3 m / 2) made odd, less one
            return (math.ceil(1.5 * m) // 2) * 2

        self.px, self.pz = physical(self.mx), physical(self.mz)
        self.phys = (self.px, self.ny, self.pz)
        self.s = self.lx * self.lz / (4 * math.pi ** 2)
        n = self.ny - 1
        i = np.arange(self.ny)
        ii, jj = np.meshgrid(i, i, indexing="ij")
        # y_i - y_j without cancellation, and the diagonal from the row sums
        dy = 2 * np.sin((ii + jj) * math.pi / (2 * n)) * np.sin((jj - ii) * math.pi / (2 * n))
        c = np.where((i == 0) | (i == n), 2.0, 1.0) * (-1.0) ** i
        d = np.outer(c, 1 / c) / (dy + np.eye(self.ny))
        np.fill_diagonal(d, 0.0)
        np.fill_diagonal(d, -d.sum(axis=1))
        self.y_np = np.cos(math.pi * i / n)
        self.y = torch.as_tensor(self.y_np, device=dev)
        self.D = torch.as_tensor(d, device=dev)
        self.D2 = self.D @ self.D
        # weights of the y-integral: the antiderivative that D, without its
        # first row and column, gives of values that vanish at y = 1
        anti = np.linalg.inv(np.block([[np.ones((1, 1)), np.zeros((1, n))], [np.zeros((n, 1)), d[1:, 1:]]]))
        w = anti[0] - anti[-1]
        w[0] = 0.0
        self.w = torch.as_tensor(w, device=dev)
        fx = torch.fft.fftfreq(self.mx, 1 / self.mx, dtype=torch.float64, device=dev).round()
        fz = torch.fft.fftfreq(self.mz, 1 / self.mz, dtype=torch.float64, device=dev).round()
        self.fx, self.fz = fx, fz
        self.kx = (fx * 2 * math.pi / self.lx)[None, :, None]
        self.kz = (fz * 2 * math.pi / self.lz)[None, None, :]
        self.k2 = self.kx ** 2 + self.kz ** 2
        # coefficient of a constant field of value 1
        self.one = math.sqrt(self.px * self.pz) / self.s

    def dy(self, f):
        """Chebyshev derivative along y of (..., ny, Mx, Mz)."""
        return torch.einsum("ij,...jab->...iab", self.D.to(f.dtype), f)

    def physical(self, f):
        """Values on the dealiased grid."""
        kx, kz = self.mx // 2, self.mz // 2
        out = torch.zeros(f.shape[:-2] + (self.px, self.pz), dtype=f.dtype, device=f.device)
        out[..., : kx + 1, : kz + 1] = f[..., : kx + 1, : kz + 1]
        out[..., : kx + 1, -kz:] = f[..., : kx + 1, kz + 1:]
        out[..., -kx:, : kz + 1] = f[..., kx + 1:, : kz + 1]
        out[..., -kx:, -kz:] = f[..., kx + 1:, kz + 1:]
        return torch.fft.ifftn(out, dim=(-2, -1), norm="ortho").real * self.s

    def spectral(self, f):
        """Coefficients |k| <= K; along x, then z, the -K entry is the conjugate of the +K one."""
        out = torch.fft.fftn(f.to(torch.complex128), dim=(-2, -1), norm="ortho") / self.s
        for ax, m in ((-2, self.mx), (-1, self.mz)):
            k, p = m // 2, out.shape[ax]
            top = out.narrow(ax, k, 1)
            out = torch.cat([out.narrow(ax, 0, k), top, top.conj(), out.narrow(ax, p - k + 1, k - 1)], dim=ax)
        return out

    def energy(self, u):
        """Kinetic energy of (3, ny, Mx, Mz)."""
        return 0.25 * ((self.physical(u) ** 2).mean(dim=(-2, -1)).sum(0) * self.w).sum()


def _start_field(box, seed, energy):
    """Solenoidal no-slip field (3, ny, Mx, Mz): damped random Chebyshev series
    times (1 - y^2)^2 for v and (1 - y^2) for omega_y, u and w from continuity."""
    dev = box.y.device
    gen = torch.Generator(device=dev).manual_seed(seed)
    n = torch.arange(box.ny, device=dev, dtype=torch.float64)
    tn = torch.cos(torch.outer(torch.arccos(box.y), n))
    mask = ((box.fx.abs() <= box.kmax)[:, None] & (box.fz.abs() <= box.kmax)[None, :]).to(torch.float64)
    mask[0, 0] = 0.0

    def series(order, last):
        c = torch.randn((2, box.ny, box.mx, box.mz), generator=gen, device=dev, dtype=torch.float64)
        c = torch.complex(c[0], c[1]) * (torch.exp(-n / 8) * (n < box.ny - last))[:, None, None]
        f = torch.einsum("ij,jab->iab", tn.to(c.dtype), c) * mask * ((1 - box.y ** 2) ** order)[:, None, None]
        back = torch.roll(torch.flip(f, (-2, -1)), (1, 1), (-2, -1))  # the entry of -k
        return (f + back.conj()) / 2

    v, om = series(2, 4), series(1, 2)
    dv = box.dy(v)
    k2 = torch.where(box.k2 == 0, torch.ones_like(box.k2), box.k2)
    u = torch.stack([1j * (box.kx * dv - box.kz * om) / k2, v, 1j * (box.kz * dv + box.kx * om) / k2])
    u[:, [0, -1]] = 0
    return u * torch.sqrt(energy / box.energy(u))


def _mean_profile(box):
    """Reichardt's law, mirrored about y = 0."""
    yp = (1 - box.y.abs()) * box.re
    return 2.5 * torch.log1p(0.4 * yp) + 7.8 * (1 - torch.exp(-yp / 11) - yp / 11 * torch.exp(-yp / 3))


def _input(case, box, seed, run=0):
    """(state (3, ny, Mx, Mz), pressure gradient, flow rate) of one run."""
    seed = 1000 * seed + run
    if case["flow"] != "channel":
        return _start_field(box, seed, GRADIENT_E0 if case["call"] == "gradient" else E0), 0.0, 0.0
    mean = _mean_profile(box)
    u = _start_field(box, seed, 1.0)
    u = u * (0.1 * mean.max() / box.physical(u).abs().max())
    u[0, :, 0, 0] += mean * box.one
    if case["call"] == "timestep":  # the equation class holds the flow rate of its start field
        flow = float((box.physical(u[0])[:, 0, 0] * box.w).sum())
        return u, -flow * 1.5 / box.re, flow
    # a seeded change of the mean flow, so that the flow-rate control has work
    flow = float(torch.dot(box.w, mean)) * (1 + 1e-3 * ((seed % 7) - 3) / 3)
    return u, -flow * 1.5 / box.re, flow


def _reynolds(case, box):
    """Reynolds number of each run."""
    return [box.re * (0.5 + 1.0 * r / case["runs"]) for r in range(case["runs"])] if case["runs"] > 1 else [box.re]


# ---------------------------------------------------------------------------
# the package's calls
# ---------------------------------------------------------------------------
_KINDS = {"channel": 0, "perturbation": 1, "linear": 1}


def _plan(case, box, flow):
    from jax_spectral_dns._plan import StepPlan

    re = _reynolds(case, box)
    return StepPlan(box.modes, box.phys, box.lx, box.lz, _KINDS[case["flow"]], re if case["runs"] > 1 else re[0], box.dt,
                    linearise=case["flow"] == "linear", constant_mass_flux=case["flow"] == "channel",
                    flow_rate_target=flow, base_u=None if case["flow"] == "channel" else 1 - box.y_np ** 2,
                    precision=case["precision"], autotune=bool(case.get("tuned")))


def prepare(case, seed):
    box = Box(case)
    call = case["call"]
    u, dpdx, flow = _input(case, box, seed)
    state = {"case": case, "dpdx": torch.tensor([dpdx], dtype=torch.float64, device="cuda")}
    if call == "gradient":
        from jax_spectral_dns.adjoint import GainProblem

        state["problem"] = GainProblem(box.modes, box.phys, box.lx, box.lz, box.re, box.dt, (case["steps"] + 0.5) * box.dt,
                                       case["flow"] == "linear", checkpoint_every=10)
        state["u"] = u.transpose(1, 2).contiguous().requires_grad_()
    elif call == "timestep":
        state["u"] = u.transpose(1, 2).contiguous()
        state["equation"] = _equation(case, box, state["u"])
        state["pressure"] = dpdx
    else:
        state["plan"] = _plan(case, box, flow)
        if case["runs"] > 1:
            u = torch.stack([_input(case, box, seed, r)[0] for r in range(case["runs"])], dim=2)
        state["u"] = u.contiguous()
        if call == "graph":
            from jax_spectral_dns._plan import GraphedSteps

            state["buffer"], state["pressure"] = state["u"].clone(), state["dpdx"].clone()
            state["graph"] = GraphedSteps(state["plan"], state["buffer"], state["pressure"], 0, case["steps"])
    return state


def _equation(case, box, u):
    from jax_spectral_dns.domain import PhysicalDomain
    from jax_spectral_dns.field import FourierField, VectorField
    from jax_spectral_dns.navier_stokes import NavierStokesVelVort
    from jax_spectral_dns.navier_stokes_perturbation import NavierStokesVelVortPerturbation

    dom = PhysicalDomain.create((case["nx"], case["ny"], case["nz"]), (True, False, True),
                                scale_factors=(box.lx, 1.0, box.lz), aliasing=3 / 2)
    field = VectorField.FromData(FourierField, dom, u)
    if case["flow"] == "channel":
        return NavierStokesVelVort(field, Re_tau=box.re, dt=box.dt, end_time=1.0, constant_mass_flux=True)
    return NavierStokesVelVortPerturbation(field, Re=box.re, dt=box.dt, end_time=1.0, linearise=case["flow"] == "linear")


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "gradient":
        from jax_spectral_dns.adjoint import gain

        value = gain(state["u"], state["problem"])
        (grad,) = torch.autograd.grad(value, state["u"])
        return {"gain": value.detach(), "gradient": grad}
    if call == "timestep":
        u, dpdx = state["equation"].perform_time_step(state["u"], state["pressure"], 0)
        return {"state": u, "dpdx": dpdx}
    if call == "graph":
        state["buffer"].copy_(state["u"])
        state["pressure"].copy_(state["dpdx"])
        state["graph"].replay()
        return {"state": state["buffer"], "dpdx": state["pressure"]}
    u, dpdx = state["u"].clone(), state["dpdx"].clone()
    state["plan"].step(u, dpdx, 0, case["steps"])
    out = {"state": u, "dpdx": dpdx}
    if case.get("energy"):
        out["energy"] = state["plan"].energy(u)
    return out


def work(case):
    """State in and out once; the transforms' and y-contractions' operations
    (real FFTs, and halves of the y-operators on even and odd parts)."""
    box_modes = (case["nx"] + 1) * (case["nz"] + 1)
    field = 16.0 * box_modes * case["ny"]
    grid = (1.5 * case["nx"]) * (1.5 * case["nz"])
    linear = case["flow"] == "linear"
    fft = 0.0 if linear else 15 * 2.5 * grid * math.log2(grid) * case["ny"]
    contraction = 2.0 * box_modes * case["ny"] ** 2  # one half-size real operator on re and im
    stage = fft + (5 if linear else 8) * contraction
    dual = 27 / 15 * fft + (5 if linear else 11) * contraction
    passes = 3 * case["steps"] * case["runs"]
    if case["call"] == "gradient":
        return {"bytes": 2 * 3 * field, "flops": passes * (stage + dual)}
    return {"bytes": 2 * 3 * field * case["runs"], "flops": passes * stage}


# ---------------------------------------------------------------------------
# 64-bit restatement
# ---------------------------------------------------------------------------
class Stepper:
    """RK3/Crank-Nicolson step of the velocity-vorticity equations with one
    dense inverse per wavenumber and stage."""

    def __init__(self, box, re, flow, target=0.0, dual=False):
        self.box, self.re, self.flow, self.dual, self.target = box, re, flow, dual, target
        self.lam = 0.0 if flow == "linear" else 1.0
        self.base = None if flow == "channel" else 1 - box.y ** 2
        self.dt_e = -box.dt if dual else box.dt
        n = box.ny - 2
        self.a = box.D2[1:-1, 1:-1]
        eye = torch.eye(n, dtype=torch.float64, device=box.y.device)
        k2 = box.k2.reshape(-1, 1, 1)
        self.poisson = torch.linalg.inv(self.a - k2 * eye)
        self.helm, self.va, self.wall, self.mean = [], [], [], []
        d_wall = box.D[[0, -1], 1:-1]
        for b in BETA:
            bt = b * box.dt / re
            helm = torch.linalg.inv((1 + bt * k2) * eye - bt * self.a)
            va = (self.poisson @ (helm @ (bt * box.D2[1:-1, :1])))[..., 0]
            both = torch.stack([va, va.flip(-1)], dim=-1)
            self.helm.append(helm)
            self.va.append(both)
            self.wall.append(torch.linalg.inv(d_wall @ both))
            self.mean.append(torch.linalg.inv(eye - bt * self.a))
        self.d_wall = d_wall

    def _modes(self, f):
        """(n, Mx, Mz) complex -> (Mx Mz, n, 2) real."""
        return torch.view_as_real(f.reshape(f.shape[0], -1).transpose(0, 1).contiguous())

    def _field(self, m):
        f = torch.view_as_complex(m.contiguous()).transpose(0, 1)
        return f.reshape(-1, self.box.mx, self.box.mz)

    def _gradient(self, u):
        """grad[i][j] = d_j u_i on the grid."""
        b = self.box
        return [[b.physical(1j * b.kx * u[i]), b.physical(b.dy(u[i])), b.physical(1j * b.kz * u[i])] for i in range(3)]

    def _terms(self, u, forward):
        """Spectral helicity terms."""
        b = self.box
        vel, grad = b.physical(u), self._gradient(u)
        div = grad[0][0] + grad[1][1] + grad[2][2]
        if self.base is not None:
            ub = self.base[:, None, None]
            dub = (b.D @ self.base)[:, None, None]
        if self.dual:
            ut = [self.lam * x for x in b.physical(forward)] if self.lam else [0.0 * x for x in vel]
            gt = self._gradient(forward) if self.lam else [[0.0 * div] * 3 for _ in range(3)]
            ut[0] = ut[0] + ub
            gt[0][1] = gt[0][1] + dub
            divt = gt[0][0] + gt[1][1] + gt[2][2]
            hel = []
            for i in range(3):
                acc = -sum(ut[j] * grad[i][j] for j in range(3)) + sum(vel[j] * gt[j][i] for j in range(3))
                hel.append(acc + 0.25 * (divt * vel[i] + div * ut[i]))
            return b.spectral(torch.stack(hel))
        hel = []
        for i in range(3):
            acc = self.lam * (0.5 * div * vel[i] - sum(vel[j] * grad[i][j] for j in range(3)))
            if self.base is not None:
                acc = acc - ub * grad[i][0]
                if i == 0:
                    acc = acc - vel[1] * dub + 0.5 * div * ub
            hel.append(acc)
        return b.spectral(torch.stack(hel))

    def _implicit(self, x, ax):
        """Interior of x + alpha dt / Re (D2 - k^2) x."""
        inner = x[1:-1]
        lap = torch.einsum("ij,jab->iab", self.a.to(x.dtype), inner) - self.box.k2 * inner
        return inner + ax * lap

    def step(self, u, dpdx, forward=None):
        b = self.box
        old = None
        for st in range(3):
            h = self._terms(u, forward)
            h_v = -b.dy(1j * b.kx * h[0] + 1j * b.kz * h[2]) - b.k2 * h[1]
            h_g = 1j * b.kz * h[0] - 1j * b.kx * h[2]
            new = (h_v, h_g, h[:, :, 0, 0])
            g, x = self.dt_e * GAMMA[st], self.dt_e * XI[st]
            ex = [g * n + (0 if old is None else x * o) for n, o in zip(new, old or new)]
            ax = ALPHA[st] * b.dt / self.re
            om = 1j * b.kz * u[0] - 1j * b.kx * u[2]
            phi = torch.einsum("ij,jab->iab", b.D2.to(u.dtype), u[1]) - b.k2 * u[1]
            rhs = torch.cat([self._modes(self._implicit(phi, ax) + ex[0][1:-1]),
                             self._modes(self._implicit(om, ax) + ex[1][1:-1])], dim=-1)
            sol = self.helm[st] @ rhs
            vp = self.poisson @ sol[..., :2]
            v = vp - self.va[st] @ (self.wall[st] @ (self.d_wall @ vp))
            pad = torch.zeros_like(u[0, :1])
            v = torch.cat([pad, self._field(v), pad])
            om = torch.cat([pad, self._field(sol[..., 2:]), pad])
            dv = b.dy(v)
            k2 = torch.where(b.k2 == 0, torch.ones_like(b.k2), b.k2)
            uu = 1j * (b.kx * dv - b.kz * om) / k2
            ww = 1j * (b.kz * dv + b.kx * om) / k2
            for c, f, drive in ((0, uu, -dpdx * b.one), (2, ww, 0.0)):
                m = u[c, 1:-1, 0, 0]
                r = m + ax * (self.a.to(m.dtype) @ m) + ex[2][c, 1:-1] + drive * (g + x)
                f[:, 0, 0] = 0
                f[1:-1, 0, 0] = self.mean[st].to(m.dtype) @ r
            inside = torch.ones_like(b.y)
            inside[[0, -1]] = 0
            u = torch.stack([uu, v, ww]) * inside[:, None, None]
            old = new
        if self.flow == "channel":
            phys = b.physical(u[0])
            off = (phys[:, 0, 0] * b.w).sum() - self.target
            dpdx = dpdx + off / self.dt_e
            u = torch.stack([b.spectral(phys - off / 2), u[1], u[2]])
        return u, dpdx


def _reference_layout(f):
    return f.transpose(-3, -2).contiguous()


def _exact_gradient(case, box, u):
    if case["flow"] == "linear":  # the derivative of the computed gain
        steps = Stepper(box, box.re, case["flow"])
        u = u.clone().requires_grad_()
        v = u
        for _ in range(case["steps"]):
            v, _ = steps.step(v, 0.0)
        gain = box.energy(v) / box.energy(u)
        (grad,) = torch.autograd.grad(gain, u)
        return gain.detach(), grad
    # the continuous dual: backward from -u(T), frozen at the forward states
    forward = Stepper(box, box.re, case["flow"])
    states = [u]
    for _ in range(case["steps"]):
        states.append(forward.step(states[-1], 0.0)[0])
    e0 = box.energy(u)
    gain = box.energy(states[-1]) / e0
    dual = Stepper(box, box.re, case["flow"], dual=True)
    v = -states[-1]
    for t in range(case["steps"]):
        v, _ = dual.step(v, 0.0, states[case["steps"] - t])
    metric = 0.5 / box.one ** 2 * box.w[:, None, None]
    return gain, (-v - gain * u) / e0 * metric


def exact(case, seed):
    box = Box(case)
    if case["call"] == "gradient":
        gain, grad = _exact_gradient(case, box, _input(case, box, seed)[0])
        return {"gain": gain, "gradient": _reference_layout(grad)}
    states, dpdx = [], 0.0
    for r, re in enumerate(_reynolds(case, box)):
        u, dpdx, flow = _input(case, box, seed, r)
        stepper = Stepper(box, re, case["flow"], flow)
        for _ in range(case["steps"]):
            u, dpdx = stepper.step(u, dpdx)
        states.append(u)
        del stepper
    if case["call"] == "timestep":
        return {"state": _reference_layout(states[0]), "dpdx": float(dpdx)}
    out = {"state": torch.stack(states, dim=2) if case["runs"] > 1 else states[0],
           "dpdx": torch.as_tensor([float(dpdx)], dtype=torch.float64)}
    if case.get("energy"):
        out["energy"] = box.energy(states[0]).reshape(1)
    return out
