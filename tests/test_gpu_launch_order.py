"""Programmatic launch order (a kernel may start while the one before it drains)
against plain order, bit for bit. A captured graph runs in plain order, so the
same calls are made directly and replayed from a graph: boxes on both sides of
the sizes up to which launches are programmatic, with the kernels that write in
place (mass flux, the adjoint's accumulating product), one run and a batch; and
directly on two streams at once, each beside the other's work."""
import numpy as np
import pytest
import torch

from jax_spectral_dns import _native
from jax_spectral_dns._plan import StepPlan, pack_runs, to_device_layout
from jax_spectral_dns.seeds import cheb_points, mode_counts, seeded_velocity_hat, turbulent_channel_hat

pytestmark = pytest.mark.gpu
LX, LZ, RE, DT = 2 * np.pi, np.pi, 4000.0, 0.005


def _kmax(modes):
    return min(8, modes[0] // 2), min(8, modes[2] // 2)


def _channel(shape, precision):
    modes, phys = mode_counts(shape)
    u = to_device_layout(turbulent_channel_hat(shape, (LX, LZ), 180.0, _kmax(modes), seed=3))
    probe = StepPlan(modes, phys, LX, LZ, _native.JSD_KIND_NS, 180.0, 0.002, precision=precision)
    q0 = 1.001 * probe.flow_rate(u[0]).item()
    return StepPlan(modes, phys, LX, LZ, _native.JSD_KIND_NS, 180.0, 0.002, constant_mass_flux=True,
                    flow_rate_target=q0, precision=precision), u


def _perturbation(shape, linearise=False, runs=1):
    modes, phys = mode_counts(shape)
    res = [RE / (1 + r) for r in range(runs)]
    u = [seeded_velocity_hat(shape, (LX, LZ), _kmax(modes), 1e-3, seed=r) for r in range(runs)]
    plan = StepPlan(modes, phys, LX, LZ, _native.JSD_KIND_PERTURBATION, res if runs > 1 else RE, DT,
                    linearise=linearise, base_u=1 - cheb_points(modes[1]) ** 2)
    return plan, pack_runs(u) if runs > 1 else to_device_layout(u[0])


def _replayed(calls, tensors):
    """The tensors after `calls` captured in a graph and replayed once."""
    bufs = [t.clone() for t in tensors]
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        calls(*bufs)
    graph.replay()
    torch.cuda.synchronize()
    return bufs


def _direct(calls, tensors):
    bufs = [t.clone() for t in tensors]
    calls(*bufs)
    torch.cuda.synchronize()
    return bufs


def _same(calls, tensors):
    plain = None
    for _ in range(3):  # (the first direct run also loads the kernels)
        direct = _direct(calls, tensors)
        plain = plain or _replayed(calls, tensors)
        for a, b in zip(direct, plain):
            assert torch.isfinite(torch.view_as_real(a) if a.is_complex() else a).all()
            assert torch.equal(a, b)


# entries per field: FP64 programmatic up to 1048576, mixed up to 80000
@pytest.mark.parametrize("shape,precision,steps", [
    ((8, 33, 8), "fp64", 30), ((40, 34, 24), "fp64", 10), ((96, 95, 112), "fp64", 1), ((100, 104, 100), "fp64", 1),
    ((8, 33, 8), "mixed", 30), ((32, 65, 36), "mixed", 4), ((36, 65, 36), "mixed", 4)])
def test_channel_with_mass_flux(cuda, shape, precision, steps):
    plan, u = _channel(shape, precision)
    dp = torch.tensor([-0.2], dtype=torch.float64, device="cuda")
    _same(lambda st, d: plan.step(st, d, 0, steps), (u, dp))


@pytest.mark.parametrize("shape,linearise,runs", [((8, 33, 8), True, 1), ((32, 65, 32), True, 1), ((8, 33, 8), False, 1),
                                                  ((16, 34, 24), False, 5), ((16, 33, 8), True, 3)])
def test_perturbation(cuda, shape, linearise, runs):
    plan, u = _perturbation(shape, linearise, runs)
    dp = torch.zeros(1, dtype=torch.float64, device="cuda")
    _same(lambda st, d: plan.step(st, d, 0, 10), (u, dp))


@pytest.mark.parametrize("shape", [(8, 33, 8), (8, 195, 8), (32, 65, 32)])  # 195: the adjoint adds a field of its own
def test_adjoint(cuda, shape):
    plan, u = _perturbation(shape, True)
    _same(lambda st: plan.step_adjoint(st, 10), (u,))


def test_two_streams_at_once(cuda):
    """Two plans stepping on two streams give what each gives alone."""
    made = [_channel((40, 34, 24), "fp64"), _perturbation((32, 65, 32))]
    dp = torch.tensor([-0.2], dtype=torch.float64, device="cuda")
    alone = [_direct(lambda st, d, plan=plan: plan.step(st, d, 0, 20), (u, dp)) for plan, u in made]
    for _ in range(3):
        bufs = [[u.clone(), dp.clone()] for _, u in made]
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in made]
        for (plan, _), (st, d), s in zip(made, bufs, streams):
            with torch.cuda.stream(s):
                plan.step(st, d, 0, 20)
        torch.cuda.synchronize()
        for got, want in zip(bufs, alone):
            assert all(torch.equal(a, b) for a, b in zip(got, want))
