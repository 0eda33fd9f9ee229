"""Every square FFT side of the FP64 transforms inside the step, against the
oracle: boxes whose x or z modes choose sides 3 to 16, narrow planes whose x-pass
blocks span two planes, channel with fixed flow rate and perturbation about a
base flow, and a batch of runs. Tolerance: the FP64 parity bar of the package."""
import numpy as np
import pytest
import torch

import jsd_oracle as O
from conftest import rel
from jax_spectral_dns._ops import SQUARE_FFT_SIDES
from jax_spectral_dns._plan import StepPlan, pack_runs, to_device_layout, to_reference_layout, unpack_runs
from jax_spectral_dns.seeds import cheb_points, mode_counts, seeded_velocity_hat, turbulent_channel_hat

pytestmark = pytest.mark.gpu
LX, LZ, RE, DT = 2 * np.pi, np.pi, 4000.0, 0.005
SHAPES = [(4, 17, 8), (8, 17, 4), (16, 19, 12), (20, 17, 8), (12, 17, 24), (32, 17, 4), (4, 18, 40), (40, 17, 8),
          (48, 17, 20), (4, 17, 48), (64, 17, 4), (88, 17, 4), (8, 17, 88), (120, 17, 8), (144, 17, 4), (4, 17, 144)]


def test_shapes_reach_every_side():
    plans = [np.sqrt(3 * (m // 2) + 1) for s in SHAPES for m in mode_counts(s)[0][::2]]
    reached = {min(side for side in SQUARE_FFT_SIDES if side >= p) for p in plans}
    assert reached == set(SQUARE_FFT_SIDES)


@pytest.mark.parametrize("shape", SHAPES)
def test_channel_step(cuda, shape):
    re_tau, dt = 180.0, 0.002
    modes, phys = mode_counts(shape)
    kmax = (modes[0] // 2, modes[2] // 2)
    u0 = turbulent_channel_hat(shape, (LX, LZ), re_tau, kmax, seed=3)
    g = O.Grid(shape, LX, LZ)
    q0 = g.flow_rate(u0[0]) * 1.001
    plan = StepPlan(modes, phys, LX, LZ, 0, re_tau, dt, constant_mass_flux=True, flow_rate_target=q0)
    st, dp = to_device_layout(u0), torch.tensor([-0.2], dtype=torch.float64, device="cuda")
    plan.step(st, dp, 0, 1)
    ref = O.make_stepper("ns", shape, LX, LZ, re_tau, dt, constant_mass_flux=True, flow_rate_target=q0)
    want, dpw, _ = O.run(ref, u0, 1, dpdx=-0.2)
    assert rel(to_reference_layout(st).cpu().numpy(), want) < 1e-10
    assert abs(dp.item() - dpw) < 1e-9 * abs(dpw)


@pytest.mark.parametrize("shape", [(16, 18, 12), (40, 17, 8), (48, 17, 20), (4, 17, 144), (120, 17, 8)])
def test_batch_about_a_base_flow(cuda, shape):
    modes, phys = mode_counts(shape)
    kmax = (min(8, modes[0] // 2), min(8, modes[2] // 2))
    runs = [(RE, 1e-3), (0.5 * RE, 1e-2), (2 * RE, 1e-4)]
    u0 = [seeded_velocity_hat(shape, (LX, LZ), kmax, e0, seed=i) for i, (_, e0) in enumerate(runs)]
    plan = StepPlan(modes, phys, LX, LZ, 1, [re for re, _ in runs], DT, base_u=1 - cheb_points(shape[1]) ** 2)
    st = pack_runs(u0)
    plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 2)
    for got, u, (re, _) in zip(unpack_runs(st), u0, runs):
        want, _, _ = O.run(O.make_stepper("perturbation", shape, LX, LZ, re, DT, linearise=False), u, 2)
        assert rel(got.cpu().numpy(), want) < 1e-10
