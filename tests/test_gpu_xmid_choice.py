"""x-pass kernels: the autotuner times each kernel once (FP64 plans without a
dual run one register kernel under variants 0 and 1), and the mixed form's two
register kernels agree with its shared-memory pass at every side they have.
Tolerance of the latter: the mixed form's bar, 1e-6."""
import numpy as np
import pytest
import torch

from conftest import rel
from jax_spectral_dns._plan import StepPlan, to_device_layout
from jax_spectral_dns.seeds import cheb_points, mode_counts, seeded_velocity_hat

pytestmark = pytest.mark.gpu
LX, LZ, RE, DT = 2 * np.pi, np.pi, 4000.0, 0.005


def _plan(mx, precision, **kw):
    modes, phys = mode_counts((mx - 1, 17, 4))
    assert modes[0] == mx
    return StepPlan(modes, phys, LX, LZ, 1, RE, DT, base_u=1 - cheb_points(17) ** 2, precision=precision, **kw)


# modes: sides 4, 6, 8, 9, 10
@pytest.mark.parametrize("mx,variant", [(9, 1), (21, 1), (41, 1), (49, 1), (65, 1)])
def test_autotuner_times_each_fp64_kernel_once(cuda, mx, variant):
    plan = _plan(mx, "fp64", autotune=True)
    times = plan.xmid_variant()[1]
    assert times[0] == 0 and times[variant] > 0 and times[2] > 0
    for v in (1, 2):
        plan.set_xmid_variant(v)
        assert plan.xmid_variant()[0] == v


@pytest.mark.parametrize("mx", [5, 9, 17, 33, 65, 121])  # sides 3, 4, 5, 7, 10, 14
def test_mixed_register_kernels_agree_with_the_shared_memory_pass(cuda, mx):
    shape = (mx - 1, 17, 4)
    u0 = seeded_velocity_hat(shape, (LX, LZ), (min(8, mx // 2), 2), 1e-3, seed=mx)
    out = {}
    for v in (0, 1, 2) if int(round((_plan(mx, "mixed").fft_sizes[0]) ** 0.5)) % 2 == 0 else (0, 2):
        plan = _plan(mx, "mixed")
        plan.set_xmid_variant(v)
        st = to_device_layout(u0)
        plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 3)
        out[v] = st.cpu().numpy()
    for v in out:
        assert rel(out[v], out[2]) < 1e-6, v
