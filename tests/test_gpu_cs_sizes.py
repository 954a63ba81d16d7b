"""The cubed-sphere stage at the edges of its launches: small panels
(every face within a stencil of a seam), odd sizes, faces that end inside a
CTA of 128 and seam faces inside a warp; both solvers, FP64 against the
oracle at relative L2 1e-12 (the bar of the other parity tests), the state
that enters a stage through each of its routes (initialize, a step, a set
rotation), and FP32 against FP64 at its 1e-5."""
import numpy as np
import pytest
import torch

from snapy_gb300 import cubed_sphere as cs
from test_gpu_cubed_sphere import errors, interior, oracle_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 11, 33])
@pytest.mark.parametrize("riemann", ["shallow-roe", "hllc"])
def test_stage_at_small_and_odd_sizes(cuda, n, riemann):
    o = oracle_sphere(n, riemann)
    u = cs.bump(n, seed=n, width=0.5)
    sp = cs.SphereSW(n, dtype=torch.float64, device=cuda, riemann=riemann)
    sp.initialize(u)
    o.fill(u)
    u0 = np.zeros_like(u)
    for step in range(3):
        dt = o.max_dt(u)
        sp.step(dt)
        for s in range(3):
            o.stage(u, u0, dt, s)
        err = errors(interior(sp.state().cpu().numpy(), n), interior(u, n))
        assert err.max() <= 1e-12, (step, err)


def test_fp32_at_an_odd_size(cuda):
    n = 11
    u = cs.bump(n, seed=3, width=0.5)
    out = []
    for dtype in (torch.float64, torch.float32):
        sp = cs.SphereSW(n, dtype=dtype, device=cuda)
        sp.initialize(u)
        sp.step(5.0)
        out.append(interior(sp.totals().cpu().numpy(), n))
    err = errors(out[1], out[0])
    assert err[[0, 2, 3]].max() <= 1e-5, err


def test_a_second_state_is_the_first_again(cuda):
    """Nothing is kept from one state to the next."""
    n = 12
    a, b = cs.bump(n, seed=1, width=0.4), cs.bump(n, seed=2, width=0.6)
    sp = cs.SphereSW(n, dtype=torch.float64, device=cuda)
    seen = []
    for u in (a, b, a):
        sp.initialize(u)
        sp.step(5.0)
        seen.append(sp.state().clone())
    assert torch.equal(seen[0], seen[2]) and not torch.equal(seen[0], seen[1])
