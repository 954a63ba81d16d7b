"""The x3 sweep where its schedule can go wrong: planes of columns that end
inside a warp's 30 entries or fill them, x3 extents that are no multiple of
the chunk or shorter than it, walls and periodic sides, with the covariance
row and without, against the oracle at relative L2 1e-12 (the bar of the
other 3-D parity tests); FP32 against FP64 at its 1e-5."""
import numpy as np
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems

pytestmark = pytest.mark.gpu


def block(cuda, nx1, nx2, nx3, precision, cov, walls=False):
    opts = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/convection3d.yaml")
    c = opts.coord()
    c.nx1, c.nx2, c.nx3 = nx1, nx2, nx3
    c.x1max, c.x2max, c.x3max = nx1 * 50.0, nx2 * 50.0, nx3 * 50.0
    opts.hydro().flux_covariance = cov
    opts.hydro().precision = precision
    opts.hydro().icorr = None
    opts.execution = "eager"
    opts.autotune = False
    if walls:
        opts.bcnames = ["reflecting_inner", "reflecting_outer"] * 3
    w = problems.convection3d(opts, "cpu", seed=nx1 + nx2 + nx3)
    g = torch.Generator().manual_seed(nx1 * nx2 * nx3)
    w[1:4] += torch.randn(w[1:4].shape, generator=g, dtype=torch.float64)
    blk = sg.MeshBlock(opts).to(cuda)
    vars = {"hydro_w": w.to(cuda)}
    blk.initialize(vars)
    return opts, blk, vars, w


SIZES = [(6, 4, 3), (28, 3, 4), (30, 5, 7), (31, 4, 17), (13, 23, 5)]


@pytest.mark.parametrize("nx1,nx2,nx3", SIZES)
@pytest.mark.parametrize("cov,walls", [(True, False), (False, True)])
def test_x3_sweep_against_the_oracle(oracle, cuda, nx1, nx2, nx3, cov, walls):
    opts, blk, vars, w = block(cuda, nx1, nx2, nx3, "float64", cov, walls)
    ob = oracle.block_from_options(opts)
    u = ob.initialize(w.numpy())
    dt = blk.max_time_step(vars)
    for s in range(3):
        blk.forward(vars, dt, s)
        ob.stage(u, dt, s)
    got = vars["hydro_u"].cpu().numpy()
    for v in range(5):
        assert np.linalg.norm(got[v] - u[v]) <= 1e-12 * np.linalg.norm(u[v]), v


@pytest.mark.parametrize("nx1,nx2,nx3", SIZES)
def test_x3_sweep_fp32(cuda, nx1, nx2, nx3):
    _, b64, v64, _ = block(cuda, nx1, nx2, nx3, "float64", True)
    _, b32, v32, _ = block(cuda, nx1, nx2, nx3, "float32", True)
    dt = b64.max_time_step(v64)
    b64.step(v64, dt)
    b32.step(v32, dt)
    got, want = b32.total_u(v32)[:, 3:-3, 3:-3, 3:-3], v64["hydro_u"][:, 3:-3, 3:-3, 3:-3]
    for v in range(5):
        err = torch.linalg.norm(got[v] - want[v]) / torch.linalg.norm(want[v])
        assert err.item() <= 1e-5, v
