"""1-D blocks without sources at the edges of their segments (8 to 64 cells a
CTA, by the batch's cells): fewer cells than a segment, full ones, one cell
more, enough for wider segments; both solvers, walls and open ends; and a
batch of 1-D and 2-D blocks, each equal to itself alone.  Against the oracle
at relative L2 1e-12 (the bar of the other FP64 parity tests)."""
import numpy as np
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems
from snapy_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def options(nx1, riemann="hllc", walls=False, nx2=1, precision="float64"):
    opts = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/sod.yaml")
    c = opts.coord()
    c.nx1, c.nx2 = nx1, nx2
    opts.hydro().riemann.type = riemann
    opts.hydro().precision = precision
    opts.execution = "eager"
    opts.autotune = False
    if nx2 > 1:
        opts.bcnames = ["extrapolation_inner", "extrapolation_outer"] * 2
    if walls:
        opts.bcnames = ["reflecting_inner", "reflecting_outer"]
    return opts


def tube(opts):
    w = problems.sod(opts, "cpu")
    g = torch.Generator().manual_seed(opts.coord().nx1)
    w[1] += 0.3 * torch.rand(w[1].shape, generator=g, dtype=torch.float64)
    return w


@pytest.mark.parametrize("nx1", [4, 8, 9, 31, 256, 1217, 2500, 2800])
@pytest.mark.parametrize("riemann,walls", [("hllc", False), ("lmars", True)])
def test_segments_against_the_oracle(oracle, cuda, nx1, riemann, walls):
    opts = options(nx1, riemann, walls)
    w = tube(opts)
    blk = sg.MeshBlock(opts).to(cuda)
    vars = {"hydro_w": w.to(cuda)}
    blk.initialize(vars)
    ob = oracle.block_from_options(opts)
    u = ob.initialize(w.numpy())
    for _ in range(2):
        dt = blk.max_time_step(vars)
        blk.step(vars, dt)
        ob.step(u, dt)
    got = vars["hydro_u"].cpu().numpy()
    for v in (0, 1, 4):
        assert np.linalg.norm(got[v] - u[v]) <= 1e-12 * np.linalg.norm(u[v]), v


def test_fp32_against_fp64(cuda):
    out = []
    for precision in ("float64", "float32"):
        opts = options(100, precision=precision)
        blk = sg.MeshBlock(opts).to(cuda)
        vars = {"hydro_w": tube(opts).to(cuda)}
        blk.initialize(vars)
        blk.step(vars, 1e-4)
        out.append(vars["hydro_u"].double())
    for v in (0, 1, 4):
        assert torch.linalg.norm(out[1][v] - out[0][v]) <= 1e-5 * torch.linalg.norm(out[0][v])


def test_lines_and_planes_in_one_batch(cuda):
    members = [options(100), options(24, nx2=10), options(40)]
    ws = [tube(m) for m in members]
    ens = Ensemble(members, device=cuda)
    ens.initialize([w.to(cuda) for w in ws], autotune=False)
    dts = torch.full((3,), 1e-4, dtype=torch.float64, device=cuda)
    for _ in range(2):
        ens.step(dts)
    for k, (m, w) in enumerate(zip(members, ws)):
        blk = sg.MeshBlock(m).to(cuda)
        vars = {"hydro_w": w.to(cuda)}
        blk.initialize(vars)
        for _ in range(2):
            blk.step(vars, 1e-4)
        assert torch.equal(vars["hydro_u"], ens.state(k)), k
