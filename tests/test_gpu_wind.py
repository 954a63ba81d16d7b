"""The refined implicit solve under a wind across the columns (x3 of a 2-D
block), strong enough that the diagonal of the tangential momenta's rows
cancels, at steps of about 7 to 50 sound crossings of a layer (the cells are
flat): the direct FP64 solve's solution at the bar it has elsewhere (1e-13),
and no column left to that solve."""
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems

pytestmark = pytest.mark.gpu


def solution(cuda, flat, wind, corrections, nx1=64, nx2=64):
    opts = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/straka.yaml")
    c = opts.coord()
    c.nx1, c.nx2, c.x1max, c.x2max = nx1, nx2, nx1 * 50.0, nx2 * 50.0 * flat
    opts.hydro().precision = opts.hydro().icorr.precision = "float32"
    opts.execution = "eager"
    opts.autotune = False
    w = problems.straka(opts, "cpu", xc=0.2 * c.x2max, zc=0.4 * c.x1max,
                        xr=0.15 * c.x2max, zr=0.3 * c.x1max)
    g = torch.Generator().manual_seed(1)
    w[1:4] += torch.randn(w[1:4].shape, generator=g, dtype=torch.float64)
    w[3] += wind
    blk = sg.MeshBlock(opts).to(cuda)
    vars = {"hydro_w": w.to(cuda)}
    blk.initialize(vars)
    blk.batch.set_solve(corrections)
    blk.forward(vars, blk.max_time_step(vars), 0)
    torch.cuda.synchronize()
    cells = nx1 * nx2
    return (blk.batch.scratch[0][85 * cells:90 * cells].clone().view(nx2, -1),
            blk.batch.solve_fallbacks()[0])


@pytest.mark.parametrize("flat,wind", [(8, 100.0), (8, 250.0), (8, 300.0), (20, 170.0),
                                       (50, 100.0), (50, 320.0)])
def test_refined_solution_in_a_strong_wind(cuda, flat, wind):
    got, left = solution(cuda, flat, wind, 2)
    want, _ = solution(cuda, flat, wind, 0)
    assert left == 0
    assert (torch.linalg.norm(got - want) / torch.linalg.norm(want)).item() <= 1e-13


@pytest.mark.parametrize("flat,wind", [(1, 0.0), (8, 0.0), (8, 300.0), (50, 0.0), (50, 100.0),
                                       (50, 300.0)])
def test_fp32_solution_is_held_to_fp32_rounding(cuda, flat, wind):
    """The FP32 form (sg_set_solve -1): every column it accepts within FP32's
    rounding of its largest value (2^-24 by its own estimate; twice that here),
    the others solved in FP64.  No column of these fails."""
    got, left = solution(cuda, flat, wind, -1)
    want, _ = solution(cuda, flat, wind, 0)
    assert left == 0
    err = (got - want).abs().amax(1) / want.abs().amax(1)
    assert err.max().item() <= 2.0 ** -23
