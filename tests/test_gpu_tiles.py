"""The refined implicit solve at the edges of its column tiles (32 columns):
one column, a tile less one, full, one more; layer counts from the fewest
with wall third points up, odd and even (the sweeps take layers in pairs),
fewer than their rings are deep and more.  Against the direct FP64 solve of
the same FP32-assembled system, at the bar the refined solve has elsewhere
(1e-13: both solve to FP64 roundoff), and no column left to it."""
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems

pytestmark = pytest.mark.gpu


def solution(cuda, nx1, nx2, corrections):
    opts = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/straka.yaml")
    c = opts.coord()
    c.nx1, c.nx2, c.x1max, c.x2max = nx1, nx2, nx1 * 50.0, nx2 * 50.0
    opts.hydro().precision = "float32"
    opts.hydro().icorr.precision = "float32"
    opts.execution = "eager"
    opts.autotune = False
    w = problems.straka(opts, "cpu", xc=0.4 * nx2 * 50.0, zc=0.4 * nx1 * 50.0,
                        xr=0.3 * nx2 * 50.0, zr=0.3 * nx1 * 50.0)
    g = torch.Generator().manual_seed(nx1 * 1000 + nx2)
    w[1:4] += torch.randn(w[1:4].shape, generator=g, dtype=torch.float64)
    blk = sg.MeshBlock(opts).to(cuda)
    vars = {"hydro_w": w.to(cuda)}
    blk.initialize(vars)
    blk.batch.set_solve(corrections)
    blk.forward(vars, blk.max_time_step(vars), 0)
    torch.cuda.synchronize()
    cells = nx1 * nx2
    return (blk.batch.scratch[0][85 * cells:90 * cells].clone(),
            blk.batch.solve_fallbacks()[0])


@pytest.mark.parametrize("nx1,nx2", [(5, 3), (6, 31), (7, 32), (12, 33), (17, 4),
                                     (33, 64), (40, 70)])
@pytest.mark.parametrize("corrections", [2, 3])
def test_refined_solution_at_tile_edges(cuda, nx1, nx2, corrections):
    got, left = solution(cuda, nx1, nx2, corrections)
    want, _ = solution(cuda, nx1, nx2, 0)
    assert left == 0
    assert (torch.linalg.norm(got - want) / torch.linalg.norm(want)).item() <= 1e-13


def test_fp32_solution_at_a_ragged_tile(cuda):
    """The FP32 solve (no corrections): the bar it has elsewhere."""
    got, left = solution(cuda, 12, 33, -1)
    want, _ = solution(cuda, 12, 33, 0)
    assert left == 0
    assert (torch.linalg.norm(got - want) / torch.linalg.norm(want)).item() <= 1e-4


def test_masked_columns_of_a_wide_batch(cuda):
    """A batch of more columns than the left-over solve has CTAs (several
    columns a CTA): a NaN in one cell leaves the columns its stencils reach to
    the FP64 solve, each counted once and failed there, the others untouched."""
    opts = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/convection3d.yaml")
    c = opts.coord()
    c.nx1, c.nx2, c.nx3 = 16, 96, 90
    c.x1max, c.x2max, c.x3max = 800.0, 4800.0, 4500.0
    opts.hydro().precision = opts.hydro().icorr.precision = "float32"
    opts.execution = "eager"
    opts.autotune = False
    blk = sg.MeshBlock(opts).to(cuda)
    vars = {"hydro_w": problems.convection3d(opts, cuda, seed=1)}
    blk.initialize(vars)
    dt = blk.max_time_step(vars)
    vars["hydro_u"][0, 3 + 40, 3 + 50, 3 + 8] = float("nan")
    blk.forward(vars, dt, 0)
    bad = torch.isnan(vars["hydro_u"][:, 3:-3, 3:-3, 3:-3]).any(dim=0).any(dim=-1)
    where = torch.nonzero(bad).cpu().tolist()
    want = {(40, 50)} | {(40 + d, 50) for d in range(-3, 4)} | {(40, 50 + d) for d in range(-3, 4)}
    assert {tuple(w) for w in where} == want
    assert blk.batch.solve_fallbacks()[0] == len(want)
