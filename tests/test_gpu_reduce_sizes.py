"""The time-step reduction over a batch of very uneven blocks (more CTAs a
block than the small ones have cells for): every block's dt is the one it has
alone, bit for bit, from a cell anywhere in it."""
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems
from snapy_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def member(nx1, nx2, precision, at):
    o = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/straka_explicit.yaml")
    c = o.coord()
    c.nx1, c.nx2, c.x1max, c.x2max = nx1, nx2, nx1 * 50.0, nx2 * 50.0
    o.hydro().precision = precision
    w = problems.straka(o, "cpu")
    # one cell, the first or the last, sets the block's dt
    i, j = (3, 3) if at == 0 else (nx1 + 2, nx2 + 2)
    w[2, 0, j, i] = 40.0 + nx1
    return o, w


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("nblock", [4, 12])
def test_dt_of_uneven_blocks(cuda, precision, nblock):
    sizes = [(7, 5), (33, 9), (96, 700), (4, 4)] + [(8 + k, 6) for k in range(nblock - 4)]
    members = [member(a, b, precision, k % 2) for k, (a, b) in enumerate(sizes)]
    ens = Ensemble([o for o, _ in members], device=cuda)
    ens.initialize([w.to(cuda) for _, w in members], autotune=False)
    got = ens.batch.max_dt().clone()
    for k, (o, w) in enumerate(members):
        one = Ensemble([o], device=cuda)
        one.initialize([w.to(cuda)], autotune=False)
        assert one.batch.max_dt()[0] == got[k], k
        blk = sg.MeshBlock(o).to(cuda)
        vars = {"hydro_w": w.to(cuda)}
        blk.initialize(vars)
        assert blk.max_time_step(vars) == got[k].item()
