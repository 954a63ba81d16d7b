"""line_kernel's longest segments (64 cells, taken where 32-cell segments are
more than the SMs): full ones and a ragged last one, in one batch, each member
against the oracle at the bar of the shorter ones (1e-12)."""
import numpy as np
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems
from snapy_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("riemann", ["hllc", "lmars"])
def test_full_and_ragged_segments(oracle, cuda, riemann):
    members = []
    for nx1 in (2000, 2048, 1217):  # 166 segments of 32 cells, 84 of 64
        o = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/sod.yaml")
        o.coord().nx1 = nx1
        o.hydro().riemann.type = riemann
        w = problems.sod(o, "cpu")
        g = torch.Generator().manual_seed(nx1)
        w[1] += 0.3 * torch.rand(w[1].shape, generator=g, dtype=torch.float64)
        members.append((o, w))
    ens = Ensemble([o for o, _ in members], device=cuda)
    ens.initialize([w.to(cuda) for _, w in members], autotune=False)
    dts = torch.full((3,), 5e-5, dtype=torch.float64, device=cuda)
    for _ in range(2):
        ens.step(dts)
    for k, (o, w) in enumerate(members):
        ob = oracle.block_from_options(o)
        u = ob.initialize(w.numpy())
        for _ in range(2):
            ob.step(u, 5e-5)
        got = ens.state(k).cpu().numpy()
        for v in (0, 1, 4):
            assert np.linalg.norm(got[v] - u[v]) <= 1e-12 * np.linalg.norm(u[v]), (k, v)
