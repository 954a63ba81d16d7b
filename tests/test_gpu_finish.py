"""The implicit solve's finish where its schedule can go wrong: one column a
CTA and several, a last CTA of fewer, layer counts from three up (odd and even
pitches), members of different lengths sharing one launch, and the partial
matrix; one implicit step against the oracle at relative L2 1e-12 (FP64: the
same operations in the same order)."""
import numpy as np
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems
from snapy_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def options(nx1, nx2, scheme=9):
    opts = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/straka.yaml")
    c = opts.coord()
    c.nx1, c.nx2, c.x1max, c.x2max = nx1, nx2, nx1 * 50.0, nx2 * 50.0
    opts.hydro().icorr.scheme = scheme
    opts.execution = "eager"
    opts.autotune = False
    w = problems.straka(opts, "cpu", xc=0.4 * nx2 * 50.0, zc=0.4 * nx1 * 50.0,
                        xr=0.3 * nx2 * 50.0, zr=0.3 * nx1 * 50.0)
    g = torch.Generator().manual_seed(nx1 * 1000 + nx2)
    w[1:4] += torch.randn(w[1:4].shape, generator=g, dtype=torch.float64)
    return opts, w


def close(got, want):
    for v in range(5):
        assert np.linalg.norm(got[v] - want[v]) <= 1e-12 * np.linalg.norm(want[v]), v


# 3 x 700 and 20 x 1000: several columns a CTA, the last CTA ragged
@pytest.mark.parametrize("nx1,nx2", [(3, 700), (4, 5), (20, 1000), (33, 309), (128, 3)])
@pytest.mark.parametrize("scheme,form", [(9, 1), (9, 2), (1, 0)])
def test_finish_against_the_oracle(oracle, cuda, nx1, nx2, scheme, form):
    opts, w = options(nx1, nx2, scheme)
    blk = sg.MeshBlock(opts).to(cuda)
    vars = {"hydro_w": w.to(cuda)}
    blk.initialize(vars)
    from snapy_gb300 import _lib
    _lib.check(blk.batch.L.sg_set_schedule(blk.batch.h, None, form), "sg_set_schedule")
    ob = oracle.block_from_options(opts)
    u = ob.initialize(w.numpy())
    dt = blk.max_time_step(vars)
    for s in range(3):
        blk.forward(vars, dt, s)
        ob.stage(u, dt, s)
    close(vars["hydro_u"].cpu().numpy(), u)


def test_members_of_different_lengths(oracle, cuda):
    members = [options(a, b) for a, b in ((3, 40), (110, 64), (17, 333))]
    ens = Ensemble([o for o, _ in members], device=cuda)
    ens.initialize([w.to(cuda) for _, w in members], autotune=False)
    dts = ens.max_time_step().clone()
    ens.step(dts)
    for k, ((o, w), dt) in enumerate(zip(members, dts.cpu().tolist())):
        ob = oracle.block_from_options(o)
        u = ob.initialize(w.numpy())
        for s in range(3):
            ob.stage(u, dt, s)
        close(ens.state(k).cpu().numpy(), u)


@pytest.mark.parametrize("sizes", [[(100, 30), (30, 900)], [(7, 3), (6, 2600)],
                                   [(64, 607)], [(64, 900)]])
def test_both_forms_of_the_direct_solve(oracle, cuda, sizes):
    """Few long columns (a warp each) and many short ones (four a warp), in
    one launch and alone, few columns and past a warp's share."""
    members = [options(a, b) for a, b in sizes]
    ens = Ensemble([o for o, _ in members], device=cuda)
    ens.initialize([w.to(cuda) for _, w in members], autotune=False)
    dts = ens.max_time_step().clone()
    ens.step(dts)
    for k, ((o, w), dt) in enumerate(zip(members, dts.cpu().tolist())):
        ob = oracle.block_from_options(o)
        u = ob.initialize(w.numpy())
        for s in range(3):
            ob.stage(u, dt, s)
        close(ens.state(k).cpu().numpy(), u)
