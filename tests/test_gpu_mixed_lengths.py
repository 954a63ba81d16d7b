"""An implicit member batched with a 1-D member far longer than any implicit
column (line_kernel's blocks have no columns to solve): the solve's kernels
are sized by the implicit blocks alone.  Lengths past which the finish's
arrays, sized by the 1-D member, would exceed a CTA's shared memory.  Each
member against itself alone, bit for bit."""
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems
from snapy_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def line(nx1):
    o = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/sod.yaml")
    c, h = o.coord(), o.hydro()
    c.nx1 = nx1
    h.riemann.type = "lmars"
    h.recon1.shock = h.recon23.shock = False
    h.precision = "float32"
    o.intg().cfl = 0.9
    w = problems.sod(o, "cpu")
    w[0] = w[4] = 1.0 + 0.1 * torch.sin(torch.arange(c.nc1, dtype=torch.float64) / 40.0)
    return o, w


def implicit(scheme, nx1, nx2):
    o = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/straka.yaml")
    c, h = o.coord(), o.hydro()
    c.nx1, c.nx2, c.x1max, c.x2max = nx1, nx2, nx1 * 50.0, nx2 * 50.0
    h.precision = h.icorr.precision = "float32"
    h.icorr.scheme = scheme
    return o, problems.straka(o, "cpu", xc=0.4 * c.x2max, zc=0.4 * c.x1max,
                              xr=0.3 * c.x2max, zr=0.3 * c.x1max)


def steps(cuda, members, dts):
    ens = Ensemble([o for o, _ in members], device=cuda)
    ens.initialize([w.to(cuda) for _, w in members], autotune=False)
    for _ in range(2):
        ens.step(torch.tensor(dts, dtype=torch.float64, device=cuda))
    torch.cuda.synchronize()
    return [ens.state(k).clone() for k in range(len(members))]


@pytest.mark.parametrize("scheme,nx1", [(9, 1500), (9, 5800), (1, 4200), (1, 5800)])
def test_long_line_beside_implicit_columns(cuda, scheme, nx1):
    members = [line(nx1), implicit(scheme, 40, 33), implicit(scheme, 9, 70)]
    dts = [2e-5, 0.1, 0.1]
    got = steps(cuda, members, dts)
    for k, (m, dt) in enumerate(zip(members, dts)):
        want = steps(cuda, [m], [dt])[0]
        assert torch.isfinite(want).all()
        assert torch.equal(got[k], want), k
