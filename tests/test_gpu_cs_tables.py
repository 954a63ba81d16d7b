"""The sphere's FP64 handle reads its caller's tables in place: tables that are
filled after sg_cs_create and before the first stage count as they then are,
also when that first stage is captured."""
import ctypes

import pytest
import torch

from snapy_gb300 import _lib, cubed_sphere

pytestmark = pytest.mark.gpu


class Late(cubed_sphere.SphereSW):
    """SphereSW whose tables hold zeros while the handle is created."""

    def __init__(self, *args, **kw):
        super().__init__(*args, **kw)
        full = [self._geo, self._gt, self._st, self._sst]
        late = [torch.zeros_like(t) for t in full]
        d = _lib.CsDesc()
        d.n, d.ng, d.dtype, d.nstage = self.n, 3, _lib.F64, self.nstage
        for s, w in enumerate(cubed_sphere.RK3):
            for q in range(3):
                d.wght[s][q] = w[q]
        d.cfl, d.riemann = 0.9, 1
        d.geo, d.ghost_tab, d.seam_tab, d.seam_state_tab = (t.data_ptr() for t in late)
        d.nghost, d.nseam, d.nseam_state = (t.shape[0] for t in full[1:])
        h = ctypes.c_void_p()
        _lib.check(self.L.sg_cs_create(ctypes.byref(d), ctypes.byref(h)), "sg_cs_create")
        self.close()
        self.h, self._late = h, late
        _lib.check(self.L.sg_cs_bind(h, *(self.store[q].data_ptr() for q in range(3)),
                                     self.scratch.data_ptr(), self.scratch.numel() * 8),
                   "sg_cs_bind")
        for a, b in zip(late, full):
            a.copy_(b)


@pytest.mark.parametrize("captured", [False, True])
def test_tables_filled_after_create(cuda, captured):
    out = []
    for kind in (cubed_sphere.SphereSW, Late):
        sp = kind(12, dtype=torch.float64, device=cuda, riemann="hllc")
        sp.initialize(cubed_sphere.bump(12, seed=2))
        if captured and kind is Late:  # every rotation's first step too
            sp._seen = {((c, b), False) for c in range(3) for b in range(3)}
        for _ in range(4):
            sp.step(40.0)
        out.append(sp.state().clone())
    assert torch.isfinite(out[0]).all()
    assert torch.equal(out[0], out[1])
