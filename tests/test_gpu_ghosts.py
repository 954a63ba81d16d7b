"""Every ghost of a filled block is its side's image of the interior, bit for
bit: walls, periodic and open sides, axes as short as the ghosts are deep and a
cell more, 1-D to 3-D, FP64 and FP32 (no base: the base's change of rows is
covered by the parity tests)."""
import pytest
import torch

import snapy_gb300 as sg
from snapy_gb300 import problems

pytestmark = pytest.mark.gpu

NG = 3
SIDES = {"w": "reflecting", "p": "periodic", "o": "extrapolation"}


def images(u, sides):
    """the ghosts from the interior, an axis at a time: x1, x2, x3"""
    u = u.clone()
    for axis, side in enumerate(sides):
        dim, n = 3 - axis, u.shape[3 - axis]
        for g in range(NG):
            for at, src in ((g, {"w": 2 * NG - 1 - g, "p": n - 2 * NG + g, "o": NG}),
                            (n - 1 - g, {"w": n - 2 * NG + g, "p": 2 * NG - 1 - g,
                                         "o": n - NG - 1})):
                row = u.select(dim, src[side]).clone()
                if side == "w":
                    row[1 + axis] *= -1
                u.select(dim, at).copy_(row)
    return u


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("size,sides", [
    ((3, 1, 1), "o"), ((40, 1, 1), "w"), ((300, 1, 1), "p"), ((9, 3, 1), "op"),
    ((3, 4, 1), "ww"), ((130, 33, 1), "wo"), ((7, 3, 3), "wpw"), ((12, 5, 4), "pwo"),
    ((20, 16, 31), "oop")])
def test_ghosts_are_images_of_the_interior(cuda, size, sides, precision):
    opts = sg.MeshBlockOptions.from_yaml("snapy_gb300/decks/sod.yaml")
    c = opts.coord()
    c.nx1, c.nx2, c.nx3 = size
    opts.hydro().precision = precision
    opts.bcnames = sum(([f"{SIDES[s]}_inner", f"{SIDES[s]}_outer"] for s in sides), [])
    opts.execution = "eager"
    opts.autotune = False
    w = problems.sod(opts, "cpu")
    g = torch.Generator().manual_seed(sum(size))
    w[0] *= 1 + 0.2 * torch.rand(w[0].shape, generator=g, dtype=torch.float64)
    w[1:4] = 0.1 * torch.randn(w[1:4].shape, generator=g, dtype=torch.float64)
    blk = sg.MeshBlock(opts).to(cuda)
    vars = {"hydro_w": w.to(cuda)}
    blk.initialize(vars)
    for _ in range(2):
        u = vars["hydro_u"].cpu()
        assert torch.equal(u, images(u, sides))
        blk.step(vars, 0.25 * blk.max_time_step(vars))
