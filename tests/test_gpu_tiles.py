"""Compiled line lengths at the edges of the tile rules, against the FP64
oracle: lines of 3 * 2^k on every axis (last radix 6 or 12), film convolutions
in split, whole and one-thread-per-component blocks, Z tiles that use fewer
rows than they hold."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# user (nx, ny, nz): Z lines of nx points, Y of 2 ny, X of 2 nz
GRIDS = [
    (3, 3, 3), (6, 6, 6), (12, 12, 12), (24, 24, 24), (48, 48, 3), (96, 24, 12), (192, 96, 2), (384, 8, 2), (768, 6, 1),
    (8, 192, 1), (8, 384, 1), (6, 768, 1), (4, 1536, 1), (6, 512, 1), (16, 128, 1), (16, 256, 1),
    (512, 64, 1), (768, 64, 1),   # one block of 4 columns per SM, and more
    (64, 147, 1), (64, 3, 50),    # rows around the number of SMs (run-time Y and X plans)
]


@pytest.mark.parametrize("grid", GRIDS)
def test_field(eng, cuda, grid):
    """2e-6 of the field's norm, as for every transform of a few stages."""
    import torch
    c = dict(grid=grid, cell=(4e-9, 4e-9, 4e-9), msat=1.1e6, aexch=1.5e-11, alpha=0.5, anis=1, k1=5e5, axis=(0, 0, 1),
             bext=(0.01, -0.02, 0.03))
    m = O.seeded_m(grid, 5, "random")
    s = eng.Solver(eng.mmx_params(**c))
    d, h = torch.from_numpy(m).cuda(), torch.empty(m.shape, device="cuda")
    s.field(d.data_ptr(), h.data_ptr())
    want = O.OracleSim(O.make_cfg(**c), m, bits=64).heff(m)
    got = h.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - want) < 2e-6 * np.linalg.norm(want)
    s.close()
