"""The B-spline deposit of positions stored cell by cell: warps over one cell,
over two to four runs of cells (summed run by run through the transpose) and
over more, runs across lane 16, unsupported positions between and inside runs,
a last warp that is not full.

Bound: as in test_gpu_bspline, (contributions to a node) * 2^-(F+1) * weight
and FP64 rounding against the oracle; and the same bits as the same positions
in random order, whose warps take the other paths (the sums are of integers)."""
import numpy as np
import pytest

import psum_b200 as P
from psum_b200 import interp as I
from oracle import oracle as O
from test_gpu_bspline import _contributions, dev

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# lanes of the runs of one warp; a negative number: positions without support
WARPS = [(32,), (16, 16), (15, 17), (1, 31), (31, 1), (5, 20, 7), (14, 3, 15), (8, 8, 8, 8), (1, 1, 29, 1), (3, 10, 2, 17),
         (6, 6, 6, 6, 8), (1,) * 32, (10, -2, 20), (-1, 31), (31, -1), (7, 9, -1, 15), (12, -3, 1, 16), (4, -2, 10, -2, 14), (-32,)]


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_runs_of_cells_in_a_warp(order, dim):
    rng = np.random.default_rng(100 * order + dim)
    cells = (40, 9, 7)[:dim]
    lower = np.array((-0.5, 0.25, 1.0)[:dim])
    upper = lower + np.array((2.3, 1.7, 1.1)[:dim])
    dx = (upper - lower) / np.array(cells)
    grid, g = P.simple_grid(lower, upper, cells), O.make_grid(cells, lower, upper, (0,) * dim)
    pos, runs_in = [], []
    for _ in range(3):
        for warp in WARPS:
            last = None
            for k in warp:
                while True:   # neighbouring runs lie in different cells; the outermost cells' stencils wrap
                    cell = np.array([rng.integers(0, c) for c in cells])
                    if last is None or (cell != last).any():
                        break
                last = cell
                p = lower[:, None] + (cell[:, None] + rng.uniform(0.01, 0.99, (dim, abs(k)))) * dx[:, None]
                if k < 0:
                    p[rng.integers(0, dim), :] = np.nan
                pos.append(p)
    pos.append(lower[:, None] + dx[:, None] * rng.uniform(0.1, 0.9, (dim, 13)))   # a last warp of 13
    pos = np.concatenate(pos, axis=1)
    nn = int(np.prod([c + 1 for c in cells]))
    w, lost = 0.37, int(np.isnan(pos).any(axis=0).sum())
    skipped = torch.zeros(1, dtype=torch.int64, device="cuda")
    out = dev(np.zeros(nn))
    P.add_back_B_spline(order, grid, dev(pos), w, out, skipped=skipped)
    got = out.cpu().numpy()
    assert int(skipped.item()) == lost
    ref, ref_skipped = O.bspline_deposit(g, order, pos, w, nn)
    assert ref_skipped == lost
    F = I.deposit_bits(pos.shape[1])
    assert (np.abs(got - ref) <= _contributions(g, order, pos, nn) * 2.0 ** -(F + 1) * w + 1e-13 * (1 + np.abs(ref))).all()
    out2 = dev(np.zeros(nn))
    P.add_back_B_spline(order, grid, dev(pos[:, rng.permutation(pos.shape[1])]), w, out2)
    assert (out2.cpu().numpy().view(np.int64) == got.view(np.int64)).all()
