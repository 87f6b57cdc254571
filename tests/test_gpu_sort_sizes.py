"""The stable cell sort, the binning and the valid count at the edges of
their tiles: one item, a tile of 4096 less and plus one, keys of one to
three 8-bit passes, equal keys, sorted and reversed input, invalid particles,
both launch shapes of the gather (a state in arbitrary order and one sorted
before)."""
import numpy as np
import pytest

import psum_b200 as P

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def particles(cells, n, order, seed):
    rng = np.random.default_rng(seed)
    dim = len(cells)
    pos = rng.random((dim, n)) * np.array(cells)[:, None]
    if order == "one cell":
        pos = np.floor(pos[:, :1]) + rng.random((dim, n)) * 0.999
    key = np.zeros(n, np.int64)
    for a in range(dim):
        key = key * cells[a] + np.floor(pos[a]).astype(np.int64)
    if order in ("sorted", "reversed"):
        at = np.argsort(key, kind="stable")
        pos = pos[:, at if order == "sorted" else at[::-1]]
    if order == "invalid":
        pos[0, rng.random(n) < 0.3] = np.nan
    return pos, rng.normal(size=(3, n))


@pytest.mark.parametrize("precision", [P.MIXED, P.FP64])
@pytest.mark.parametrize("cells", [(3, 5), (100,), (200, 300), (70, 80, 90)])
@pytest.mark.parametrize("n,order", [(1, "random"), (3, "random"), (4095, "random"), (4096, "sorted"), (4097, "reversed"),
                                     (20000, "invalid"), (33333, "one cell"), (100001, "random")])
def test_sort_is_stable_and_complete(precision, cells, n, order):
    pos, vel = particles(cells, n, order, n + len(cells))
    dim = len(cells)
    ctx = P.ParticleContext(cells, (0.0,) * dim, tuple(float(c) for c in cells), (0,) * dim, precision)
    sp = ctx.add_species(1.0, 1.0, 1.0, n)
    ctx.load(sp, pos, vel)
    loaded, _ = ctx.get_state(sp)   # FP32 offsets may round onto a cell face
    keys = torch.empty(n, dtype=torch.int32, device="cuda")
    ctx.get_keys(sp, keys)
    k = keys.cpu().numpy().astype(np.int64)
    valid = int((k >= 0).sum())
    assert ctx.count(sp) == (n, valid)
    at = np.argsort(np.where(k < 0, np.iinfo(np.int64).max, k), kind="stable")[:valid]
    for _ in range(2):   # arbitrary order, then a state sorted before
        ctx.sort()
        assert ctx.count(sp) == (valid, valid)
        got_pos, got_vel = ctx.get_state(sp)
        assert (got_pos == loaded[:, at]).all()
        assert (got_vel == (vel if precision == P.FP64 else vel.astype(np.float32).astype(np.float64))[:, at]).all()


@pytest.mark.parametrize("n", [1, 4095, 4097, 50000])
def test_bin_twice(n):
    """Binning keeps its workspaces: a second call, on other sizes, gives the same answers as the first."""
    for cells in ((30, 40), (64, 65), (7, 9)):
        pos, vel = particles(cells, n, "random", n)
        ctx = P.ParticleContext(cells, (0.0, 0.0), tuple(float(c) for c in cells), (0, 0), P.FP64)
        sp = ctx.add_species(1.0, 1.0, 1.0, n)
        key = np.floor(pos[0]).astype(np.int64) * cells[1] + np.floor(pos[1]).astype(np.int64)
        for _ in range(2):
            ctx.load(sp, pos, vel)
            keys, perm = (torch.empty(n, dtype=torch.int64, device="cuda") for _ in range(2))
            counts, offsets = (torch.empty(cells[0] * cells[1], dtype=torch.int64, device="cuda") for _ in range(2))
            assert ctx.bin(sp, keys, counts, offsets, perm) == n
            ref = np.bincount(key, minlength=cells[0] * cells[1])
            assert (keys.cpu().numpy() == key).all() and (counts.cpu().numpy() == ref).all()
            assert (offsets.cpu().numpy() == np.cumsum(ref) - ref).all()
            assert (perm.cpu().numpy() == np.argsort(key, kind="stable")).all()
