"""Solves that run beside other work: graphs of the caller replayed at the
same time, direct solves of other handles between them."""
import numpy as np
import pytest

import psum_b200 as P

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BACKENDS = ["cuda_multigrid32f_gpu", "cuda_multigrid64_gpu"]


def solver(kind, nodes, options="tol 1e-9 max_cycles 24"):
    wall = np.ones(nodes, bool)
    wall[tuple(slice(1, -1) for _ in nodes)] = False
    fixed = np.flatnonzero(wall).astype(np.uint64)
    grid = P.simple_grid((0.0,) * len(nodes), tuple(float(k - 1) for k in nodes), tuple(k - 1 for k in nodes))
    r, c, v = P.assemble_poisson(grid, fixed, 1.0)
    b = np.random.default_rng(sum(nodes)).normal(size=int(np.prod(nodes)))
    b[fixed.astype(np.int64)] = 0.0
    s = P.solver_backend(kind)
    k = tuple(nodes) + (1,) * (3 - len(nodes))
    s.set_options(f"I {k[0]} J {k[1]} K {k[2]} depth 4 pre_relax 2 post_relax 2 correction_interval 2 " + options)
    s.set_matrix(b.size, b.size, r.size, r, c, v)
    return s, b


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("nodes", [(400, 410), (64, 96), (96, 96, 120)])
def test_callers_graphs_beside_one_another(kind, nodes):
    """Two graphs of the caller and a direct solve on three streams at once: each gives the bits of a direct solve
    alone (graphs of solves above 100,000 rows hold launched kernels, none that waits over the whole GPU)."""
    s0, b = solver(kind, nodes)
    ref_b, ref = torch.tensor(b, device="cuda"), torch.zeros(b.size, dtype=torch.float64, device="cuda")
    s0.solve(ref_b, ref)
    runs = []
    for _ in range(2):
        s, _ = solver(kind, nodes)
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            bd, x = torch.tensor(b, device="cuda"), torch.zeros(b.size, dtype=torch.float64, device="cuda")
        s.solve_async(bd, x, st)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            x.zero_()
            s.solve_async(bd, x, st)
        runs.append((s, st, bd, x, g))
    direct = torch.cuda.Stream()
    for _ in range(4):
        for s, st, _, _, g in runs:
            with torch.cuda.stream(st):
                g.replay()
        with torch.cuda.stream(direct):
            y = torch.zeros_like(ref)
        s0.solve_async(ref_b, y, direct)
        torch.cuda.synchronize()
        assert (y == ref).all()
        for s, _, _, x, _ in runs:
            assert (x == ref).all()
    for s, _, _, _, g in runs:
        assert s.last_stats()["rel_residual"] <= 1e-9
        g.reset()
