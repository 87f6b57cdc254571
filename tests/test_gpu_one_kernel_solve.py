"""Solves in one kernel (option `persist 1`, the default) against the same
solves with one kernel per step (`persist 0`).

Both work every row with the same operations in the same order and sum the
norms in one fixed order, so iterates, cycle counts and residuals are equal
bit for bit.  The cases lie at the edges of the kernel's dispatch: problems
that fit one block, one cluster, the whole GPU, and ones whose finest levels
stay launched; rows that wrap, rows with coefficients of their own, stencils
of no usual shape; no, one and three smoothing sweeps; coarse systems solved
by one block and by all."""
import threading

import numpy as np
import pytest

import psum_b200 as P

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BACKENDS = ["cuda_multigrid32f_gpu", "cuda_multigrid64_gpu"]


def box(nodes, periodic, pinned=True):
    """Poisson operator on a box: grounded faces, or wrapping with one pinned node."""
    cells = tuple(k - 1 for k in nodes)
    grid = P.simple_grid((0.0,) * len(nodes), tuple(float(c) for c in cells), cells)
    if periodic:
        fixed = np.zeros(1 if pinned else 0, np.uint64)
    else:
        wall = np.ones(nodes, bool)
        wall[tuple(slice(1, -1) for _ in nodes)] = False
        fixed = np.flatnonzero(wall).astype(np.uint64)
    r, c, v = P.assemble_poisson(grid, fixed, 1.0)
    b = np.random.default_rng(sum(nodes)).normal(size=int(np.prod(nodes)))
    b[fixed.astype(np.int64)] = 0.0
    return r, c, v, b, fixed


def solve(kind, opts, r, c, v, b, fixed=None, value=0.0):
    s = P.solver_backend(kind)
    s.set_options(opts)
    s.set_matrix(b.size, b.size, r.size, r, c, v)
    if fixed is not None and fixed.size:
        s.set_source_replace(fixed, np.full(fixed.size, value))
        s.set_source_addback(np.array([b.size // 2], np.uint64), np.array([0.125]))
    bd = torch.tensor(b, device="cuda")
    xd = torch.tensor(np.random.default_rng(1).normal(size=b.size) * 0.1, device="cuda")
    codes = [s.solve(bd, xd), s.solve(bd, xd)]
    k0 = P.lib().psum_kernel_launches()
    s.solve(bd, xd)
    return xd.cpu().numpy(), bd.cpu().numpy(), codes, s.last_stats(), P.lib().psum_kernel_launches() - k0


def both(kind, opts, *problem, **kw):
    one, many = (solve(kind, f"{opts} persist {p}", *problem, **kw) for p in (1, 0))
    assert (one[0].view(np.int64) == many[0].view(np.int64)).all()
    assert (one[1].view(np.int64) == many[1].view(np.int64)).all()
    assert one[2] == many[2] and one[3] == many[3]
    return one, many


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("nodes,periodic,depth", [
    ((64, 64), True, 4), ((17, 9), False, 2), ((5, 41), False, 1), ((95, 129), False, 4), ((130, 257), False, 5),
    ((320, 330), False, 4), ((96, 416), True, 5), ((8, 16, 32), True, 2), ((33, 41, 29), False, 3),
    ((47, 52, 50), False, 3), ((64, 48, 32), True, 4), ((9, 70, 11), False, 2), ((97, 33), False, 1)])
def test_equals_one_kernel_per_step(kind, nodes, periodic, depth):
    opts = (f"I {nodes[0]} J {nodes[1]} K {nodes[2] if len(nodes) == 3 else 1} depth {depth} pre_relax 2 post_relax 2 "
            f"max_cycles 20 correction_interval 2 tol 1e-9"
            + (" periodic_I 1 periodic_J 1" + (" periodic_K 1" if len(nodes) == 3 else "") if periodic else ""))
    r, c, v, b, fixed = box(nodes, periodic)
    one, many = both(kind, opts, r, c, v, b, fixed=fixed, value=0.25)
    assert one[4] == 1 and many[4] > 1


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("pre,post", [(0, 2), (1, 1), (2, 1), (3, 2), (2, 0), (5, 3)])
@pytest.mark.parametrize("nodes,periodic", [((65, 33), False), ((160, 640), True), ((24, 24, 40), False)])
def test_smoothing_counts_and_fixed_cycles(kind, pre, post, nodes, periodic):
    opts = (f"I {nodes[0]} J {nodes[1]} K {nodes[2] if len(nodes) == 3 else 1} depth 3 pre_relax {pre} post_relax {post} "
            "max_cycles 4 correction_interval 4" + (" periodic_I 1 periodic_J 1" if periodic else ""))
    r, c, v, b, fixed = box(nodes, periodic)
    both(kind, opts, r, c, v, b, fixed=fixed)


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("nodes", [(64, 96), (512, 256), (32, 32, 32)])
def test_mean_zero_gauge(kind, nodes):
    opts = (f"I {nodes[0]} J {nodes[1]} K {nodes[2] if len(nodes) == 3 else 1} depth 3 pre_relax 2 post_relax 2 "
            "max_cycles 20 correction_interval 2 tol 1e-9 periodic_I 1 periodic_J 1 periodic_K 1 null_space 1")
    r, c, v, b, _ = box(nodes, True, pinned=False)
    both(kind, opts, r, c, v, b + 0.3)


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("nodes,min_rows", [((48, 48, 48), 1 << 16), ((128, 128, 64), 1 << 20)])
def test_launched_finest_level(kind, nodes, min_rows):
    """A level that the TMA-staged sweep takes stays launched; the levels below it are one kernel per cycle (of one
    cluster, of one block per SM), captured into the solve's graph and its conditional loop."""
    opts = (f"I {nodes[0]} J {nodes[1]} K {nodes[2]} depth 3 pre_relax 2 post_relax 1 max_cycles 6 correction_interval 2 "
            f"tol 1e-9 periodic_I 1 periodic_J 1 periodic_K 1 tma_min_rows {min_rows}")
    r, c, v, b, fixed = box(nodes, True)
    one, many = both(kind, opts, r, c, v, b, fixed=fixed)
    assert 1 < one[4] < many[4]


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("nodes", [(64, 48), (96, 200), (400, 410)])
def test_captured_by_the_caller(kind, nodes):
    """A solve on a stream that the caller captures replays in the caller's graph with the bits of a direct one."""
    opts = f"I {nodes[0]} J {nodes[1]} depth 4 pre_relax 2 post_relax 2 max_cycles 8 correction_interval 2 tol 1e-9"
    r, c, v, b, fixed = box(nodes, False)
    s = P.solver_backend(kind)
    s.set_options(opts)
    s.set_matrix(b.size, b.size, r.size, r, c, v)
    bd, x, y = (torch.tensor(q, device="cuda") for q in (b, 0 * b, 0 * b))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    s.solve_async(bd, x, stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        s.solve_async(bd, y, stream)
    for _ in range(2):
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert (x == y).all()
    g.reset()


@pytest.mark.parametrize("kind", BACKENDS)
def test_unusual_stencils(kind):
    """1-D, cylindrical and variable-epsilon operators: three-point levels, levels that are mostly exception rows, and
    stencils of no usual shape."""
    g1 = P.simple_grid((0.0,), (1.0,), (200,))
    p1 = P.Poisson_solver_1d()
    p1.assemble(g1, [P.Dirichlet_point(g1, "L", 0.0), P.Dirichlet_point(g1, "R", 1.0)], 1.0)
    g2 = P.simple_grid((0.0, 0.0), (1.0, 1.2), (40, 48))
    p2 = P.Poisson_solver_2d()
    p2.assemble(g2, p2.Cylindrical, [P.Dirichlet_line(g2, d, 0.0) for d in "EWN"], 1.0)
    p3 = P.Poisson_solver_2d()
    p3.assemble(g2, p3.Cartesian, [P.Dirichlet_line(g2, d, 0.0) for d in "EW"], lambda x, y: 1.0 + x * y,
                [P.Neumann_line(g2, d, 0.0) for d in "NS"])
    for p, opts in ((p1, "I 201 J 1 K 1 depth 4"), (p2, "I 41 J 49 depth 3"), (p3, "I 41 J 49 depth 3")):
        r, c, v = p.coeff_matrix()
        b = np.random.default_rng(3).normal(size=p.grid.n_nodes)
        both(kind, opts + " pre_relax 2 post_relax 2 max_cycles 6 correction_interval 2 tol 1e-8", r, c, v, b,
             fixed=p.replace_idx, value=0.5)


def enqueue(s, stream, bs, xs):
    for b, x in zip(bs, xs):
        s.solve_async(b, x, stream)


@pytest.mark.parametrize("nodes", [(400, 410), (96, 96)])
def test_handles_on_two_streams_and_threads(nodes):
    """Solves of two handles on two streams, enqueued by two threads without a wait between them, equal solves alone."""
    r, c, v, b, fixed = box(nodes, False)
    opts = f"I {nodes[0]} J {nodes[1]} depth 4 pre_relax 2 post_relax 2 max_cycles 12 correction_interval 2 tol 1e-9"
    ref = solve(BACKENDS[0], opts, r, c, v, b)[0]
    runs = []
    for _ in range(2):
        s = P.solver_backend(BACKENDS[0])
        s.set_options(opts)
        s.set_matrix(b.size, b.size, r.size, r, c, v)
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            runs.append((s, st, [torch.tensor(b, device="cuda") for _ in range(8)],
                         [torch.tensor(np.random.default_rng(1).normal(size=b.size) * 0.1, device="cuda") for _ in range(8)]))
    torch.cuda.synchronize()
    threads = [threading.Thread(target=enqueue, args=run) for run in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for s, _, _, xs in runs:
        assert s.last_stats()["rel_residual"] <= 1e-9
        for x in xs[1:]:
            assert (x == xs[0]).all()
    assert (runs[0][3][0] == runs[1][3][0]).all()
    assert np.linalg.norm(runs[0][3][0].cpu().numpy() - ref) <= 1e-6 * np.linalg.norm(ref)
