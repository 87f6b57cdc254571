"""Edges of the fused sorted step: the particle counts of a cell around the 63
up to which its moment sums stay in 32 bits, and the step beside whose second
pass the whole GPU works a solve."""
import numpy as np
import pytest

import psum_b200 as P
from test_gpu_solves_beside import solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def identity_solver(nodes):
    """phi stays what it is: no cycles of an identity operator."""
    n = int(np.prod(nodes))
    s = P.solver_backend("cuda_multigrid64_gpu")
    k = tuple(nodes) + (1,) * (3 - len(nodes))
    s.set_options(f"I {k[0]} J {k[1]} K {k[2]} depth 1 max_cycles 0")
    idx = np.arange(n, dtype=np.uint64)
    s.set_matrix(n, n, n, idx, idx, np.ones(n))
    return s


@pytest.mark.parametrize("cells", [(60,), (8, 9), (4, 5, 4)])
@pytest.mark.parametrize("vel_scale", [0.0, 0.5])
def test_moment_sums_around_63_particles_in_a_cell(cells, vel_scale):
    """Cells of 0 to 97 particles (fewer than 64 on average), many of them in the cell's far corner, where a moment is
    largest; at rest (every particle stays in its cell's class) and moving: the fused step's density and state equal
    those of the general step and stable sort, bit for bit."""
    rng = np.random.default_rng(len(cells))
    dim, nc = len(cells), int(np.prod(cells))
    count = np.resize([63, 64, 62, 65, 0, 1, 31, 32, 33, 97, 63, 64], nc)
    assert count.mean() < 64
    cell = np.repeat(np.stack(np.unravel_index(np.arange(nc), cells)), count, axis=1)
    frac = rng.random((dim, cell.shape[1]))
    corner = rng.random(cell.shape[1]) < 0.5
    frac[:, corner] = 1.0 - 2.0 ** -20
    pos = cell + frac
    vel = rng.normal(size=(3, pos.shape[1])) * vel_scale
    nodes = [c + 1 for c in cells]
    out = []
    for interval in (1, 0):
        ctx = P.ParticleContext(cells, (0.0,) * dim, tuple(float(c) for c in cells), (1,) * dim, P.MIXED)
        ctx.set_options(f"sort_interval {interval}")
        sp = ctx.add_species(-1.0, 1.0, 0.5, pos.shape[1])
        ctx.load(sp, pos, vel)
        ctx.sort()
        ctx.deposit()
        phi = torch.tensor(np.random.default_rng(9).normal(size=int(np.prod(nodes))) * vel_scale, device="cuda")
        rho = torch.zeros_like(phi)
        ctx.step(identity_solver(nodes), 0.0, rho, phi, 0.1)
        if interval == 0:
            ctx.sort()
        density = torch.zeros_like(phi)
        ctx.density(sp, density)
        out.append((density.cpu().numpy(), *ctx.get_state(sp)))
    for a, b in zip(*out):
        assert (a.view(np.int64) == b.view(np.int64)).all()


@pytest.mark.parametrize("cells,per_cell", [((400, 400), 4), ((400, 400), 300), ((70, 60, 50), 20)])
def test_whole_gpu_solve_beside_a_second_pass(cells, per_cell):
    """Solves above 100,000 rows leave SMs to the pending second pass of the fused step: steps with them equal steps
    with the launched kernels, bit for bit (particles at every density the rule tells apart)."""
    dim, n = len(cells), int(np.prod(cells)) * per_cell
    nodes = tuple(c + 1 for c in cells)
    out = []
    for persist in (1, 0):
        s, b = solver("cuda_multigrid32f_gpu", nodes, f"tol 1e-8 max_cycles 12 persist {persist}")
        ctx = P.ParticleContext(cells, (0.0,) * dim, tuple(float(c) for c in cells), (0,) * dim, P.MIXED)
        ctx.set_options("sort_interval 1")
        sp = ctx.add_species(-1.0, 1.0, 1.0 / per_cell, n)
        g = torch.Generator(device="cuda").manual_seed(4)
        top = torch.tensor(cells, dtype=torch.float64, device="cuda")[:, None]
        pos = torch.rand(dim, n, dtype=torch.float64, device="cuda", generator=g) * top
        vel = torch.randn(3, n, dtype=torch.float64, device="cuda", generator=g)
        ctx.load(sp, pos, vel)
        del pos, vel
        ctx.sort()
        ctx.deposit()
        rho = torch.zeros(b.size, dtype=torch.float64, device="cuda")
        phi = torch.zeros_like(rho)
        for _ in range(4):
            ctx.step(s, 1.0, rho, phi, 0.1)
        out.append((phi, *ctx.get_state_device(sp)))
        torch.cuda.synchronize()
    for a, b in zip(*out):
        assert (a.view(torch.int64) == b.view(torch.int64)).all()
