"""A whole-GPU barrier that gives up is told to the caller.  Option
`barrier_polls 1` lets the barriers run out: their blocks go on with what is
there (all indices are the grid's, none come from data), end, and the next
call on the handle answers PSUM_ERR_INTERNAL."""
import numpy as np
import pytest

import psum_b200 as P
from test_gpu_solves_beside import solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cuda_multigrid32f_gpu", "cuda_multigrid64_gpu"])
@pytest.mark.parametrize("nodes,options", [((401, 401), ""), ((128, 128, 64), " tma_min_rows 1000000")])
def test_barrier_that_runs_out(kind, nodes, options):
    """The whole solve as one kernel, and the kernel of a cycle's coarse levels in the solve's graph."""
    s, b = solver(kind, nodes, "tol 1e-6 max_cycles 24" + options)
    k3 = f"K {nodes[2]} " if len(nodes) == 3 else ""
    bd = torch.tensor(b, device="cuda")
    ref, x = torch.zeros_like(bd), torch.zeros_like(bd)
    assert s.solve(bd, ref) == 0
    st = torch.cuda.Stream()
    s.set_options(k3 + "barrier_polls 1")

    def told(call):
        with pytest.raises(P.PsumError) as e:
            call()
        assert e.value.code == 8 and "stopped waiting" in str(e.value)

    s.solve_async(bd, x, st)
    told(s.last_stats)
    s.last_stats()                      # told once
    x.zero_()
    told(lambda: s.solve(bd, x))
    s.solve_async(bd, x, st)
    torch.cuda.synchronize()
    told(lambda: s.solve_async(bd, x, st))
    s.set_options(k3 + f"barrier_polls {1 << 22}")
    x.zero_()
    assert s.solve(bd, x) == 0
    assert (x == ref).all()


def test_step_after_a_stalled_solve():
    cells = (400, 400)
    s, b = solver("cuda_multigrid32f_gpu", (401, 401))
    ctx = P.ParticleContext(cells, (0.0, 0.0), (400.0, 400.0), (0, 0), P.MIXED)
    n = 200000
    rng = np.random.default_rng(3)
    e = ctx.add_species(1.0, 1.0, 1.0, n)
    ctx.load(e, rng.random((2, n)) * 400.0, rng.normal(size=(3, n)) * 0.1)
    ctx.sort()
    ctx.deposit()
    rho = torch.zeros(b.size, dtype=torch.float64, device="cuda")
    phi = torch.zeros_like(rho)
    ctx.step(s, 0.0, rho, phi, 0.1)
    s.set_options("barrier_polls 1")
    ctx.step(s, 0.0, rho, phi, 0.1)
    torch.cuda.synchronize()
    with pytest.raises(P.PsumError) as err:
        ctx.step(s, 0.0, rho, phi, 0.1)
    assert err.value.code == 8
