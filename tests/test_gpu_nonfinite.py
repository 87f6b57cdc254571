"""Infinite and NaN values in a solve's vectors: the status and the residuals
that the caller reads, the same from the one-kernel solve and the launched
kernels."""
import math

import numpy as np
import pytest

import psum_b200 as P
from test_gpu_solves_beside import solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BACKENDS = ["cuda_multigrid32f_gpu", "cuda_multigrid64_gpu"]


def outcome(kind, nodes, options, node, value):
    s, b = solver(kind, nodes, "tol 1e-9 max_cycles 6 " + options)
    bd = torch.tensor(b, device="cuda")
    x = torch.zeros_like(bd)
    x[node] = value
    code = P.lib().psum_mg_solve(s.handle, bd.data_ptr(), x.data_ptr())
    return code, s.last_stats()


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("nodes", [(17, 9), (96, 130), (320, 400), (24, 24, 40), (48, 52, 56)])
@pytest.mark.parametrize("node", [0, -1])
def test_infinite_guess_at_a_fixed_node(kind, nodes, node):
    """Rows beside the walls have fewer taps than the stencil: a value that they do not read is not read."""
    one, many = (outcome(kind, nodes, f"persist {p}", node, math.inf) for p in (1, 0))
    assert one == many
    assert one[0] == 5 and one[1]["rel_residual"] == math.inf


@pytest.mark.parametrize("kind", BACKENDS)
@pytest.mark.parametrize("persist", [1, 0])
def test_nan_residual_is_told(kind, persist):
    """A residual that is no number is read as one that is none (the adjoint's convergence check asks whether it is
    finite), not as zero."""
    code, stats = outcome(kind, (33, 41), f"persist {persist}", 500, math.nan)
    assert code == 5 and math.isnan(stats["rel_residual"]) and math.isnan(stats["initial_rel_residual"])
