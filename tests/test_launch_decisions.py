"""What the library's host code launches, without a GPU: the objects of the
library run over a fake CUDA runtime (tests/fake_cuda.py) that refuses what a
device would refuse and logs every launch."""
import ctypes as C
import shutil

import numpy as np
import pytest

import fake_cuda as F

M32, M64 = "cuda_multigrid32f_gpu", "cuda_multigrid64_gpu"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or shutil.which("nvcc") is None:
        pytest.skip("no compiler")
    return F.Fake(str(tmp_path_factory.mktemp("fake") / "libpsum_fake.so"))


@pytest.fixture
def fake(lib):
    lib.reset()
    yield lib
    lib.reset()


@pytest.mark.parametrize("kind,nodes,options,blocks", [
    (M64, (64, 64), "", 1), (M32, (96, 96), "", 16), (M32, (400, 410), "", "sms"), (M64, (48, 48, 48), "", "sms"),
    (M32, (32, 32, 32), "tma_min_rows 1000", None), (M64, (32, 32, 32), "tma_min_rows 1000", None)])
def test_a_second_device_of_the_process(fake, kind, nodes, options, blocks):
    """Kernel attributes and SM counts belong to a device: what ran on the first runs on the second, with its SMs."""
    for device, sms in ((0, 148), (1, 100)):
        fake.lib.fake_device(device, sms)
        s = F.Solver(fake, kind, nodes, options)
        fake.lib.fake_clear_log()
        s.check(s.solve_async(fake.stream()))
        if blocks:
            (k,) = fake.kernels("k_mg_persist")
            assert (k.device, k.grid) == (device, sms if blocks == "sms" else blocks)
        else:
            assert fake.kernels("k_level_op_tma")
        s.close()


@pytest.mark.parametrize("kind", [M32, M64])
@pytest.mark.parametrize("how", [1, 4])
def test_whole_gpu_solve_refused(fake, kind, how):
    """A device, or a share of one, that does not take the cooperative kernel solves with the launched kernels."""
    if how == 4:
        fake.lib.fake_device(2, 148)   # asked for once per device
    fake.lib.fake_refuse_cooperative(how)
    s = F.Solver(fake, kind, (400, 410))
    s.set_source(np.array([7]), np.array([1.0]))
    fake.lib.fake_clear_log()
    st = fake.stream()
    for _ in range(2):
        s.check(s.solve_async(st))
    assert not fake.kernels("k_mg_persist") and fake.kernels("k_level_op<")
    assert len([q for q in fake.kernels("k_addback") if q.captured != 1]) == 2
    s.close()


@pytest.mark.parametrize("kind,options", [(M32, "tol 1e-9"), (M32, ""), (M64, "tol 1e-9")])
@pytest.mark.parametrize("how", [1, 2])
def test_whole_gpu_cycle_refused(fake, kind, options, how):
    """The same for the kernel of a cycle's coarse levels, in the solve's graph (refused when it is instantiated) and
    launched on a stream that takes no graph."""
    fake.lib.fake_refuse_cooperative(how)
    s = F.Solver(fake, kind, (64, 64, 272), "depth 4 tma_min_rows 1000000 " + options)
    s.set_source(np.array([7]), np.array([1.0]))
    fake.lib.fake_clear_log()
    st = fake.stream() if how == 2 else C.c_void_p(1)   # 1: the legacy default stream
    for _ in range(2):
        s.check(s.solve_async(st))
    ran = [q for q in fake.log() if q.captured != 1]
    assert not [q for q in ran if b"k_mg_persist" in q.name]
    names = [q.name.split(b"<")[0].split(b"(")[0] for q in ran]
    assert names.count(b"psum_b200::k_addback") == 2
    assert sum(b"k_dense_mv" in n for n in names) > 0
    s.close()


@pytest.mark.parametrize("kind,nodes,options,one_kernel", [
    (M32, (400, 410), "tol 1e-9", False), (M64, (400, 410), "", False), (M32, (64, 64, 272), "depth 4 tol 1e-9 tma_min_rows 1000000", False),
    (M64, (64, 64), "", True), (M32, (96, 96), "tol 1e-9", True)])
def test_solve_captured_by_the_caller(fake, kind, nodes, options, one_kernel):
    """The caller may replay its graphs beside one another and beside direct solves: nothing in them may wait for blocks
    over the whole GPU.  One block, or one cluster, is placed whole and may."""
    s = F.Solver(fake, kind, nodes, options)
    st = fake.stream()
    fake.lib.fake_clear_log()
    s.check(s.solve_async(st))
    assert any(q.cooperative for q in fake.log()) != one_kernel   # a direct solve takes the whole-GPU kernel
    fake.lib.fake_clear_log()
    assert fake.lib.cudaStreamBeginCapture(st, 0) == 0
    s.check(s.solve_async(st))
    g = C.c_void_p()
    fake.lib.cudaStreamEndCapture(st, C.byref(g))
    log = fake.log()
    assert log and not any(q.cooperative for q in log)
    assert (len(log) == 1) == one_kernel
    fake.lib.fake_clear_log()
    s.check(s.solve_async(st))   # and the next direct solve takes it again
    assert any(q.cooperative for q in fake.log()) != one_kernel
    s.close()


def test_a_stall_is_told_by_the_next_call(fake):
    """The pinned word that a kernel sets when it gives up a wait reaches the caller whichever call comes next, once."""
    s = F.Solver(fake, M32, (33, 33))
    step, close = F.step_context(fake, (32, 32))
    st = fake.stream()
    for call in (s.solve, lambda: s.solve_async(st), s.last_stats, lambda: step(s)):
        assert call() == 0
        fake.set_host_words(1)
        assert call() == 8 and b"stopped waiting" in fake.lib.psum_last_error()
        assert call() == 0
    close()
    fake.set_host_words(1)
    s.close()
    s = F.Solver(fake, M32, (33, 33))   # the word of a handle that is gone
    assert s.solve() == 0
    s.close()


def test_graph_of_a_solve_is_the_same_beside_a_pending_pass(fake):
    """A graph captured while a fused step's second pass is pending is replayed by solves that run alone: its kernels
    take every SM whatever was pending at the capture."""
    nodes = (64, 64, 272)
    s = F.Solver(fake, M32, nodes, "depth 4 tma_min_rows 1000000")
    step, close = F.step_context(fake, tuple(k - 1 for k in nodes), n=1000)
    assert step(s) == 0 and step(s) == 0
    s.set_options("K 272 max_cycles 2")   # the graph is captured again, beside the pending pass
    fake.lib.fake_clear_log()
    assert step(s) == 0
    assert fake.kernels("k_cls_pass2")    # there is one
    s.check(s.solve_async(fake.stream()))
    assert {q.grid for q in fake.kernels("k_mg_persist") if q.captured != 1} == {148}
    close()
    s.close()


@pytest.mark.parametrize("per_row,blocks", [(0.01, 148), (7.9, 148), (8, 98)])
def test_share_of_the_gpu_beside_a_pending_pass(fake, per_row, blocks):
    """A whole solve leaves SMs to the pending second pass where that lasts; a short one (few particles per row) would
    not use them."""
    s = F.Solver(fake, M32, (331, 331))
    step, close = F.step_context(fake, (330, 330), n=int(per_row * 331 * 331 + 1))
    fake.lib.fake_clear_log()
    assert step(s) == 0 and step(s) == 0
    assert [q.grid for q in fake.kernels("k_mg_persist")] == [148, blocks]   # nothing is pending at the first
    close()
    s.close()


def test_tables_only_where_a_kernel_reads_them(fake):
    """The one-kernel solve's own copies of the exception rows (with varying coefficients: many) are made
    for the levels that it can work, and not with `persist 0`."""
    def bytes_of(nodes, options):
        before = fake.lib.fake_device_bytes()
        eps = 1.0 + np.random.default_rng(2).random(nodes[0])   # per row of nodes; the uniform half gives the stencil
        eps[:nodes[0] // 2] = 1.0
        s = F.Solver(fake, M64, nodes, options, eps=np.broadcast_to(eps[:, None], nodes))
        return s, fake.lib.fake_device_bytes() - before

    nodes = (160, 160)
    s1, with_ = bytes_of(nodes, "persist 1")
    s0, without = bytes_of(nodes, "persist 0")
    assert with_ - without > 160 * 160 // 2 * 5 * 8       # the fine operator's exception rows alone
    before = fake.lib.fake_device_bytes()
    s0.set_options("persist 1")                           # asked for later: made then
    assert fake.lib.fake_device_bytes() - before == with_ - without
    fake.lib.fake_clear_log()
    s0.check(s0.solve_async(fake.stream()))
    assert len(fake.log()) == 1
    s0.close()
    s1.close()
    nodes = (1049, 2000)                                  # 1000 rows above the largest level that the kernel takes
    s1, with_ = bytes_of(nodes, "depth 7 persist 1")
    s1.close()
    s0, without = bytes_of(nodes, "depth 7 persist 0")
    s0.close()
    n = nodes[0] * nodes[1]
    assert with_ - without < (n // 4 + n // 16 + n // 64) * 1.1 * (9 * 8 + 2)
