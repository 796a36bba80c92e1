"""The entry point whose scratch the library keeps per host thread (the reference's launcher signatures carry none):
under graph capture, where it may not grow, and when it grows while a graph holds it."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

BIG = (1024, 11008, 1024, 8)        # the named plan needs no scratch, the one a call prefers 39 MB
SMALL = (64, 1408, 1024, 8)         # under 8 MB either way: the block a thread starts with


def in_a_new_thread(body):
    """A thread has no scratch yet; what it raises is raised here."""
    failed = []

    def run():
        try:
            body()
        except BaseException as e:  # noqa: BLE001
            failed.append(e)
    thread = threading.Thread(target=run)
    thread.start()
    thread.join()
    if failed:
        raise failed[0]


def problem(pkg, shape):
    M, N, K, n_keep = shape
    p = pkg.formats.make_random(M, N, K, n_keep, seed=M)
    op = pkg.NMSpMM.from_problem(p)
    A, C = torch.from_numpy(p.A_km).cuda(), torch.empty((M, N), device="cuda")

    def launch():
        pkg.nmGEMM_huge_matrices_high_sparsity(A, op.B, op.D, op.column_info, C, M, N, K, op.W, 0.75, 1)
    launch()                                                             # (in this thread: loads the kernels)
    return op, A, C, launch


def test_a_first_call_under_capture_runs_the_plan_that_needs_no_scratch(pkg):
    op, A, C, launch = problem(pkg, BIG)
    want = op.matmul(A, tile=pkg.plan(op.desc(BIG[0])).tile)
    assert pkg.workspace_bytes(op.desc(BIG[0])) == 0 < pkg.call_workspace_bytes(op.desc(BIG[0]))

    def body():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            launch()
        C.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
    in_a_new_thread(body)
    assert torch.equal(C, want) and pkg.device_status() == 0


def test_a_graphs_scratch_outlives_a_larger_one(pkg):
    op, A, C, launch = problem(pkg, SMALL)
    big_op, big_A, big_C, big_launch = problem(pkg, BIG)
    assert 0 < pkg.call_workspace_bytes(op.desc(SMALL[0])) <= 8 << 20
    more = pkg.call_workspace_bytes(big_op.desc(BIG[0]))
    want, big_want = C.clone(), big_C.clone()

    def body():
        launch()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            launch()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        big_launch()
        torch.cuda.synchronize()
        assert free - torch.cuda.mem_get_info()[0] >= more - (2 << 20), "the block that the graph writes must not have been given back"
        C.fill_(float("nan"))
        big_C.fill_(float("nan"))
        for _ in range(2):
            graph.replay()
            big_launch()
        torch.cuda.synchronize()
        del graph
        assert pkg.load_library().nmspmm_release_cached() == 0
        assert torch.cuda.mem_get_info()[0] >= free
    in_a_new_thread(body)
    assert torch.equal(C, want) and torch.equal(big_C, big_want) and pkg.device_status() == 0
