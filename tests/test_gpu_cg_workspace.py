"""The work vectors that a storage keeps between CG solves: a solve gives the same bits whatever was
solved before it and on whichever stream, nothing of it runs after the call, and the buffers go back
on request and when the device runs out of memory."""
import numpy as np
import pytest

import hyteg_b200 as hg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    if hg.device_count() == 0:
        pytest.skip("no CUDA device")


def storage(level, cubes=1):
    return hg.PrimitiveStorage.cuboid((0, 0, 0), (1, 1, 1), cubes, cubes, cubes, level)


def solve(st, L, seed, iterations, dtype=np.float64, operator=hg.P1ConstantLaplaceOperator, spoil=False):
    A = operator(st, L, L)
    x, b = hg.P1Function("x", st, L, L, dtype=dtype), hg.P1Function("b", st, L, L, dtype=dtype)
    b.fill_random(seed, L)
    if spoil:
        b.interpolate(float("nan"), L, hg.Inner)
    hg.CGSolver(st, L, L, maxIter=iterations).solve(A, x, b, L)
    return x.to_numpy(L)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("L", [1, 3])
def test_solve_does_not_depend_on_earlier_ones(gpu, L, dtype):
    fresh = solve(storage(L), L, 5, 4, dtype)
    st = storage(L)
    solve(st, L, 6, 3, dtype, hg.P1ConstantMassOperator)
    solve(st, L, 7, 3, dtype, spoil=True)
    assert np.isfinite(fresh).all()
    assert np.array_equal(fresh, solve(st, L, 5, 4, dtype))


def test_stream_change_between_solves(gpu):
    import torch
    L = 6
    one = storage(L, 2)
    ref = [solve(one, L, 10 + k, 3) for k in range(4)]
    st = storage(L, 2)
    A = hg.P1ConstantLaplaceOperator(st, L, L)
    xs = [hg.P1Function("x", st, L, L) for _ in ref]
    bs = [hg.P1Function("b", st, L, L) for _ in ref]
    for k, b in enumerate(bs):
        b.fill_random(10 + k, L)
    st.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    cg = hg.CGSolver(st, L, L, maxIter=3)
    for k in range(len(ref)):
        st.set_stream(streams[k % 2].cuda_stream)
        cg.solve(A, xs[k], bs[k], L)
    assert all(s.query() for s in streams)  # the calls have returned, so their work is done
    for x, r in zip(xs, ref):
        assert np.array_equal(x.to_numpy(L), r)


def test_no_iterations(gpu):
    L = 2
    st = storage(L)
    assert not solve(st, L, 3, 0).any()
    assert st.release_workspace() == 0


def test_release(gpu):
    L = 3
    st = storage(L)
    first = solve(st, L, 5, 4)
    assert st.release_workspace() == 3 * 8 * st.level_size(L)
    assert st.release_workspace() == 0
    assert np.array_equal(first, solve(st, L, 5, 4))


def test_given_back_when_memory_runs_out(gpu):
    # two storages keep three vectors each; the memory left then holds none, so that a function of
    # a third storage and its second SOR buffer need what was kept
    import torch
    L = 7
    keepers = [storage(L, 2), storage(L, 2)]
    st = storage(L, 2)
    vector = 8 * st.level_size(L)
    A = hg.P1ConstantLaplaceOperator(st, L, L)
    x, b = hg.P1Function("x", st, L, L), hg.P1Function("b", st, L, L)
    b.fill_random(4, L)
    for k in keepers:
        solve(k, L, 5, 2)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - vector // 2, dtype=torch.uint8, device="cuda")
    try:
        y = hg.P1Function("y", st, L, L)
        assert [k.release_workspace() for k in keepers] == [0, 0]
        assert not y.to_numpy(L).any()
        A.smooth_sor(x, b, 1.0, L, hg.Inner)  # its second buffer
        st.synchronize()
    finally:
        del filler
        torch.cuda.empty_cache()


def test_release_while_another_thread_solves(gpu):
    import threading
    L = 3
    ref = solve(storage(L), L, 5, 4)
    stores, out = [storage(L), storage(L)], [[], []]

    def work(k):
        for _ in range(20):
            out[k].append(solve(stores[k], L, 5, 4))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    while any(t.is_alive() for t in threads):
        for st in stores:
            st.release_workspace()
    for t in threads:
        t.join()
    assert [len(o) for o in out] == [20, 20]
    assert all(np.array_equal(ref, x) for o in out for x in o)
