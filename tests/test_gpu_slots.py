"""Slots of chain sweeps (mfcfd_debug_slots): held while a chunk runs, all
returned when every call is over, however it ended."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _held():
    from mfcfd import _lib
    v = ctypes.c_int32(-1)
    assert _lib.lib().mfcfd_debug_slots(0, ctypes.byref(v)) == 0
    return v.value


def _solvers(cloud, count, **kw):
    from mfcfd.solver import Solver
    ss = [Solver(cloud, 0.5, 1.0, **kw) for _ in range(count)]
    for s in ss:
        s.initial_conditions()
    return ss


def test_run_between_launch_and_complete_keeps_the_count(mfcfd_lib, small_cloud):
    from mfcfd import batch
    ss = _solvers(small_cloud, 2)
    budget = ss[0].info()["chain_slots"]
    ss[0].launch(1, 3)
    assert _held() == budget
    ss[0].q_lskum(2, t0=4)                 # its own slots; the launch keeps its
    assert _held() == budget
    batch.run_batch(ss, 2)
    assert _held() == budget
    ss[0].complete()
    assert _held() == 0
    ss[1].launch(3, 2)                     # never completed
    assert _held() == budget
    for s in ss:
        s.close()
    assert _held() == 0


def test_failed_runs_return_their_slots(mfcfd_lib, small_cloud):
    from mfcfd import batch
    from mfcfd._lib import MfcfdError
    ss = _solvers(small_cloud, 2)
    prim = ss[0].get(mfcfd_lib.FIELD_PRIM)
    prim[7, 4] = np.nan                    # a residual that is not finite
    for run in (lambda: ss[0].q_lskum(2), lambda: batch.run_batch(ss, 2), lambda: batch.run_group(ss, 2)):
        for s in ss:
            s.initial_conditions(prim)
        with pytest.raises(MfcfdError):
            run()
        assert _held() == 0
    for s in ss:
        s.close()


def test_runs_from_two_threads_give_the_bits_of_runs_alone(mfcfd_lib):
    import threading
    from mfcfd import batch, cloud
    from mfcfd.solver import Solver
    clouds = [cloud.shell_cloud(26, 361, seed=s, knn_device=0) for s in (1, 2, 3)]
    ref = [Solver(c, 0.5, 1.0) for c in clouds]
    ss = [Solver(c, 0.5, 1.0) for c in clouds]
    for s in ref + ss:
        s.initial_conditions()
    want = [s.q_lskum(70) for s in ref]
    got = [None] * 3

    def run():
        got[0] = ss[0].q_lskum(70)

    def group():
        got[1] = batch.run_group(ss[1:2], 70)[0]

    threads = [threading.Thread(target=run), threading.Thread(target=group)]
    for t in threads:
        t.start()
    ss[2].launch(1, 70)
    got[2] = ss[2].complete()
    for t in threads:
        t.join()
    for s, r, g, w in zip(ss, ref, got, want):
        assert np.array_equal(g, w)
        assert np.array_equal(s.get(mfcfd_lib.FIELD_PRIM), r.get(mfcfd_lib.FIELD_PRIM))
    assert _held() == 0
    for s in ss + ref:
        s.close()


def test_batch_of_different_block_sizes_gives_the_bits_of_runs_alone(mfcfd_lib):
    from mfcfd import batch, cloud
    from mfcfd.solver import Solver
    c = cloud.shell_cloud(26, 361, seed=4, knn_device=0)
    kinds = [{}, {"precision": 1}, {"precision": 2}, {"chain_spread": 1}, {"chain_warps": 40}] * 3
    ref = [Solver(c, 0.5, 1.0, **k) for k in kinds[:5]]
    ss = [Solver(c, 0.5, 1.0, **k) for k in kinds]
    for s in ref + ss:
        s.initial_conditions()
    want = [s.q_lskum(6) for s in ref]
    got = batch.run_batch(ss, 6)
    for i, s in enumerate(ss):
        assert np.array_equal(got[i], want[i % 5])
        assert np.array_equal(s.get(mfcfd_lib.FIELD_PRIM), ref[i % 5].get(mfcfd_lib.FIELD_PRIM))
    assert _held() == 0
    for s in ss + ref:
        s.close()


def test_chunks_beyond_the_budget_are_parts_of_longer_ones(mfcfd_lib, small_cloud):
    """A batch of 100 iterations and a server's chunks of 100 run in parts of at
    most 64 where they hold more slots than their budgets: same bits, and a
    request ends with a whole chunk."""
    from mfcfd import batch, serve
    ref, s = _solvers(small_cloud, 2)
    want = ref.q_lskum(200)
    for k in (0, 1):
        assert np.array_equal(batch.run_batch([s], 100)[0], want[100 * k:100 * k + 100])
    with serve.Server(chunk=100) as srv:
        r = srv.wait(srv.submit(small_cloud, 0.5, 1.0, max_iters=150, residue_target=-99.0), timeout=120)
        st = srv.stats()
    assert r["status"] == 0 and r["iters"] == 200
    assert np.array_equal(r["prim"], ref.get(mfcfd_lib.FIELD_PRIM)) and r["res_new"] == want[-1, 0]
    assert st["rounds"] == 2 and st["iterations"] == 200
    ref.close()
    s.close()


def test_a_small_cloud_steps_beside_a_run_that_fills_the_device(mfcfd_lib):
    """A run that holds every slot leaves another thread's cloud room from its
    next chunk on, so that it steps while the run goes on."""
    import threading
    import time
    from mfcfd import cloud
    from mfcfd.solver import Solver
    big = Solver(cloud.shell_cloud(96, 11500, seed=7, knn_device=0), 0.5, 1.0, gpu_setup=1)
    (small,) = _solvers(cloud.small_sphere(6, 100, r1=1.5, seed=3), 1)
    big.initial_conditions()
    (ref,) = _solvers(cloud.small_sphere(6, 100, r1=1.5, seed=3), 1)
    over = []
    th = threading.Thread(target=lambda: (big.q_lskum(100), over.append(1)))
    th.start()
    time.sleep(0.2)                        # of about 2.6 s
    steps = 0
    while not over and steps < 200:
        steps += 1
        small.fpi_solver(steps)
    th.join()
    assert steps >= 100
    ref.q_lskum(steps)
    assert np.array_equal(small.get(mfcfd_lib.FIELD_PRIM), ref.get(mfcfd_lib.FIELD_PRIM))
    for s in (big, small, ref):
        s.close()
