"""The chain sweep's teams against the level schedule.

A handle alone sweeps with teams of up to four warps per chain; launched beside
others it keeps to its budget (chain_warps: teams of one at 3 and 8 here, of
two at 32).  Every budget, alone, launched and in a batch, gives the level
schedule's bits: one chain, chains shorter than a team, more chains than points
per level, walls and varying frames (points outside the shared frame),
supersonic copies and the backup driver (terms from before the sweep).
"""
import dataclasses
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _cloud(kind):
    from mfcfd import cloud
    c = cloud.small_sphere(6, 100, r1=1.5, seed=3)
    if kind == "supersonic":
        return cloud.with_supersonic_boundary(cloud.small_sphere(8, 150, seed=4))
    if kind == "frames":
        # one interior point with turned axes: no shared frame
        t1, t2 = c.tan1.copy(), c.tan2.copy()
        i = int(np.flatnonzero(c.status == 0)[5])
        t1[i], t2[i] = (0.0, 1.0, 0.0), (-1.0, 0.0, 0.0)
        return dataclasses.replace(c, tan1=t1, tan2=t2)
    return c


CASES = {"sphere": {}, "supersonic": {}, "frames": {}, "backup": {"sweep_variant": 1}}


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("warps", [1, 3, 8, 32, 400])
def test_team_sweeps_equal_the_level_schedule(mfcfd_lib, case, warps):
    from mfcfd import batch
    from mfcfd.solver import Solver
    c = _cloud(case)
    # the backup driver reaches NaN at outer points within a few iterations
    iters = 1 if case == "backup" else 4
    ss = [Solver(c, 0.5, 1.0, sweep_mode=1, **CASES[case])] + \
         [Solver(c, 0.5, 1.0, chain_warps=warps, **CASES[case]) for _ in range(4)]
    for s in ss:
        s.initial_conditions()
    ss[0].q_lskum(iters)
    ss[1].q_lskum(iters)                       # alone: the largest team
    ss[2].launch(1, iters)                     # within its budget
    ss[2].complete()
    batch.run_batch(ss[3:], iters)             # a share of the device each
    for f in ("DELUP", "DELUN", "PRIM"):
        want = ss[0].get(getattr(mfcfd_lib, "FIELD_" + f))
        for s in ss[1:]:
            assert np.array_equal(s.get(getattr(mfcfd_lib, "FIELD_" + f)).view(np.uint64), want.view(np.uint64)), f
    for s in ss:
        s.close()


@pytest.mark.parametrize("name,args", [("ieee_check", ["128"]), ("flux_check", [])])
def test_straight_line_functions_equal_the_operators(tmp_path, name, args):
    """mfcfd_ieee.cuh and state_flux against the operators (tests/NAME.cu): no
    result differs."""
    exe = str(tmp_path / name)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-o", exe,
                    os.path.join(REPO, "tests", name + ".cu")], check=True)
    out = subprocess.run([exe] + args, capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.parametrize("iters", [1, 6])
def test_turned_shared_frame_equals_the_level_schedule(mfcfd_lib, iters):
    """Interior points that share a frame other than the global axes: its own
    kernels, in every team size, and in a group beside a cloud in the axes."""
    from mfcfd import batch, cloud
    from mfcfd.solver import Solver
    c = cloud.small_sphere(6, 100, r1=1.5, seed=3)
    t1, t2, nor = c.tan1.copy(), c.tan2.copy(), c.nor.copy()
    (ca, sa), (cb, sb) = (np.cos(0.3), np.sin(0.3)), (np.cos(0.5), np.sin(0.5))
    inner = c.status == 0
    t1[inner], t2[inner], nor[inner] = (ca, sa, 0.0), (-sa * cb, ca * cb, sb), (sa * sb, -ca * sb, cb)
    axes = c
    c = dataclasses.replace(c, tan1=t1, tan2=t2, nor=nor)
    ss = [Solver(c, 0.5, 1.0, sweep_mode=1)] + [Solver(c, 0.5, 1.0, chain_warps=w) for w in (0, 3, 32, 32)]
    others = [Solver(axes, 0.5, 1.0, chain_warps=32) for _ in range(2)]
    for s in ss + others:
        s.initial_conditions()
        assert s.info()["shared_frame"] == 1
    for s in ss[:2]:
        s.q_lskum(iters)                       # alone: the largest team
    for s in ss[2:4]:
        s.launch(1, iters)                     # teams of one and of two
        s.complete()
    others[0].q_lskum(iters)
    batch.run_group([others[1], ss[4]], iters)
    assert np.array_equal(*[s.get(mfcfd_lib.FIELD_PRIM) for s in others])
    for f in ("DELUP", "DELUN", "PRIM"):
        want = ss[0].get(getattr(mfcfd_lib, "FIELD_" + f))
        for s in ss[1:]:
            assert np.array_equal(s.get(getattr(mfcfd_lib, "FIELD_" + f)).view(np.uint64), want.view(np.uint64)), f
    for s in ss + others:
        s.close()
