"""Passes over several steps (four, two or one: step.cu pass_at) against one pass per step, FP64.

The passes sum the same products; those with Dirichlet values of the pass's own steps are added
after the rest.  Bound: FP64 sums of a few hundred products in another order, amplified over at most
a hundred steps by less than 1e3 (measured 1e-15 over 64 steps), so 1e-12 relative L2.
"""
import numpy as np
import pytest

from helpers import rel_l2, sine_acc, sphere_small
from pppm_b200 import Solver, scenes

pytestmark = pytest.mark.gpu


def _run(geom, many, calls, chunk=32, precision="fp64", pml=0):
    v, f, h, mn, dt, res, cell = geom
    s = Solver(res, h, dt, mn, precision=precision, pml_width=pml)
    s.set_option("conv_pairs", many[0])
    s.set_option("terms_pairs", many[1])
    s.set_option("graph_chunk", chunk)
    s.set_mesh(v, f)
    s.add_listener(*cell)
    acc = sine_acc(sum(calls), len(f), 1500.0, dt)
    # a triangle-dependent factor, so that no two neighbours' values are interchangeable
    acc = (acc * (1 + 0.1 * np.sin(np.arange(len(f))))).astype(np.float32)
    at = 0
    for n in calls:
        s.step(acc[at: at + n])
        at += n
    out = s.series(), s.grid(0).copy(), s.dump("dirichlet")
    counts = s.dump("counts")
    s.close()
    return out, counts


def _small():
    v, f, h, mn, dt = sphere_small()
    return v, f, h, mn, dt, 24, (20, 20, 20)


# every remainder of a pass at a call's end, calls of one to three steps (direct launches) between,
# chunks that whole passes do not divide, calls of several chunks
@pytest.mark.parametrize("many", [(1, 1), (1, 0), (0, 1)])
@pytest.mark.parametrize("calls,chunk", [((4, 5, 6, 7, 8, 9), 32), ((12, 1, 13, 3, 14, 2), 32), ((41, 42, 15), 6),
                                         ((43, 40), 0), ((70,), 32)])
def test_passes_match_single_steps(gpu, many, calls, chunk):
    (a, ga, da), _ = _run(_small(), (0, 0), calls, chunk)
    (b, gb, db), _ = _run(_small(), many, calls, chunk)
    assert np.all(np.isfinite(b)) and np.abs(b).max() > 0
    assert rel_l2(b, a) < 1e-12 and rel_l2(gb, ga) < 1e-12 and rel_l2(db, da) < 1e-12


@pytest.mark.parametrize("many", [(1, 1), (1, 0), (0, 1)])
@pytest.mark.parametrize("calls", [(4, 5, 6, 7), (41, 2, 15, 1)])
def test_pml_passes_match_single_steps(gpu, many, calls):
    (a, ga, da), _ = _run(_small(), (0, 0), calls, pml=4)
    (b, gb, db), _ = _run(_small(), many, calls, pml=4)
    assert np.all(np.isfinite(b)) and np.abs(b).max() > 0
    assert rel_l2(b, a) < 1e-12 and rel_l2(gb, ga) < 1e-12 and rel_l2(db, da) < 1e-12


def _dense(sub, res, precision):
    """A dense scene in passes against one pass per step.  FP32: the sums in another order, below 1e-6 over
    so few steps (as test_pairs_match_single_pass_fp32)."""
    rng = np.random.default_rng(3)
    v, f = scenes.perturbed_sphere(sub, 0.1, 0.1, rng)
    h, mn = scenes.grid_for_bbox(v.min(0), v.max(0), res, 2.0)
    dt = np.float32(0.5 * h / (np.sqrt(3) * 340.3))
    geom = (v.astype(np.float32), f, h, mn, dt, res, (res // 2, res // 2, res - 4))
    (a, ga, da), counts = _run(geom, (0, 0), (22,), precision=precision)
    (b, gb, db), _ = _run(geom, (1, 1), (22,), precision=precision)
    tol = 1e-12 if precision == "fp64" else 1e-6
    assert rel_l2(b, a) < tol and rel_l2(gb, ga) < tol and rel_l2(db, da) < tol
    return len(f), counts[4] * 5 // 4  # pairs: the lists have a quarter to spare


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_dense_scene_completes_by_groups(gpu, precision):
    """20480 triangles in a res-56 grid, 3.6 M pairs: more triangles and pairs than the thresholds from
    which the completion of the convolution takes a group of centres per warp (step.cu: make_launch)."""
    nt, pairs = _dense(5, 56, precision)
    assert nt >= 15000 and pairs >= 1250000


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_dense_scene_completes_by_triangle(gpu, precision):
    """5120 triangles in a res-24 grid, 1.3 M pairs: as many pairs, too few triangles for groups."""
    nt, pairs = _dense(4, 24, precision)
    assert nt < 15000 and pairs >= 1250000


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("pml", [0, 4])
def test_first_steps_on_one_branch(gpu, pml, precision):
    """A handle's first steps replay one-branch graphs, later ones (step.cu: branch_steps, at most 1024 steps
    behind or before the handle) branched graphs with the split stencil.  The same calls on a new handle and
    on one that has 1100 steps behind it and was set back to rest, absorbing boundary and PML: every sample
    and the whole state (grids, auxiliary fields, histories) bit-identical."""
    v, f, h, mn, dt, res, cell = _small()
    calls = (64, 37, 100, 9, 4, 33, 70, 5)
    acc = sine_acc(1100, len(f), 1500.0, dt)
    out = []
    for before in (0, 1100):
        s = Solver(res, h, dt, mn, pml_width=pml, precision=precision)
        s.set_mesh(v, f)
        s.add_listener(*cell)
        if before:
            s.step(acc[:before])
            s.reset_fields()
            s.rewind_listeners()
            s.t = -1
        at = 0
        for n in calls:
            s.step(acc[at: at + n])
            at += n
        out.append((s.series(0, at), s.grid(0).copy(), s.grid(-1).copy(), s.grid(-2).copy(), s.dump("dirichlet"),
                    s.dump("neumann"), np.frombuffer(s.save_state(), np.uint8)))
        s.close()
    assert np.all(np.isfinite(out[0][0]))
    for a, b in zip(*out):
        assert np.any(a) and np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 3])
def test_short_calls_replay_their_kernels(gpu, n):
    """From a handle's 16th call of fewer than four steps on, the call's kernels are replayed as a graph;
    moved to a new handle every 10 calls (state saved and restored), the same run launches them
    directly.  Bit-identical."""
    v, f, h, mn, dt, res, cell = _small()
    calls = 40
    acc = sine_acc(calls * n, len(f), 1500.0, dt)

    def new(state=None):
        s = Solver(res, h, dt, mn)
        s.set_mesh(v, f)
        s.add_listener(*cell)
        if state is not None:
            s.restore_state(state)
        return s

    s = new()
    for k in range(calls):
        s.step(acc[k * n: (k + 1) * n])
    a, ga = s.series(), s.grid(0).copy()
    s.close()
    s, b = new(), []
    for k in range(calls):
        if k and k % 10 == 0:
            b.append(s.series())
            state = s.save_state()
            s.close()
            s = new(state)
        s.step(acc[k * n: (k + 1) * n])
    b.append(s.series())
    gb = s.grid(0).copy()
    s.close()
    assert np.array_equal(a, np.concatenate(b)) and np.array_equal(ga, gb)


@pytest.mark.parametrize("pml", [0, 4])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_recorded_single_steps_equal_direct_launches(gpu, precision, pml):
    """One step per pass, recorded in calls of 13 and 4 steps, against the same steps in calls of one
    (fused face stage): both sum a triangle's face pairs in the same association.  Bit-identical."""
    v, f, h, mn, dt, res, cell = _small()
    acc = sine_acc(34, len(f), 1500.0, dt)
    out = []
    for calls in ((13, 4, 17), (1,) * 34):
        s = Solver(res, h, dt, mn, precision=precision, pml_width=pml)
        s.set_option("conv_pairs", 0)
        s.set_option("terms_pairs", 0)
        s.set_mesh(v, f)
        s.add_listener(*cell)
        at = 0
        for n in calls:
            s.step(acc[at: at + n])
            at += n
        out.append((s.series(), s.grid(0).copy(), s.grid(-1).copy(), s.dump("dirichlet")))
        s.close()
    for a, b in zip(*out):
        assert np.any(a) and np.array_equal(a, b)


def test_short_calls_on_a_stream_that_cannot_be_captured(gpu):
    """Calls of one to three steps and a gradient over less than 128 reverse steps on the legacy default
    stream, which cannot be captured: their kernels are recorded on a stream of the handle's own.  The same
    bits as on a stream that the handle makes."""
    v, f, h, mn, dt, res, cell = _small()
    acc = sine_acc(60, len(f), 1500.0, dt)
    out = []
    for stream in (None, 1):  # 1: cudaStreamLegacy
        s = Solver(res, h, dt, mn, stream=stream)
        s.set_mesh(v, f)
        s.add_listener(*cell)
        for k in range(0, 60, 3):
            s.step(acc[k: k + 3])
        out.append((s.series(), s.grid(0).copy(), s.adjoint(np.ones((60, 1), np.float32))))
        s.close()
    for a, b in zip(*out):
        assert np.any(a) and np.array_equal(a, b)


def test_short_calls_keep_the_recorded_graphs(gpu):
    """A program that steps in eight lengths (as many as a handle keeps recorded graphs) with calls of one
    to three steps between: the short calls' graphs have slots of their own, so no longer call is
    recorded again.  A cycle of the mixture queues 53 kernels more than one without the short calls (1.4 times
    its time); recorded again in every call it took 15 times as long."""
    import time

    import torch

    v, f, h, mn, dt, res, cell = _small()
    acc = torch.from_numpy(sine_acc(1100, len(f), 1500.0, dt)).cuda()
    best = []
    for mixed in (False, True):
        s = Solver(res, h, dt, mn)
        s.set_mesh(v, f)
        s.step(acc)  # past the one-branch graphs of a handle's first steps
        times = []
        for cycle in range(40):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for i in range(8):
                s.step(acc[:4 + i])
                if mixed:
                    s.step(acc[:1 + i % 3])
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
        best.append(min(times[20:]))
        s.close()
    assert best[1] < 5 * best[0], best


def test_short_calls_with_changing_launches_stay_direct(gpu):
    """One-step calls whose launch set changes from call to call (here by options, 24 sets in turn; a moving
    ghost-cell scene does so at every frame) are not recorded again and again: they cost direct launches
    (less than twice the replayed ones); recorded in every call they took eight times as long."""
    import itertools
    import time

    import torch

    v, f, h, mn, dt, res, cell = _small()
    acc = torch.from_numpy(sine_acc(24, len(f), 1500.0, dt)).cuda()
    best = []
    sets = list(itertools.product((0, 1), (0, 1), (64, 128, 256), (0, 1)))
    for change in (False, True):
        s = Solver(res, h, dt, mn)
        s.set_mesh(v, f)
        times = []
        for cycle in range(30):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for k in range(len(sets)):
                for name, value in zip(("conv_pairs", "terms_pairs", "face_threads", "stencil_vec4"), sets[k * change]):
                    s.set_option(name, value)
                s.step(acc[k: k + 1])
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
        best.append(min(times[10:]))
        s.close()
    assert best[1] < 5 * best[0], best
