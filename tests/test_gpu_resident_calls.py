"""Calls that the resident kernels take over from the tick kernels: what callers could do with
those, they can do with these."""
import time

import numpy as np
import pytest
import torch

from mun_b200 import Batch, SEMPlan, _lib
from tests.test_gpu_resident import _compare, _plan, _same, _spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,nt,mode", [((20, 10), 60, "gradient"), ((60, 30), 90, "gradient"), ((60, 30), 91, "forward")])
def test_captured_run_replays_with_new_inputs(shape, nt, mode):
    # a captured run is replayed with new velocities; runs of the same batch come between
    p, c = _plan(*shape, 4, nt, 9, circle=True)
    kw = {"ckpt_k": 25} if mode == "gradient" else {}
    s = _spec(p, c, 1, mode, **kw)
    b, stream, graph = Batch(kernel=5), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        b.run([s])
    stream.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        b.run([s])
    first = s.velocity.clone()
    for scale in (1.0, 0.9, 1.02, 0.97, 1.0):
        s.velocity.copy_(first * scale)
        ref = _spec(p, c, 1, mode, **kw)
        ref.velocity = first * scale
        Batch(kernel=1).run([ref])
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert b.last_kernel == "resident"
        _same([ref], [s])
        b.run([s])
        torch.cuda.synchronize()
        _same([ref], [s])


def test_dense_array_on_one_side_stays_resident():
    # most receivers lie in one tile of a tiling that divides the mesh unevenly
    p, c = _plan(56, 31, 5, 60, 1)
    p = SEMPlan(**dict(p.kwargs, receivers=np.array([(181.0 + 0.2 * i, 61.0 + 1.7 * i) for i in range(81)])))
    ref, got = ([_spec(p, c, 20 + i, "gradient") for i in range(16)] for _ in range(2))
    Batch(kernel=1).run(ref)
    b = Batch(kernel=5)
    b.run(got)
    torch.cuda.synchronize()
    assert b.last_kernel == "resident"
    for r, s in zip(ref, got):
        assert torch.equal(r.rec, s.rec) and torch.equal(r.loglik, s.loglik) and torch.equal(r.grad, s.grad)


@pytest.mark.parametrize("mode,kw", [("forward", {}), ("likelihood", {}), ("gradient", {"ckpt_k": 20})])
def test_memory_budget_is_for_automatic_intervals(mode, kw):
    # a batch without automatic intervals runs as it does without a budget
    p, c = _plan(20, 10, 4, 50, 7, circle=True)
    b, seen, ref = Batch(), [], None
    for budget in (None, 2 * p.workspace_bytes(13 if mode == "gradient" else 0, 20)):
        got = [_spec(p, c, i, mode, **kw) for i in range(12)]
        b.run(got, memory_budget=budget)
        torch.cuda.synchronize()
        seen.append((b.last_kernel, b.last_groups, b.last_launches))
        _same(ref or got, got)
        ref = got
    assert seen[0] == seen[1] and seen[0][0] == "resident"


@pytest.mark.parametrize("npol,shape,nt,models,boundary,mode,kw,kernel", [
    (7, (23, 11), 40, 1, "sponge", "gradient", {}, "tile"),        # a tick's least time is less than a step's
    (7, (23, 11), 40, 4, "stacey", "gradient", {}, "tile"),
    (7, (23, 11), 40, 1, "stacey", "forward", {}, "tile"),
    (7, (157, 79), 20, 2, "sponge", "gradient", {}, "strip"),      # strips fill the GPU
    (4, (20, 10), 5, 1, "sponge", "forward", {}, "tile"),          # few steps
    (4, (100, 50), 8, 33, "sponge", "gradient", {}, "strip"),
    (4, (20, 10), 6, 1, "sponge", "forward", {}, "resident"),
    (4, (100, 50), 9, 33, "sponge", "gradient", {}, "resident"),
    (4, (20, 10), 30, 1, "sponge", "gradient", {"ckpt_k": 2}, "tile"),      # short segments
    (4, (20, 10), 30, 1, "sponge", "gradient", {"ckpt_k": 3}, "resident"),
    (5, (20, 10), 30, 2, "stacey", "gradient", {"ckpt_k": 3}, "tile"),
    (5, (20, 10), 30, 2, "stacey", "gradient", {"ckpt_k": 4}, "resident"),
    (6, (20, 10), 30, 1, "sponge", "gradient", {"ckpt_k": 7}, "tile"),
    (6, (20, 10), 30, 1, "sponge", "gradient", {"ckpt_k": 8}, "resident"),
    (2, (20, 10), 30, 1, "sponge", "gradient", {"ckpt_k": 2}, "resident"),
    (7, (57, 29), 30, 2, "sponge", "gradient", {"ckpt_k": 15}, "tile"),
    (7, (57, 29), 30, 2, "sponge", "gradient", {"ckpt_k": 16}, "resident"),
    (7, (11, 6), 40, 1, "sponge", "gradient", {}, "resident"),
    (7, (23, 11), 40, 1, "sponge", "forward", {}, "resident"),
    (7, (57, 29), 40, 2, "stacey", "gradient", {}, "resident"),
])
def test_automatic_kernel_is_the_faster_one(npol, shape, nt, models, boundary, mode, kw, kernel):
    p, c = _plan(*shape, npol, nt, 9, boundary, circle=shape[0] > 8)
    ref, got = ([_spec(p, c, 3 + i, mode, **kw) for i in range(models)] for _ in range(2))
    Batch(kernel=5).run(ref)
    b = Batch()
    b.run(got)
    torch.cuda.synchronize()
    assert b.last_kernel == kernel
    for r, s in zip(ref, got):
        assert int(r.status.item()) == int(s.status.item()) == 0 and torch.equal(r.rec, s.rec)
        assert r.grad is None or torch.equal(r.grad, s.grad)


@pytest.mark.parametrize("window", [(13, 88, 3), (0, 20, 1), (90, 97, 2)])
def test_stacey_edges_with_a_misfit_window(window):
    # (the waves of the first 20 steps do not meet: that window's gradient is 0)
    p, c = _plan(11, 12, 4, 97, 8, "stacey")
    for k in (0, 7):
        ref, got = (_spec(p, c, 3, "gradient", ckpt_k=k, window=window) for _ in range(2))
        Batch(kernel=1).run([ref])
        b = Batch(kernel=5)
        b.run([got])
        torch.cuda.synchronize()
        assert b.last_kernel == "resident" and int(ref.status.item()) == int(got.status.item()) == 0
        assert torch.equal(ref.rec, got.rec) and torch.equal(ref.loglik, got.loglik) and torch.equal(ref.grad, got.grad)
        assert window[1] == 20 or float(got.grad.abs().max()) > 0.0


@pytest.mark.parametrize("nelx,nelz,boundary", [(330, 171, "sponge"), (345, 180, "stacey")])
def test_fields_in_memory_over_several_segments(nelx, nelz, boundary):
    # an automatic interval below the number of steps: the adjoint fields pass from segment to segment
    p, c = _plan(nelx, nelz, 4, 120, 8, boundary, circle=True)
    b = _compare(lambda: [_spec(p, c, 3, "gradient")], memory_budget=p.workspace_bytes(13, 35))
    assert b.last_ticks > 2 * 120 + 2  # steps were replayed


@pytest.mark.parametrize("kernel", [1, 2])
def test_schedule_of_ticks_with_explicit_and_forward_solves(kernel):
    # explicit intervals and forward solves keep their settings inside a batch that ticks run in groups
    p, c = _plan(20, 10, 3, 90, 7, circle=True)

    def make(k, k1):
        return [_spec(p, c, i, "gradient", ckpt_k=(k, k1)[i == 1]) for i in range(4)] + [_spec(p, c, 9, "forward")]
    ref, got, b = make(90, 90), make(0, 7), Batch(kernel=kernel)
    Batch(kernel=5).run(ref)
    b.run(got, memory_budget=int(0.6 * (3 * p.workspace_bytes(13, 13) + p.workspace_bytes(13, 7) + p.workspace_bytes(0, 2))))
    torch.cuda.synchronize()
    assert b.last_groups >= 2 and b.last_kernel == {1: "tile", 2: "strip"}[kernel]
    _same(ref, got)


def test_exchange_wait_gives_up_with_status():
    # a tile that never runs: its neighbours' waits for its words run out, and the next call is right again
    p, c = _plan(60, 30, 4, 40, 9, circle=True)
    b, ref, got = Batch(kernel=5), _spec(p, c, 1, "forward"), _spec(p, c, 1, "forward")
    Batch(kernel=1).run([ref])
    b.run([got])
    torch.cuda.synchronize()
    assert b.last_kernel == "resident"
    _same([ref], [got])
    _lib.check(b._lib.sem_selftest_drop_tile(b.handle))
    t0 = time.perf_counter()
    b.run([got])
    torch.cuda.synchronize()
    dt = time.perf_counter() - t0
    assert int(got.status.item()) == _lib.SEM_ERR_TIMEOUT and 1.5 < dt < 30.0
    b.run([got])
    torch.cuda.synchronize()
    _same([ref], [got])


@pytest.mark.parametrize("npol,shape,nt,models,mode,kw", [
    (4, (100, 50), 5, 16, "forward", {}), (5, (60, 30), 20, 24, "gradient", {"ckpt_k": 2})])
def test_what_ticks_refuse_stays_resident(npol, shape, nt, models, mode, kw):
    # more receivers in one strip's band than strips take, in batches that are faster by ticks
    p, c = _plan(*shape, npol, nt, 1)
    p = SEMPlan(**dict(p.kwargs, receivers=np.stack([np.linspace(3.0, 340.0, 300), np.full(300, 10.0)], 1)))
    ref, got = ([_spec(p, c, 3 + i, mode, **kw) for i in range(models)] for _ in range(2))
    with pytest.raises(ValueError):
        Batch(kernel=2).run([_spec(p, c, 3, mode, **kw)])
    Batch(kernel=5).run(ref)
    b = Batch()
    b.run(got)
    torch.cuda.synchronize()
    assert b.last_kernel == "resident"
    for r, s in zip(ref, got):
        assert torch.equal(r.rec, s.rec) and (r.grad is None or torch.equal(r.grad, s.grad))
