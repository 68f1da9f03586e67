"""Calls that the resident kernels take over from the tick kernels: what callers could do with
those, they can do with these."""
import numpy as np
import pytest
import torch

from mun_b200 import Batch, SEMPlan
from tests.test_gpu_resident import _plan, _same, _spec

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
