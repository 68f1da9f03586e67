"""Serving engine (continuous batching): results bitwise equal alone and in a mix,
admission under a memory cap, and a Poisson request stream through the request loop."""
import numpy as np
import pytest
import torch

from mun_b200 import Batch, SolveSpec, _lib
from mun_b200.serving import Engine, Request, serve
from tests.goldens import INJECT, load
from tests.gpu_cases import aligned_obs, dev, plan_for

pytestmark = pytest.mark.gpu


def _specs():
    out = []
    for name in INJECT + ["circle_n5"]:
        g = load(name)
        plan = plan_for(g["config"], g["dt"], g["nt"])
        y = dev(aligned_obs(g))
        inv = 1.0 / float(g["sigma"]) ** 2
        v = np.asarray(g["velocity"])
        out.append(lambda p=plan, v=v, y=y, inv=inv: SolveSpec(p, dev(v), adjoint=True, y_obs=y,
                                                                inv_sigma2=inv, ckpt_k=7))
        out.append(lambda p=plan, v=v, y=y, inv=inv: SolveSpec(p, dev(v * 1.01), misfit=True, y_obs=y,
                                                                inv_sigma2=inv, shift=True))
        out.append(lambda p=plan, v=v: SolveSpec(p, dev(v * 0.98)))
    return out


@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_engine_mix_is_bitwise_equal_to_alone(kernel):
    makers = _specs()
    alone = []
    for mk in makers:
        s = mk()
        Batch(kernel=kernel).run([s])
        alone.append(s)
    eng = Engine(max_solves=6, memory_cap_bytes=2 << 30, ticks_per_step=13, kernel=kernel)
    tickets = []
    for i, mk in enumerate(makers):  # staggered: a new request every few steps
        tickets.append(eng.submit(mk()))
        for _ in range(i % 3):
            eng.step()
    eng.run_until_done(tickets)
    torch.cuda.synchronize()
    for t, a in zip(tickets, alone):
        b = eng.release(t)
        assert torch.equal(a.rec, b.rec)
        if a.loglik is not None:
            assert torch.equal(a.loglik, b.loglik)
        if a.grad is not None:
            assert torch.equal(a.grad, b.grad)
        assert int(b.status.item()) == 0


def test_engine_memory_cap_queues_and_completes():
    makers = _specs()
    specs = [makers[12]() for _ in range(6)]  # six equal-size forward+adjoint solves (order 5)
    one = specs[0].plan.workspace_bytes(specs[0].flags, 7)
    assert one > (4 << 20)
    eng = Engine(max_solves=64, memory_cap_bytes=int(2.5 * one), ticks_per_step=32)
    tickets = [eng.submit(s) for s in specs]
    eng.step()
    st = eng.stats()
    assert st["running"] <= 2 and st["queued"] >= len(specs) - 2
    eng.run_until_done(tickets)
    for t in tickets:
        assert int(eng.release(t).status.item()) == 0
    assert eng.stats()["bytes_in_use"] == 0


def test_request_loop_poisson_stream():
    makers = _specs()
    rng = np.random.default_rng(0)
    arrivals = np.cumsum(rng.exponential(1.0 / 200.0, size=24))
    reqs = [Request(float(a), makers[i % len(makers)](), "mix") for i, a in enumerate(arrivals)]
    eng = Engine(max_solves=16, memory_cap_bytes=2 << 30, ticks_per_step=16)
    done, lat, wall = serve(eng, reqs)
    assert len(done) == len(reqs)
    assert np.all(lat > 0)
    print(f"served {len(done)} requests in {wall:.3f} s, p50 {1e3 * np.percentile(lat, 50):.1f} ms, "
          f"p99 {1e3 * np.percentile(lat, 99):.1f} ms")


def test_engine_marches_beside_ticks():
    # a solve too long for one march runs by ticks beside marched ones, whose workspaces are reused
    # by the next march while the last one may still run
    g = load(INJECT[0])
    y, v = dev(aligned_obs(g)), np.asarray(g["velocity"])
    inv = 1.0 / float(g["sigma"]) ** 2
    short, long_ = plan_for(g["config"], g["dt"], g["nt"]), plan_for(g["config"], g["dt"], 20100)

    def make(i):
        if i == 3:
            return SolveSpec(long_, dev(v))
        return SolveSpec(short, dev(v * (1.0 + 0.003 * i)), adjoint=i % 2 == 0, misfit=True, y_obs=y, inv_sigma2=inv,
                         shift=True, ckpt_k=(0, 7)[i % 4 == 0])
    alone = [make(i) for i in range(12)]
    for s in alone:
        Batch().run([s])
    one = max(s.plan.workspace_bytes(s.flags, s.ckpt_k or s.plan.nt) for s in alone)
    eng = Engine(max_solves=5, memory_cap_bytes=max(1 << 20, int(3.5 * one)), ticks_per_step=64)
    tickets = [eng.submit(make(i)) for i in range(12)]
    eng.run_until_done(tickets)
    for t, a in zip(tickets, alone):
        b = eng.release(t)
        assert int(b.status.item()) == 0
        assert torch.equal(a.rec, b.rec)
        assert a.loglik is None or torch.equal(a.loglik, b.loglik)
        assert a.grad is None or torch.equal(a.grad, b.grad)
    assert eng.stats()["bytes_in_use"] == 0 and eng.stats()["running"] == 0


@pytest.mark.parametrize("skip", [0, 1, 2])
def test_failed_march_gives_its_requests_back(skip):
    # a march's group cannot be set up: the requests of the groups before it are done, the others,
    # a solve by ticks among them, wait in the queue and finish with the next steps
    makers = _specs()
    kinds = [0, 1, 2, 3, 4, 5, 12, 13]  # gradients, likelihoods and forward solves of two orders and more
    g = load(INJECT[0])
    long_ = plan_for(g["config"], g["dt"], 20100)

    def make(i):
        return SolveSpec(long_, dev(np.asarray(g["velocity"]))) if i == 3 else makers[kinds[i]]()
    alone = [make(i) for i in range(len(kinds))]
    for s in alone:
        Batch().run([s])
    eng = Engine(max_solves=32, memory_cap_bytes=2 << 30, ticks_per_step=64)
    tickets = [eng.submit(make(i)) for i in range(len(kinds))]
    _lib.check(eng._lib.sem_selftest_fail_marches(eng.handle, skip, 2))
    for _ in range(2):
        before = eng.stats()
        with pytest.raises(MemoryError):
            eng.step()
        torch.cuda.synchronize()
        done = [t for t in tickets if eng.state(t) == 2]
        assert all(eng.state(t) == 0 for t in tickets if t not in done)
        assert len(done) + eng.stats()["queued"] == len(tickets) and before["queued"] >= eng.stats()["queued"]
        assert (len(done) > 0) == (skip > 0)
        assert eng.stats()["bytes_in_use"] == 0 and eng.stats()["running"] == 0
    eng.run_until_done(tickets)
    torch.cuda.synchronize()
    for t, a in zip(tickets, alone):
        b = eng.release(t)
        assert int(b.status.item()) == 0
        assert torch.equal(a.rec, b.rec)
        assert a.loglik is None or torch.equal(a.loglik, b.loglik)
        assert a.grad is None or torch.equal(a.grad, b.grad)
    assert eng.stats()["bytes_in_use"] == 0 and eng.stats()["running"] == 0 and eng.stats()["queued"] == 0
