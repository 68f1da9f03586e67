"""Resident kernels (kernel 5: tiles held on chip for a whole sweep, edge nodes exchanged as
tagged words) against the tile kernel: bitwise the same traces, log-likelihoods and gradients,
for every order, both boundary modes, windows, replay, ragged meshes and mixed batches."""
import numpy as np
import pytest
import torch

from mun_b200 import Batch, SEMPlan, SolveSpec
from mun_b200.mesh import create_global_mesh

pytestmark = pytest.mark.gpu


def _plan(nelx, nelz, npol, nt, nrec, boundary="sponge", circle=False):
    X, Z = 20.0 * nelx, 20.0 * nelz
    coords, _, grid = create_global_mesh(0.0, X, 0.0, Z, nelx, nelz, npol)
    if circle:
        a = np.linspace(0, 2 * np.pi, nrec, endpoint=False)
        R = min(0.4 * X, 0.3 * Z, 60.0)  # around the source, so that few steps reach the receivers
        rec = np.stack([0.45 * X + R * np.cos(a), 0.3 * Z + R * np.sin(a)], 1)
    else:
        rec = np.stack([np.linspace(0.0, X, nrec), np.full(nrec, 10.0)], 1)
    dt = 0.35 * (20.0 / (npol + 1)) / (3300.0 * (npol + 1) * np.sqrt(2.0))
    return SEMPlan(xmin=0.0, xmax=X, zmin=0.0, zmax=Z, nelx=nelx, nelz=nelz, npol=npol, dt=dt, nt=nt,
                   src_xz=(0.45 * X, 0.3 * Z), f0=25.0, amp=1.0, receivers=rec, pml_thickness=0.15 * X,
                   sponge_cmax=3000.0, coords=coords, node_grid=grid, boundary=boundary), coords


def _velocity(coords, seed):
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(80, 300, 2)
    return torch.as_tensor(2300.0 + 700.0 * np.sin(coords[:, 0] / a) * np.cos(coords[:, 1] / b), device="cuda")


def _spec(p, coords, seed, mode, **kw):
    s = SolveSpec(p, _velocity(coords, seed), **kw)
    if mode != "forward":
        it0, it1, dec = s.window or (0, p.nt, 1)
        g = torch.Generator().manual_seed(seed)
        s.y_obs = 1e-9 * torch.randn(-(-(it1 - it0) // dec), p.nrec, generator=g, dtype=torch.float64).cuda()
        s.misfit, s.inv_sigma2, s.adjoint = True, 1e12, mode == "gradient"
    return s


def _same(ref, got):
    for a, b in zip(ref, got):
        assert int(a.status.item()) == 0 and int(b.status.item()) == 0
        for o in ("rec", "loglik", "grad"):
            x, y = getattr(a, o), getattr(b, o)
            assert (x is None) == (y is None)
            if x is not None:
                assert torch.equal(x, y), o
                assert o != "grad" or x.numel() < 100 or float(x.abs().max()) > 0.0


def _compare(make, **kw):
    ref, got = make(), make()
    Batch(kernel=1).run(ref)
    b = Batch(kernel=5)
    b.run(got, **kw)
    torch.cuda.synchronize()
    assert b.last_kernel == "resident"
    _same(ref, got)
    return b


@pytest.mark.parametrize("npol", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("boundary", ["sponge", "stacey"])
def test_gradient_of_every_order(npol, boundary):
    p, c = _plan(13, 9, npol, 60 + 40 * npol, 11, boundary)
    _compare(lambda: [_spec(p, c, 1, "gradient", exact=npol % 2 == 0)])


@pytest.mark.parametrize("shape", [(1, 1), (1, 9), (2, 1), (8, 5), (37, 23), (100, 50)])
@pytest.mark.parametrize("mode", ["forward", "likelihood", "gradient"])
def test_mesh_shapes_and_modes(shape, mode):
    p, c = _plan(*shape, 4, 70, 9, circle=shape[0] > 8)
    _compare(lambda: [_spec(p, c, 2, mode, shift=mode == "likelihood")])


@pytest.mark.parametrize("k", [2, 7, 40])
@pytest.mark.parametrize("boundary", ["sponge", "stacey"])
def test_replay_and_window(k, boundary):
    p, c = _plan(11, 12, 4, 97, 8, boundary)
    window = None if boundary == "stacey" else (13, 88, 3)
    _compare(lambda: [_spec(p, c, 3, "gradient", ckpt_k=k, window=window)])


def test_large_tiles_and_waves():
    # enough solves that tiles grow and several waves run one after another
    p, c = _plan(100, 50, 4, 60, 100, circle=True)
    b = _compare(lambda: [_spec(p, c, 10 + i, "gradient") for i in range(33)])
    assert b.last_groups >= 2


def test_mixed_batch_and_budget():
    ps = [_plan(17, 9, 3, 60, 9, circle=True), _plan(21, 10, 4, 80, 13, circle=True),
          _plan(12, 15, 5, 90, 7, circle=True), _plan(9, 9, 4, 70, 6, "stacey", circle=True)]
    kinds = ["gradient", "forward", "gradient", "likelihood", "gradient"]

    def make():
        return [_spec(*ps[i % 4], i, kinds[i % 5]) for i in range(10)]
    _compare(make)
    one = ps[1][0].workspace_bytes(5 | 8, 8)
    _compare(make, memory_budget=int(1.5 * one))


def test_many_receivers_in_one_tile():
    p, c = _plan(6, 6, 4, 40, 60, circle=True)
    _compare(lambda: [_spec(p, c, 5, "gradient")])


def test_non_finite_velocity_is_reported():
    p, c = _plan(10, 8, 4, 40, 5)
    s = _spec(p, c, 6, "gradient")
    s.velocity = s.velocity.clone()
    s.velocity[17] = float("inf")
    Batch(kernel=5).run([s])
    assert int(s.status.item()) != 0


@pytest.mark.parametrize("npol,nelx,nelz,boundary", [
    (3, 420, 270, "sponge"), (4, 330, 171, "sponge"), (4, 345, 180, "stacey")])
def test_adjoint_tiles_with_fields_in_memory(npol, nelx, nelz, boundary):
    # meshes whose adjoint tiles only fit with the increment and the partial gradient in memory
    p, c = _plan(nelx, nelz, npol, 120, 8, boundary, circle=True)
    b = _compare(lambda: [_spec(p, c, 3, "gradient")])
    assert b.last_kernel == "resident"


@pytest.mark.parametrize("npol,nelx,nelz,models,boundary", [
    (4, 4, 4, 3, "sponge"), (4, 17, 5, 21, "sponge"), (3, 40, 20, 16, "stacey"), (5, 37, 31, 9, "sponge"),
    (2, 9, 33, 40, "sponge"), (7, 8, 8, 5, "stacey")])
def test_solves_as_clusters(npol, nelx, nelz, models, boundary):
    # a solve per thread-block cluster, alone and with more clusters than the GPU holds at once
    p, c = _plan(nelx, nelz, npol, 90, 9, boundary, circle=nelx > 8)
    _compare(lambda: [_spec(p, c, 4, "gradient", ckpt_k=31)])
    _compare(lambda: [_spec(p, c, 5 + i, "gradient" if i % 3 else "likelihood") for i in range(models)])
