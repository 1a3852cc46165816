"""2D solves where the device has no memory left for the diagonal walk's scratch
(its model planes and field copies): the walk in place, which needs none, gives
the same times, for one source and for many in a call, and the solver's later
allocations still find room."""
import numpy as np
import pytest

from test_gpu_solver2d_diag import _model, _oracle

pytestmark = pytest.mark.gpu

H = 10.0


@pytest.fixture
def fill(fk):
    """fill(left): a tensor over the free device memory but `left` bytes."""
    import torch
    held = []

    def take(left):
        torch.cuda.synchronize()
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda"))
    yield take
    held.clear()
    torch.cuda.empty_cache()


def _solver(fk, nz, nx, vel, zs, xs):
    s = fk.fteik2d()
    s.initialize(nx, nz, H, H, nsweep=1, eps=5.0)
    s.setCellVelocityNatural(vel)
    s.setSources(xs, zs)
    return s


def _first_call(fk):
    """The library's stream, buffers and kernels, before memory gets short."""
    s = _solver(fk, 20, 600, _model(20, 600, 1), [50.0], [300.0])
    s.solveSourceLSM(1)
    s.free()


def test_one_source(fk, fill):
    nz, nx = 4000, 500                    # 369 MB of model planes, 37 MB of field copies
    vel, src = _model(nz, nx, 3), (21000.0, 2300.0)
    want = _oracle(nz, nx, (H, H), vel, src, 5.0, 1)
    _first_call(fk)
    fill(192 << 20)
    s = _solver(fk, nz, nx, vel, [src[0]], [src[1]])
    s.solveSourceLSM(1)
    assert np.max(np.abs(s.getTravelTimeField() - want)) <= 1e-12 * np.max(want)
    s.free()


def test_many_sources_then_a_gradient(fk, fill):
    nz, nx, ns = 500, 500, 300            # 82 MB of model planes, 8 MB of field copies a source
    vel = _model(nz, nx, 4)
    rng = np.random.default_rng(5)
    zs, xs = rng.uniform(0, (nz - 1) * H, ns), rng.uniform(0, (nx - 1) * H, ns)
    _first_call(fk)
    fill(1600 << 20)                      # 600 MB of them for the sources' fields
    s = _solver(fk, nz, nx, vel, zs, xs)
    s.setReceivers(np.linspace(0, (nx - 1) * H, 9), np.zeros(9))
    s.solveLSM()
    want = _oracle(nz, nx, (H, H), vel, (zs[-1], xs[-1]), 5.0, 1)
    assert np.max(np.abs(s.getTravelTimeField() - want)) <= 1e-12 * np.max(want)
    few = s.getTravelTimes()
    s.getTravelTimeGradient()
    s.free()
    import torch
    torch.cuda.empty_cache()
    assert np.isfinite(few).all() and few.shape[0] == ns


@pytest.mark.parametrize("nz,nx,eps,nsweep", [(200, 300, 5.0, 2), (401, 210, 9.0, 1), (150, 512, 0.0, 3)])
def test_both_walks_give_the_same_bits(fk, fill, nz, nx, eps, nsweep):
    vel = _model(nz, nx, nz + nx)
    s = fk.fteik2d()
    s.initialize(nx, nz, 7.5, H, nsweep=nsweep, eps=eps)
    s.setCellVelocityNatural(vel)
    s.setSources([0.31 * (nx - 1) * 7.5], [0.63 * (nz - 1) * H])
    s.solveSourceLSM(1)
    want = s.getTravelTimeField()
    s.free()
    _first_call(fk)
    fill(24 << 20)                        # the model planes alone take 21 MB or more
    s.initialize(nx, nz, 7.5, H, nsweep=nsweep, eps=eps)
    s.setCellVelocityNatural(vel)
    s.setSources([0.31 * (nx - 1) * 7.5], [0.63 * (nz - 1) * H])
    s.solveSourceLSM(1)
    assert np.array_equal(s.getTravelTimeField(), want)
    s.free()
