"""The adjoint at the edges of its kernels: walls in memory and in the tiles at
two to four ghost layers and on grids narrower than twice that, tiles with one
row or column, faces next to dry islands, against torch.autograd through the
plain FP64 transcription (tests/torch_step.py).  1e-8 relative, as for the
larger grids: the sums differ in order and the reciprocals by half an ulp.
"""
import numpy as np
import pytest

from rakali_b200.adjoint import GaugeMisfit
from tests.helpers import gaussian_bed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ng", [(4, 9, 4), (5, 4, 3), (17, 16, 2), (33, 31, 3), (48, 15, 2)])
@pytest.mark.parametrize("hllc", [False, True])
def test_gradient(nx, ny, ng, hllc):
    import torch

    from tests import torch_step as ts
    steps, dx = 6, 10.0
    rng = np.random.default_rng(nx + 100 * ny)
    b = gaussian_bed(nx, ny, dx, dx, 4, seed=nx, base=-2.0, amp=(-1.0, 1.0), width=(20.0, 60.0))
    if nx > 16:  # an island
        b = b + 3.0 * gaussian_bed(nx, ny, dx, dx, 1, seed=ny, base=0.0, amp=(1.0, 1.0),
                                   width=(15.0, 20.0))
    h = np.asfortranarray(np.maximum(0.1 * rng.random((nx, ny)) - b, 0.0))
    hu, hv = (np.asfortranarray(rng.normal(0.0, 0.2, (nx, ny)) * h) for _ in range(2))
    n = np.asfortranarray(0.02 + 0.01 * rng.random((nx, ny)))
    cells = rng.choice(nx * ny, size=5, replace=False)
    gauges = [(int(c % nx), int(c // nx)) for c in cells]
    p = GaugeMisfit(nx, ny, dx, dx, h, gauges, steps, hu0=hu, hv0=hv, nghost=ng, use_hllc=hllc)
    p.record_dt(b, n)
    obs = p.forward(b + 0.05 * rng.random((nx, ny)), n)[1]
    p.set_observations(obs)
    J, gb, gn = p.gradient(b, n)
    t = [torch.tensor(x, dtype=torch.float64, requires_grad=True) for x in (b, n)]
    Jt = ts.misfit(*t, *(torch.from_numpy(x) for x in (h, hu, hv)), gauges, torch.from_numpy(obs),
                   list(p.dt), ng, dx, dx, hllc=hllc)
    Jt.backward()
    assert abs(Jt.item() - J) <= 1e-10 * abs(J)
    for got, want in zip((gb, gn), t):
        want = want.grad.numpy()
        assert np.abs(got - want).max() <= 1e-8 * np.abs(want).max()
    p.close()


@pytest.mark.parametrize("precision", [64, 32])
def test_memory_order_of_the_fields_does_not_matter(precision):
    """b and n in every order of axes, strided and reversed views: the same bits."""
    from rakali_b200.adjoint import GaugeMisfitBatch
    nm, nx, ny = 3, 21, 18
    rng = np.random.default_rng(4)
    b = -2.0 + 0.3 * rng.random((nm, nx, ny))
    n = 0.02 + 0.01 * rng.random((nm, nx, ny))
    p = GaugeMisfitBatch(nm, nx, ny, 10.0, 10.0, 0.1 * rng.random((nm, nx, ny)) - b,
                         [[(3, 4), (9, 11)]] * nm, 5, precision=precision)
    p.record_dt(b, n)
    want = p.gradient(b, n)
    wide = np.zeros((nm, nx, 2 * ny))
    wide[:, :, ::2] = b
    flipped = np.ascontiguousarray(b[::-1])[::-1]
    for bv in (np.asfortranarray(b), np.ascontiguousarray(b.transpose(0, 2, 1)).transpose(0, 2, 1),
               np.ascontiguousarray(b.transpose(1, 0, 2)).transpose(1, 0, 2), wide[:, :, ::2], flipped):
        got = p.gradient(bv, np.asfortranarray(n))
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y)
        assert got[1].shape == (nm, nx, ny)
    p.close()


def test_initial_state_is_taken_by_the_constructor():
    """Page-locked initial fields overwritten as soon as the constructor has
    returned: the run starts from what they held (dt shows every cell's state)."""
    import torch
    nx, ny, steps = 1024, 768, 2  # the copies queue behind the clearing of 0.6 GB
    rng = np.random.default_rng(3)
    b = np.full((nx, ny), -2.0, order="F")
    fields = [2.0 + 0.1 * rng.random((nx, ny)), rng.normal(0.0, 0.2, (nx, ny)),
              rng.normal(0.0, 0.2, (nx, ny))]
    pinned = [torch.from_numpy(np.ascontiguousarray(x.T)).pin_memory() for x in fields]
    views = [t.numpy().T for t in pinned]  # Fortran order: passed on without a copy
    runs = []
    for h, hu, hv in (fields, views):
        with GaugeMisfit(nx, ny, 10.0, 10.0, h, [(5, 6), (500, 700)], steps, hu0=hu, hv0=hv) as p:
            for t in reversed(pinned if h is views[0] else []):
                t.fill_(9.0)
            J, eta = p.record_dt(b, 0.02)
            runs.append((J, eta, p.dt, *p.gradient(b, 0.02)))
    for x, y in zip(*runs):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("ny", [393206, 393207, 400001])
def test_gradient_of_more_rows_than_one_launch_gathers(ny):
    """65535 blocks of six rows gather the ny + 4 rows up to ny = 393206, beyond
    it a second launch the rest.  Gauges next to both ends: the gradients there
    are those of the first and of the last 60 rows alone, and zero between."""
    from rakali_b200.adjoint import GaugeMisfitBatch
    nx, m, half = 4, 60, 30  # two steps carry a gauge's gradient 8 rows
    rng = np.random.default_rng(ny)
    b = -2.0 + 0.2 * rng.random((1, nx, ny))
    h, hu = 2.0 + 0.1 * rng.random((1, nx, ny)), rng.normal(0.0, 0.3, (1, nx, ny))

    def gradients(rows, gauges):
        bp, hp, hup = (np.ascontiguousarray(x[:, :, rows]) for x in (b, h, hu))
        with GaugeMisfitBatch(1, nx, bp.shape[2], 10.0, 10.0, hp, [gauges], 2, precision=32,
                              hu0=hup) as p:
            p.set_dt(np.full((1, 2), 0.5))
            return p.gradient(bp, 0.02)[1:]

    full = gradients(slice(None), [(1, 3), (2, ny - 4)])
    low = gradients(slice(0, m), [(1, 3)])
    high = gradients(slice(ny - m, ny), [(2, m - 4)])
    for x, lo, hi in zip(full, low, high):
        assert lo.any() and hi.any()
        np.testing.assert_array_equal(x[:, :, :half], lo[:, :, :half])
        np.testing.assert_array_equal(x[:, :, -half:], hi[:, :, -half:])
        assert not x[:, :, half:-half].any()


@pytest.mark.parametrize("precision", [64, 32])
def test_fields_in_any_order_take_no_device_memory_of_their_own(precision):
    """Members that interleave in memory (Fortran order) go through the
    problem's own arrays: the calls leave the free device memory as it was."""
    import torch

    from rakali_b200.adjoint import GaugeMisfitBatch

    def problem(nm, nx, ny):
        rng = np.random.default_rng(nx)
        b = np.asfortranarray(-2.0 + 0.3 * rng.random((nm, nx, ny)))
        n = np.asfortranarray(0.02 + 0.01 * rng.random((nm, nx, ny)))
        return b, n, GaugeMisfitBatch(nm, nx, ny, 10.0, 10.0, 0.1 * rng.random(b.shape) - b,
                                      [[(3, 4), (9, 11)]] * nm, 2, precision=precision)

    b, n, p = problem(2, 20, 18)  # the library's kernels are loaded by their first use
    p.record_dt(b, n)
    p.gradient(b, n)
    p.close()
    b, n, p = problem(10, 1024, 1024)  # 84 MB a field on the host
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    p.record_dt(b, n)
    p.gradient(b, n)
    p.forward(np.ascontiguousarray(b), n)
    assert free - torch.cuda.mem_get_info()[0] < 8 << 20  # the observations take a page
    p.close()
