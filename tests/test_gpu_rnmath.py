"""Quotients and roots of the FP64 stage (rkb_rnmath.cuh) bit for bit against
IEEE division, square root and the correctly rounded cube root, on random
operands and on the operands whose results lie closest to a rounding
boundary; and whole steps with values outside the range they serve, against
the oracle.
"""
import numpy as np
import pytest

from tests.helpers import compare_state, gaussian_bed, pair

pytestmark = pytest.mark.gpu


def _run(op, a, b):
    import torch
    from rakali_b200 import _lib
    ta, tb = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, b))
    out = torch.zeros_like(ta)
    rc = _lib.load().rkb_test_rn_math(op, ta.data_ptr(), tb.data_ptr(), out.data_ptr(), a.size)
    assert rc == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _random(n, seed, lo=-200, hi=200):
    rng = np.random.default_rng(seed)
    m = rng.integers(1 << 52, 1 << 53, n)
    m[::5] |= (1 << 52) - (1 << 20)  # significands next to 2
    return np.ldexp(m.astype(np.float64), rng.integers(lo, hi, n) - 52) * rng.choice([-1.0, 1.0], n)


def _hard_quotients(seed):
    """a / b within 2^-106 .. 2^-102 of a midpoint: b odd, a 2^k - b (odd) = j."""
    rng = np.random.default_rng(seed)
    a, b = [], []
    for t in range(6000):
        B = (1 << 53) - 3 - 2 * t if t < 2000 else int(rng.integers(1 << 52, 1 << 53)) | 1
        for sh in (53, 54):
            inv = pow(B, -1, 1 << sh)
            for j in (-3, -1, 1, 3):
                N = (-j * inv) % (1 << sh)
                N += (1 << 53) if sh == 53 else 0
                A = (B * N + j) >> sh
                if (1 << 53) <= N < (1 << 54) and (1 << 52) <= A < (1 << 53):
                    a.append(A)
                    b.append(B)
    return np.array(a, dtype=np.float64), np.array(b, dtype=np.float64)


def _hard_roots():
    """x = m^2 + k 2^-106 for the 54-bit m next to sqrt(x), small k = 1 mod 8."""
    out = []
    for k in range(1 - 8 * 300, 8 * 300, 8):
        for sh in (54, 55):
            r = 1
            for n in range(3, sh):  # Hensel: r^2 = k mod 2^sh
                if (r * r - k) % (1 << (n + 1)):
                    r += 1 << (n - 1)
            h = 1 << (sh - 1)
            for s in (r, -r, r + h, h - r):
                for N in {s % (1 << sh), s % (1 << 54)}:
                    if not (1 << 53) <= N < (1 << 54) or (N * N - k) % (1 << sh):
                        continue
                    X = (N * N - k) >> sh
                    if (1 << 52) <= X < (1 << 53):
                        out.append(X * 2.0 ** (-52 if sh == 54 else -51))
    x = np.array(out)
    return np.concatenate([x, np.ldexp(x, 60), np.ldexp(x, -180)])


def test_quotients():
    a, b = _random(200000, 1), np.abs(_random(200000, 2, -60, 60))
    a[::17] = 0.0
    a[::34] = -0.0
    for x, y in ((a, b), _hard_quotients(3)):
        np.testing.assert_array_equal(_run(0, x, y).view(np.int64), (x / y).view(np.int64))
        np.testing.assert_array_equal(_run(1, x, y).view(np.int64), ((y * x) / y).view(np.int64))
        np.testing.assert_array_equal(_run(2, x, y).view(np.int64), (1.0 / y).view(np.int64))


def test_square_roots():
    x = np.concatenate([np.abs(_random(200000, 4)), _hard_roots()])
    np.testing.assert_array_equal(_run(3, x, x).view(np.int64), np.sqrt(x).view(np.int64))


def test_cube_roots():
    from rakali_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(5)
    h = np.concatenate([np.exp(rng.uniform(np.log(1.1e-6), np.log(1e12), 20000)),
                        1.0 + rng.integers(-4000, 4000, 4000) * 2.0 ** -52])
    want = np.array([lib.rkb_cr_pow_third(float(x)) for x in h])
    np.testing.assert_array_equal(_run(4, h, h).view(np.int64), want.view(np.int64))


def _state(kind, shape, rng):
    """(h, hu, hv) of moving water with patches of the given extreme."""
    h = 2.0 + 0.3 * rng.random(shape)
    hu, hv = rng.normal(0, 0.5, shape), rng.normal(0, 0.5, shape)
    spot = rng.random(shape) < 0.02
    n = int(spot.sum())
    if kind == "tiny":  # momenta down to the subnormals
        hu[spot] = 10.0 ** rng.uniform(-322, -60, n)
        hv[spot] = -10.0 ** rng.uniform(-322, -60, n)
    elif kind == "still":  # exact zeros of both signs
        hu[:] = 0.0
        hv[:] = -0.0
    elif kind == "thin":  # depths around the wet/dry and thin-film thresholds
        h[spot] = 10.0 ** rng.uniform(-9, -2, n)
        hu[spot] *= h[spot]
        hv[spot] *= h[spot]
    elif kind == "ones":  # depths whose significand is all ones
        h[spot] = np.nextafter(2.0, 0.0)
        hu[spot] = 0.5
        hv[spot] = 0.25
    elif kind == "fast":  # supercritical, some beyond the Froude backstop
        hu[spot] *= 10.0 ** rng.uniform(1, 4, n)
    elif kind == "huge":  # beyond 2^40
        hu[spot] = 1.0e13
    return tuple(np.asfortranarray(x) for x in (h, hu, hv))


def _same_bits(sim, orc):
    for name in ("h", "hu", "hv"):
        got, want = (np.ascontiguousarray(x).view(np.int64)
                     for x in (getattr(sim, name), orc.arrays[name]))
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("tile", [10, 8])
@pytest.mark.parametrize("hllc", [False, True])
@pytest.mark.parametrize("kind", ["tiny", "still", "thin", "ones", "fast", "huge"])
def test_steps_with_extreme_values(kind, hllc, tile):
    """Two steps on a flat bed (spread of tiny momenta, exact depths) and on a
    sloping one: the same bits as the oracle."""
    nx, ny = 53, 41
    for b in (np.zeros((nx, ny), order="F"),
              gaussian_bed(nx, ny, 10.0, 10.0, 4, seed=8, base=-1.0, amp=(-0.5, 0.6))):
        cfg = dict(nx=nx, ny=ny, dx=10.0, dy=7.0, t_end=1.0e9, cfl=0.45, manning_n=0.03,
                   use_hllc=hllc)
        h, hu, hv = _state(kind, (nx, ny), np.random.default_rng(9))
        sim, orc = pair(cfg, bathymetry=b, initial_h=h)
        with sim:
            sim.set_tile(tile)
            for name, f in (("hu", hu), ("hv", hv)):
                getattr(sim, f"set_{name}")(f)
                orc.interior(name)[:] = f
            sim.step(2)
            orc.step(2)
            assert sim.dt == orc.dt
            compare_state(sim, orc, rtol=0.0)
            _same_bits(sim, orc)


@pytest.mark.parametrize("tile", [10, 8])
@pytest.mark.parametrize("hllc", [False, True])
@pytest.mark.parametrize("kind", ["rest", "hump", "rows", "patches"])
def test_zeros_keep_their_sign(kind, hllc, tile):
    """Momenta that are zeros of both signs, at rest, beside a hump, across a
    one-dimensional flow and between moving cells: the oracle's bit patterns
    (a wall ghost negates, so a lake at rest has zeros of both signs too)."""
    nx, ny = 53, 41
    rng = np.random.default_rng(9)
    h = np.full((nx, ny), 2.0, order="F")
    hu, hv = (rng.choice([0.0, -0.0], (nx, ny)) for _ in range(2))
    if kind == "hump":
        h[20:25, 20:25] = 2.5
        hv[:], hu[:] = 0.0, 0.0
        hv[:, ::2], hu[::2] = -0.0, -0.0
    elif kind == "rows":
        h[:] = 2.0 + 0.3 * rng.random((nx, 1))
        hu[:] = rng.normal(0.0, 0.3, (nx, 1))
    elif kind == "patches":
        h[:] = 2.0 + 0.3 * rng.random((nx, ny))
        moving = rng.random((nx, ny)) < 0.3
        hu[moving] = rng.choice([0.5, -0.5], moving.sum())
        hv[moving] = rng.choice([0.3, -0.3], moving.sum())
    cfg = dict(nx=nx, ny=ny, dx=10.0, dy=7.0, t_end=1.0e9, cfl=0.45, manning_n=0.03, use_hllc=hllc)
    for steps in (1, 3):
        sim, orc = pair(cfg, bathymetry=np.zeros((nx, ny), order="F"), initial_h=h)
        with sim:
            sim.set_tile(tile)
            for name, f in (("hu", hu), ("hv", hv)):
                getattr(sim, f"set_{name}")(np.asfortranarray(f))
                orc.interior(name)[:] = f
            sim.step(steps)
            orc.step(steps)
            _same_bits(sim, orc)
