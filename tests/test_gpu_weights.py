"""The B-spline weights of the fused deposit, bit for bit: the exact total of lone particles (one per 4x4-pencil
block and z plane, so every contribution is the float32 product of its weights, rounded at 2^-29) against the same
float32 operations on the host, fused multiply-adds included.  Equal for every tile shape, whatever the compiler
makes of an instance."""
from fractions import Fraction

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F = np.float32


def _round(q):
    """Fraction -> nearest float32, ties to even (normal range)."""
    f = F(float(q))
    best = min((np.nextafter(f, F(-9)), f, np.nextafter(f, F(9))),
               key=lambda v: (abs(Fraction(float(v)) - q), int(v.view(np.int32)) & 1))
    return best


def _fma(a, b, c):
    return _round(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)))


def _weights(d, mas):
    """Node weights at offset d in [0, 1) from the lower node."""
    if mas == 3:
        s = F(d - F(1)) if d >= F(0.5) else d
        l, r = F(F(0.5) - s), F(F(0.5) + s)
        return [F(F(F(0.5) * l) * l), _fma(-s, s, F(0.75)), F(F(F(0.5) * r) * r)]
    c6 = F(F(1) / F(6))
    t, m = d, F(F(1) - d)
    cube = lambda v: F(F(F(v * v) * v) * c6)
    inner = lambda v: F(_fma(F(F(F(3) * v) * v), v, _fma(F(F(-6) * v), v, F(4))) * c6)
    return [cube(m), inner(t), inner(m), cube(t)]


def _total(u, mas, half):
    """Sum over particles and nodes of the contributions in units of 2^-29."""
    total = 0
    for p in u:
        w = []
        for v in p:
            d = F(v - np.floor(v))
            if half:
                d = F(d + F(0.5))
                d = F(d - F(1)) if d >= F(1) else d
            w.append(_weights(d, mas))
        for a in w[0]:
            for b in w[1]:
                for c in w[2]:
                    total += int(np.rint(float(F(F(a * b) * c)) * 2.0 ** 29))
    return total


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("mas", [3, 4])
@pytest.mark.parametrize("interlace", [False, True])
def test_lone_particles_have_the_host_weights(N, mas, interlace):
    from gbpowspec import PkConfig, PowerSpectrum, _native, read_stats
    rng = np.random.default_rng(N + mas)
    i = np.arange(0, 64, 8)
    cell = np.stack(np.meshgrid(i, i, indexing="ij"), -1).reshape(-1, 2)
    u = np.column_stack([cell, rng.integers(0, N, len(cell))]) + rng.random((len(cell), 3))
    u = np.minimum(u.astype(F), F(N) - F(0.01))
    x, y, z = (torch.from_numpy(np.ascontiguousarray(u[:, a])).cuda() for a in range(3))
    want = [_total(u, mas, g) * 2.0 ** -29 for g in range(1 + interlace)]
    for tiles in _native.tile_variants(N):
        r = PowerSpectrum(PkConfig(n_mesh=N, box_size=float(N), mas={3: "tsc", 4: "pcs"}[mas], interlace=interlace),
                          tiles=tiles).run(x, y, z)
        torch.cuda.synchronize()
        assert list(read_stats(r.stats).mass[: len(want)]) == want, tiles
