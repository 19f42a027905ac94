"""The bit-exact line sweeps' tiles: ragged and short lines around the tiles'
and tasks' edges, the quotients from reciprocals against the divide, and the
fallback to the divide."""
import random
from fractions import Fraction

import numpy as np
import pytest

import mts_b200 as M
import oracle as O


def _fma(a, b, c):
    # the correctly rounded a*b + c (int / int and Fraction to float round to nearest)
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _quotient(n, b):
    """The kernels' quotient (forward_rows), operation by operation."""
    y = 1.0 / b
    yl = y * _fma(-b, y, 1.0)
    q0 = _fma(n, y, n * yl)
    return _fma(_fma(-b, q0, n), y, q0)


def test_quotient_from_reciprocal_is_the_divide():
    rng = random.Random(7)
    pairs = []
    for _ in range(4000):
        n = rng.choice((-1, 1)) * rng.uniform(1, 2) * 2.0 ** rng.randrange(-700, 700)
        pairs.append((n, rng.choice((-1, 1)) * rng.uniform(1, 2) * 2.0 ** rng.randrange(-100, 100)))
    # numerators whose quotient lies next to a midpoint of two doubles:
    # A 2^54 = +-c (mod B) for the divisor's odd significand B
    for _ in range(1500):
        B = rng.randrange(2**52 + 1, 2**53, 2)
        for c in (1, -1, 3, -3):
            A = c * pow(2**54, -1, B) % B
            if A >= 2**52:
                pairs.append((float(A), float(B)))
    # significands next to 1 and 2
    for i in range(40):
        for k in range(40):
            pairs.append((2.0 - (i + 1) * 2.0**-52, 2.0 - (k + 1) * 2.0**-52))
            pairs.append((1.0 + i * 2.0**-52, 1.0 + k * 2.0**-52))
            pairs.append((2.0 - (i + 1) * 2.0**-52, 1.0 + k * 2.0**-52))
    for n, b in pairs:
        assert _quotient(n, b) == n / b, (n.hex(), b.hex())


def _check(spec, u, steps):
    tags, cr, _ = M.setup_host(spec)
    p = O.Problem(n=spec.n, surface=spec.surface, surface_params=spec.surface_params, beta_in=spec.beta_in,
                  beta_out=spec.beta_out, eq=spec.eq, method=spec.method, mib=spec.mib, dt=spec.dt, t0=spec.t0)
    u = O.port_init(p, tags) if u is None else u
    want = O.port_run(p, tags, cr, u, steps=steps)
    with M.Solver(spec) as s:
        s.set_solution(u)
        s.advance(steps)
        assert np.array_equal(s.solution(), want, equal_nan=True)


ELL = dict(surface="ellipsoid", surface_params=(0.6123, 0.4517, 0.3739, 1.0, 0.0713, -0.1127, 0.0391))


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-ie", "lod-cn", "ts"])
@pytest.mark.parametrize("n", [(17, 34, 35), (36, 33, 19), (40, 129, 23), (193, 18, 20), (20, 21, 260)])
def test_ragged_tiles_give_the_oracle_bits(method, n):
    _check(M.Spec(n=n, method=method, mib=2, beta_out=37.5, dt=0.05, **ELL), None, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-cn", "ts"])
def test_lines_shorter_than_a_task_give_the_oracle_bits(method):
    """Grids of a few nodes, without an interface inside."""
    spec = M.Spec(n=(5, 4, 6), method=method, surface="ellipsoid", surface_params=(1, 1, 1, 0.01, 0.03, 0.02, 0.01),
                  dt=0.1)
    _check(spec, None, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-ie", "ts"])
@pytest.mark.parametrize("value", [0.0, 1e-290, 1e290])
def test_quotients_out_of_range_take_the_divide(method, value):
    """Fields whose quotients are zero, tiny or huge: whole tiles are solved
    with the divide, and give its bits."""
    spec = M.Spec(n=(33, 25, 37), method=method, mib=1, dt=0.05, **ELL)
    u = np.zeros(spec.nodes)
    u[:: 3] = value
    _check(spec, u, 2)


@pytest.mark.gpu
def test_factors_out_of_range_take_the_divide():
    """A time step so long that the factors pass 2^100."""
    spec = M.Spec(n=(25, 25, 25), method="lod-ie", mib=1, dt=1e32, t0=0.0, **ELL)
    _check(spec, None, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-cn", "ts"])
@pytest.mark.parametrize("n", [(1455, 17, 18), (17, 1455, 18), (18, 17, 815)])
def test_a_sweep_takes_its_shape_by_its_own_axis(method, n):
    """Grids with one long axis: the sweeps along the short ones take every
    shape, the one along the long axis those whose tiles hold its lines."""
    spec = M.Spec(n=n, method=method, mib=2, beta_out=37.5, dt=0.02, **ELL)
    _check(spec, None, 2)
    lines = (32, 32, 32, 16, 8, 16, 8, 16, 4, 4)  # of each shape's tile

    def fits(d, shape):  # the tile's rows (x tiles padded by one) and a side's factors
        return n[d] * (8 * (lines[shape] + (d == 0)) + 24) <= 226 * 1024

    with M.Solver(spec) as s:
        dirs = (2, 1, 0) if method == "ts" else (0, 1, 2)
        for sweep, d in enumerate(dirs):
            for shape in range(len(lines)):
                if fits(d, shape):
                    s.set_sweep_shape(sweep, shape)
                else:
                    with pytest.raises(M.MtsError, match="shared memory"):
                        s.set_sweep_shape(sweep, shape)
        assert all(fits(d, shape) for d, shape in zip(dirs, s.autotune(1)))


def _ring_default(s):
    """Whether the default shapes name a ring: its data comes with the first
    plain step."""
    before = s.device_bytes()
    s.advance(1)
    return s.device_bytes() > before


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-ie", "lod-cn", "ts"])
def test_rings_beside_tiles_give_the_oracle_bits(method):
    """Each sweep on a ring of staged rows, the others on tiles: the first,
    the second, the third; then all three."""
    n = (45, 38, 51)
    spec = M.Spec(n=n, method=method, mib=2, beta_out=37.5, dt=0.03, **ELL)
    tags, cr, _ = M.setup_host(spec)
    p = O.Problem(n=n, surface=spec.surface, surface_params=spec.surface_params, beta_in=spec.beta_in,
                  beta_out=spec.beta_out, method=method, mib=2, dt=spec.dt)
    u = O.port_init(p, tags)
    want = O.port_run(p, tags, cr, u, steps=2)
    for rings in ((0,), (1,), (2,), (0, 1, 2)):
        for ring in (10, 11, 12):
            with M.Solver(spec) as s:
                for k in rings:
                    s.set_sweep_shape(k, ring)
                s.set_solution(u)
                s.advance(2)
                assert np.array_equal(s.solution(), want), (rings, ring)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-ie", "lod-cn", "ts"])
def test_grids_of_very_many_lines_take_rings_and_give_the_oracle_bits(method):
    """389 x 18 x 397: 1043 y lines an SM on a B200, on rings by default."""
    spec = M.Spec(n=(389, 18, 397), method=method, mib=1, beta_out=37.5, dt=0.01, setup="device", **ELL)
    with M.Solver(spec) as s:
        s.initialize()
        assert _ring_default(s)
        many = s.device_bytes()
        s.autotune(1)
        assert s.device_bytes() <= many + 16 * 3 * spec.nodes * 2  # what the kept shapes do not use is given back
    with M.Solver(M.Spec(n=(33, 33, 33), method=method)) as s:
        s.initialize()
        assert not _ring_default(s)
        held = s.device_bytes()
        shapes = s.autotune(1)
        assert max(shapes) >= 10 or s.device_bytes() == held
    _check(spec, None, 2)
