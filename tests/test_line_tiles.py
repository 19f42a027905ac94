"""The bit-exact line sweeps: ragged, short and long lines around the tiles' and
tasks' edges, the quotients from reciprocals against the divide, the fallback
to the divide, and the rings beside the tiles."""
import math
import random
from fractions import Fraction

import numpy as np
import pytest

import mts_b200 as M
import oracle as O
from mts_b200 import workloads


def _fma(a, b, c):
    # the correctly rounded a*b + c (int / int and Fraction to float round to nearest)
    if not all(map(math.isfinite, (a, b, c))):
        return a * b + c
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


def _oracle(spec, u, steps):
    tags, cr, _ = M.setup_host(spec)
    p = O.Problem(n=spec.n, surface=spec.surface, surface_params=spec.surface_params, beta_in=spec.beta_in,
                  beta_out=spec.beta_out, eq=spec.eq, method=spec.method, mib=spec.mib, dt=spec.dt, t0=spec.t0)
    u = O.port_init(p, tags) if u is None else u
    return u, O.port_run(p, tags, cr, u, steps=steps)


def _same(got, want):
    """Bit for bit, the signs of zeros included (any NaN equals any NaN)."""
    return np.array_equal(got, want, equal_nan=True) and np.array_equal(
        np.signbit(got) & ~np.isnan(got), np.signbit(want) & ~np.isnan(want))


def _check(spec, u, steps):
    u, want = _oracle(spec, u, steps)
    with M.Solver(spec) as s:
        s.set_solution(u)
        s.advance(steps)
        assert _same(s.solution(), want)


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
def test_fields_of_zeros_and_of_tiny_and_huge_values(method, value):
    """Every third node set, the others zero.  1e290 has quotients past 2^800,
    which take the divide (and which the reciprocals would give as well)."""
    spec = M.Spec(n=(33, 25, 37), method=method, mib=1, dt=0.05, **ELL)
    u = np.zeros(spec.nodes)
    u[:: 3] = value
    _check(spec, u, 2)


LATE = 800.0  # exp(-t) is 0 from about t = 745 on: no boundary data, source or jumps


def _hard_field(kind, nodes):
    """Fields of quotients out of range: "subnormal" (and next to it), where
    the reciprocals round otherwise than the divide; zeros of the other sign
    and infinities, where they give another zero, or NaN."""
    if kind == "subnormal":
        return np.random.default_rng(5).uniform(1.0, 2.0, nodes) * 1e-307
    u = np.full(nodes, -0.0)
    if kind == "infinite":
        u[nodes // 2 + 7] = np.inf
        u[nodes // 3] = -np.inf
    return u


def _line(r, c, quotient):
    """(1 + 2c) u_j - c (u_{j-1} + u_{j+1}) = r_j between zero ends, as the
    sweeps solve it."""
    n = len(r)
    bet, gam = [1.0], [0.0]
    for j in range(1, n):
        end = j == n - 1
        gam.append((0.0 if j == 1 else -c) / bet[-1])
        bet.append((1.0 if end else 1.0 + 2.0 * c) - (0.0 if end else -c) * gam[-1])
    d = [quotient(r[0], 1.0)]
    for j in range(1, n):
        d.append(quotient(r[j] - (0.0 if j == n - 1 else -c) * d[-1], bet[j]))
    for j in range(n - 2, -1, -1):
        d[j] -= gam[j + 1] * d[j + 1]
    return d


def test_subnormal_fields_need_the_divide():
    """What the tests below rest on: lines of such a field solved with the
    quotients from reciprocals differ from the divide's."""
    field = _hard_field("subnormal", 100 * 33).reshape(100, 33)
    wrong = 0
    for r in field:
        r = [0.0, *map(float, r[1:-1]), 0.0]
        wrong += _line(r, 12.8, _quotient) != _line(r, 12.8, lambda n, b: n / b)
    assert wrong >= 10, wrong
    assert _quotient(-0.0, 3.0) == 0.0 and math.copysign(1.0, _quotient(-0.0, 3.0)) == 1.0
    assert math.isnan(_quotient(math.inf, 3.0))


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-ie", "lod-cn", "ts"])
@pytest.mark.parametrize("kind", ["subnormal", "negative zero", "infinite"])
def test_quotients_out_of_range_take_the_divide(method, kind):
    if method == "ts" and kind == "infinite":
        pytest.skip("the oracle writes the z faces after TS's z sweep, the sweep keeps 0 * NaN there")
    spec = M.Spec(n=(33, 25, 37), method=method, mib=1, dt=0.05, t0=LATE, **ELL)
    _check(spec, _hard_field(kind, spec.nodes), 2)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-ie", "lod-cn", "ts"])
def test_batched_quotients_out_of_range_take_the_divide(method):
    """The same in one batch, with a problem whose factors pass 2^100, one
    with long lines and an ordinary one."""
    ok = dict(method=method, mib=1, **ELL)
    specs = [M.Spec(n=(33, 25, 37), dt=0.05, t0=LATE, **ok) for _ in range(3)]
    kinds = ("subnormal", "negative zero", "subnormal" if method == "ts" else "infinite")
    fields = [_hard_field(k, specs[0].nodes) for k in kinds]
    specs += [M.Spec(n=(25, 25, 25), dt=1e32, **ok), M.Spec(n=(17, 18, 300), dt=0.05, t0=LATE, **ok),
              M.Spec(n=(25, 33, 17), dt=0.05, **ok)]
    fields += [None, _hard_field("subnormal", specs[4].nodes), None]
    pairs = [_oracle(sp, u, 2) for sp, u in zip(specs, fields)]
    solvers = [M.Solver(sp) for sp in specs]
    try:
        for s, (u, _) in zip(solvers, pairs):
            s.set_solution(u)
        M.batch_advance(solvers, 2)
        for s, (_, want) in zip(solvers, pairs):
            assert _same(s.solution(), want), s.spec
    finally:
        for s in solvers:
            s.close()


@pytest.mark.gpu
def test_factors_past_2_100():
    """A time step so long that the factors pass 2^100, where the quotients
    from reciprocals are not relied on."""
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
        assert many <= workloads.device_bytes_bound(spec, sum(s.counts()["crossings"]))
        s.autotune(1)
        assert s.device_bytes() <= many + 16 * 3 * spec.nodes * 2  # what the kept shapes do not use is given back
    with M.Solver(M.Spec(n=(33, 33, 33), method=method)) as s:
        s.initialize()
        assert not _ring_default(s)
        held = s.device_bytes()
        shapes = s.autotune(1)
        assert max(shapes) >= 10 or s.device_bytes() == held
    _check(spec, None, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "ts"])
def test_a_problem_on_rings_steps_by_itself_in_a_batch(method):
    specs = [M.Spec(n=(389, 18, 397), method=method, mib=1, beta_out=37.5, dt=0.01, setup="device", **ELL),
             M.Spec(n=(25, 33, 17), method=method, mib=2, dt=0.05, **ELL)]
    solvers = [M.Solver(sp) for sp in specs]
    try:
        for s in solvers:
            s.initialize()
        held = solvers[0].device_bytes()
        M.batch_advance_steps(solvers, [2, 3])
        assert solvers[0].device_bytes() > held
        for sp, s, k in zip(specs, solvers, (2, 3)):
            _, want = _oracle(sp, None, k)
            assert _same(s.solution(), want)
    finally:
        for s in solvers:
            s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["adi", "lod-cn", "ts"])
def test_a_captured_step_without_ring_data_takes_the_tiles(method):
    """Ring shapes whose data is not there and cannot be allocated (the stream
    is being captured): the tiles take the sweeps, with the same bits; the next
    step outside builds the data and takes the rings."""
    import torch

    spec = M.Spec(n=(45, 38, 51), method=method, mib=2, beta_out=37.5, dt=0.03, **ELL)
    u, want = _oracle(spec, None, 1)
    with M.Solver(spec) as s:
        for k in range(3):
            s.set_sweep_shape(k, 10 + k)
        s.set_solution(u)
        s.synchronize()
        held = s.device_bytes()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(s.stream()), capture_error_mode="relaxed"):
            s.advance(1)
        assert s.device_bytes() == held
        graph.replay()
        torch.cuda.synchronize()
        assert _same(s.solution(), want)
        s.time = spec.t0
        s.set_solution(u)
        s.advance(1)
        assert s.device_bytes() > held
        assert _same(s.solution(), want)
