"""The FP64 step with its transforms as split GEMMs (digit products on the
tensor cores): sizes at the edges of its tiles and of the rule that chooses it,
against the transforms inside the passes, which the parity tests hold to the
oracle; batches that mix the two forms; the solid mask that leaves it; its
failure paths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10  # the FP64 step's bound (test_gpu_parity.py)


@pytest.fixture(scope="module")
def R():
    from rustpde_gb300 import build
    build.build()
    import rustpde_gb300
    return rustpde_gb300


@pytest.fixture(scope="module")
def O():
    from oracle import oracle
    oracle.build()
    return oracle


# (nx, ny, kind): list lengths of 47-64 terms and 16-divisible ones, last tiles
# of 1, 16 and 17 outputs, odd and even lengths on either axis, one and several
# lane blocks, the shortest axis with the longest, a prime Fourier length
SIZES = [(96, 94, 0), (95, 129, 1), (98, 97, 0), (16, 600, 0), (600, 16, 1), (66, 142, 0),
         (96, 96, 2), (101, 98, 2), (97, 95, 2), (16, 576, 2), (640, 20, 2), (128, 71, 2),
         (176, 64, 0), (200, 150, 1), (513, 100, 0), (257, 130, 1)]


def _ic(c):
    c.set_velocity(0.2, 1, 1)
    c.set_temperature(0.2, 1, 2)


@pytest.mark.parametrize("nx,ny,kind", SIZES)
def test_step_matches_transforms_inside_the_passes(R, nx, ny, kind):
    args = (nx, ny, 1e5, 0.7, 2e-3, 1.3, kind)
    g, d = R.Navier2D(*args), R.Navier2D(*args)
    _ic(g)
    _ic(d)
    d.solid = [np.zeros((nx, ny)), np.zeros((nx, ny))]  # damps nothing; its passes hold the transforms
    g.update(3)
    d.update(3)
    for f in (R.TEMP, R.UX, R.UY, R.PRES, R.PSEUDO_PRES):
        a, b = g.get(f), d.get(f)
        err = np.linalg.norm(a - b) / np.linalg.norm(b)
        assert err <= TOL, (f, err)
    assert g.status() == 0 and d.status() == 0


MIX = [(64, 64, 1e5, 1.0, 5e-3, 1.0, 0), (100, 95, 1e5, 1.0, 5e-3, 1.2, 0), (64, 33, 1e5, 0.7, 5e-3, 1.0, 2),
       (130, 111, 1e5, 7.0, 5e-3, 1.5, 2), (129, 129, 1e5, 1.0, 5e-3, 1.0, 1)]


def test_batch_of_both_forms_equals_single_cases(R):
    b = R.Batch(MIX)
    singles = [R.Navier2D(*p) for p in MIX]
    for c, s in zip(b.cases, singles):
        _ic(c)
        _ic(s)
        s.update(3)
    b.update(3)
    b.synchronize()
    for c, s in zip(b.cases, singles):
        for f in (R.TEMP, R.UX, R.UY, R.PRES, R.PSEUDO_PRES):
            np.testing.assert_array_equal(c.get(f), s.get(f))


@pytest.mark.parametrize("kind", [0, 2])
def test_solid_mask_leaves_and_returns(R, O, kind):
    args = (100, 96, 1e5, 1.0, 2e-3, 1.0, kind)
    mask = np.zeros((100, 96))
    mask[30:40, 20:50] = 1.0
    g, o, plain = R.Navier2D(*args), O.Navier2D(*args), R.Navier2D(*args)
    for c in (g, o, plain):
        _ic(c)
    g.solid = [mask, 0.1 * mask]
    o.set_solid(mask, 0.1 * mask)
    g.update(2)
    o.update(2)
    for f in (R.TEMP, R.UX, R.UY):
        assert np.linalg.norm(g.get(f) - o.get(f)) <= TOL * np.linalg.norm(o.get(f)), f
    g.solid = None
    for f in (R.TEMP, R.UX, R.UY, R.PRES, R.PSEUDO_PRES):
        plain.set(f, g.get(f))
    g.update(2)
    plain.update(2)
    for f in (R.TEMP, R.UX, R.UY, R.PRES, R.PSEUDO_PRES):
        np.testing.assert_array_equal(g.get(f), plain.get(f))


@pytest.mark.parametrize("kind", [0, 2])
def test_nonfinite_and_timeout_are_reported(R, kind):
    args = (100, 96, 1e5, 1.0, 2e-3, 1.0, kind)
    g = R.Navier2D(*args)
    _ic(g)
    t = g.get(R.TEMP)
    t[3, 4] = np.inf
    g.set(R.TEMP, t)
    g.update(1)
    assert g.status() & 1
    h = R.Navier2D(*args)
    _ic(h)
    R.set_gemm_wait_limit(0)
    try:
        h.update(1)
        h.synchronize()
        assert h.status() & 2
    finally:
        R.set_gemm_wait_limit(-1)
    k = R.Navier2D(*args)
    _ic(k)
    k.update(1)
    assert k.status() == 0 and np.isfinite(k.get(R.TEMP)).all()


@pytest.mark.parametrize("nx,ny", [(17, 16), (22, 17), (23, 16), (26, 33), (47, 17), (106, 33), (599, 16)])
def test_small_prime_fourier_lengths(R, nx, ny):
    # a Fourier length with a prime factor above 8 takes the digit GEMMs at any
    # size from 16 x 16 on: few rows, short lists, one lane block
    test_step_matches_transforms_inside_the_passes(R, nx, ny, 2)


@pytest.mark.parametrize("limit", [0, 1, 2, 4, 16])
def test_space_that_gives_up_midway(R, limit):
    # waits that run out somewhere along a tile's chunks: an output is the
    # product or NaN, and the next call is as if nothing had happened
    s = R.Space2(R.Base(1, 264), R.Base(1, 265))
    v = np.random.default_rng(8).standard_normal((264, 265))
    spec = s.forward(v)
    ref = s.backward(spec)
    R.set_gemm_wait_limit(limit)
    try:
        got = s.backward(spec)
    finally:
        R.set_gemm_wait_limit(-1)
    assert (np.isnan(got) | (got == ref)).all()
    np.testing.assert_array_equal(s.backward(spec), ref)


@pytest.mark.parametrize("kind", [0, 2])
def test_fp64_step_that_gives_up_does_not_look_well(R, kind):
    # a caller that steps in FP64 and asks for no status sees it in the fields
    c = R.Navier2D(100, 96, 1e5, 1.0, 2e-3, 1.0, kind)
    _ic(c)
    R.set_gemm_wait_limit(0)
    try:
        c.update(1)
        c.synchronize()
    finally:
        R.set_gemm_wait_limit(-1)
    assert c.status() & 2
    for f in (R.TEMP, R.UX, R.UY):
        assert np.isnan(c.get(f)).any()
    assert c.exit()


def _values(n):
    """Chebyshev coefficients -> values, and back, in extended precision."""
    N = n - 1
    j = np.arange(n)
    pi = np.longdouble("3.14159265358979323846264338327950288")
    cos = np.cos(pi * (np.outer(j, j) % (2 * N)).astype(np.longdouble) / N)
    sign = np.where(j % 2, -1, 1).astype(np.longdouble)
    end = np.where((j == 0) | (j == N), 0.5, 1.0).astype(np.longdouble)
    return cos * sign[None, :], cos * (2 / np.longdouble(N) * sign * end)[:, None] * end[None, :]


@pytest.mark.parametrize("n", [49, 130, 263, 640])
def test_digit_products_of_uneven_lanes(R, n):
    # lanes over 300 decades, near both ends of the exponent range, subnormal,
    # with values that differ in their last bit, with the largest digits.  The
    # bound is a dot product's in FP64, n 2^-53 sum |w x|, plus the fixed point of
    # a lane and of the operator against their largest values, n 2^-54 |w| |x|
    lanes = -(-4_000_000 // (n * n))
    rng = np.random.default_rng(n)
    k = np.arange(n)
    x = rng.standard_normal((lanes, n))
    x[1::9] *= 10.0 ** (-300.0 * k / n)
    x[2::9] *= 1e300
    x[3::9] *= 1e-310
    x[4::9] = 1.0 + k * 2.0**-52
    x[5::9] = np.where(k % 2, -1, 1) * (2.0 - 2.0**-52)
    x[6::9] = np.where(k == n // 3, np.pi, 0.0)
    x[7::9] = np.where(rng.integers(0, 2, n), 1, -1) * np.ldexp(float(0x10808080808080), -52)
    x[8::9] *= np.where(k % 2, 1e10, 1e-6)
    L = R.Lanes(R.Base(0, n))
    B, F = _values(n)
    X = x.astype(np.longdouble)
    for op, M in ((R.OP_BACKWARD, B), (R.OP_FORWARD, F)):
        got = L.apply(op, x)
        want = X @ M.T
        bound = n * 2.0**-53 * (np.abs(X) @ np.abs(M).T) + n * 2.0**-54 * np.abs(M).max() * np.abs(X).max(axis=1)[:, None]
        worst = (np.abs(got - want) / (bound + 2.0**-1073)).max(axis=1)
        assert worst.max() <= 1, (op, worst.argmax() % 9, float(worst.max()))
        print(n, op, [float(worst[r::9].max()) for r in range(9)])
    assert L.status() == 0
