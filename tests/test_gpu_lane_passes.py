"""The single-axis passes on real lanes: one lane per CTA below 608 lanes, pairs
of lanes from there on (an odd last lane alone), and the dense Chebyshev
transform on its parity tables (odd and even lengths; the centre node).  Held
to the oracle at the FP64 lanes' bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12  # FP64 lanes against the oracle (test_gpu_lanes.py)


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


@pytest.mark.parametrize("lanes", [1, 607, 608, 609])
@pytest.mark.parametrize("kind,n", [(1, 8), (2, 15), (1, 17), (2, 46), (1, 263)])
def test_lanes_and_pairs_match_oracle(R, O, kind, n, lanes):
    rng = np.random.default_rng(100 * n + lanes)
    L = R.Lanes(R.Base(kind, n), R.PREC_FP64, hholtz_c=5e-4)
    phys = rng.standard_normal((lanes, n))
    spec = rng.standard_normal((lanes, L.m)) * np.exp(-np.arange(L.m) / 20.0)
    for op in (R.OP_FORWARD, R.OP_BACKWARD, R.OP_TO_ORTHO, R.OP_FROM_ORTHO, R.OP_HHOLTZ):
        x = spec if op in (R.OP_BACKWARD, R.OP_TO_ORTHO) else phys
        want = O.lanes_apply(kind, n, op, x, c=5e-4)
        got = L.apply(op, x)
        err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() <= TOL, (op, err.argmax(), err.max())


@pytest.mark.parametrize("k0,n0,k1,n1", [(1, 264, 2, 265), (2, 50, 1, 640), (1, 640, 1, 48), (0, 178, 1, 163),
                                         (5, 301, 2, 190), (1, 257, 0, 250)])
def test_space_transforms_match_oracle(R, O, k0, n0, k1, n1):
    """2-D transforms whose dense axes run as split GEMMs (either axis alone, both, a last tile of 1)."""
    s, o = R.Space2(R.Base(k0, n0), R.Base(k1, n1)), O.Space2(k0, n0, k1, n1)
    rng = np.random.default_rng(n0 + n1)
    v = rng.standard_normal((n0, n1))
    want = o.forward(v)
    got = s.forward(v)
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)
    back, ref = s.backward(want), o.backward(want)
    assert np.linalg.norm(back - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("n0,n1", [(257, 256), (178, 201)])
def test_poisson_with_split_eigenbasis_matches_oracle(R, O, n0, n1):
    """The eigenbasis products themselves are held to the dense ones at 1e-10 by
    the boxes of test_gpu_split.py.  Against the oracle the library's own
    eigensolver counts, which on Dirichlet bases of this length is 8e-9 from
    64-bit dense algebra: 4x that."""
    s, o = R.Space2(R.Base(1, n0), R.Base(1, n1)), O.Space2(1, n0, 1, n1)
    rng = np.random.default_rng(n0)
    rhs = rng.standard_normal((n0, n1)) * np.exp(-8.0 * np.add.outer(np.arange(n0) / n0, np.arange(n1) / n1))
    got = R.Poisson(s, (1.0, 0.8)).solve(rhs)
    want = O.Solver(o, O.POISSON, (1.0, 0.8)).solve(rhs)
    assert np.linalg.norm(got - want) <= 3.2e-8 * np.linalg.norm(want)


def test_lanes_on_two_streams_share_the_scratch_in_order(R):
    torch = pytest.importorskip("torch")
    n, lanes = 130, 5000  # two scratch-sized parts
    L = R.Lanes(R.Base(1, n))
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((2, lanes, n))
    ref = [L.apply(R.OP_FORWARD, x) for x in (a, b)]
    st = [torch.cuda.Stream(), torch.cuda.Stream()]
    ins = [R.DeviceArray.from_host(x) for x in (a, b)]
    outs = [R.DeviceArray((lanes, L.m)) for _ in range(2)]
    for _ in range(4):
        for k in range(2):
            L.apply_dev(R.OP_FORWARD, ins[k], outs[k], lanes, st[k].cuda_stream)
    torch.cuda.synchronize()
    for k in range(2):
        np.testing.assert_array_equal(outs[k].to_host(), ref[k])
    assert L.status() == 0


def test_captured_lanes_replay(R):
    torch = pytest.importorskip("torch")
    n, lanes = 130, 1000
    L = R.Lanes(R.Base(1, n))
    x = np.random.default_rng(4).standard_normal((lanes, n))
    ref = L.apply(R.OP_FORWARD, x)
    d_in, d_out = R.DeviceArray.from_host(x), R.DeviceArray((lanes, L.m))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        L.apply_dev(R.OP_FORWARD, d_in, d_out, lanes, torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    got = d_out.to_host()  # the pass without scratch: another rounding
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)


def test_space_timeout_leaves_nan(R):
    s = R.Space2(R.Base(1, 264), R.Base(1, 265))
    v = np.random.default_rng(5).standard_normal((264, 265))
    ref = s.forward(v)
    R.set_gemm_wait_limit(0)
    try:
        assert np.isnan(s.forward(v)).all()
    finally:
        R.set_gemm_wait_limit(-1)
    np.testing.assert_array_equal(s.forward(v), ref)


@pytest.mark.parametrize("n", [95, 96, 97, 130, 511, 512])
def test_mixed_lanes_in_one_call_equal_parts(R, n):
    # from 1024 lanes and n = 96 the input is packed first (in parts of the
    # scratch's 4096 lanes); the calls of 1000 lanes are not: the same products
    # in the same order, so the same bits
    L = R.Lanes(R.Base(1, n), R.PREC_MIXED, hholtz_c=5e-4)
    rng = np.random.default_rng(n)
    for lanes in (1024, 4097):
        phys = rng.standard_normal((lanes, n))
        spec = rng.standard_normal((lanes, L.m))
        for op in (R.OP_FORWARD, R.OP_BACKWARD, R.OP_TO_ORTHO, R.OP_HHOLTZ):
            x = spec if op in (R.OP_BACKWARD, R.OP_TO_ORTHO) else phys
            parts = np.concatenate([L.apply(op, x[k:k + 1000]) for k in range(0, lanes, 1000)])
            np.testing.assert_array_equal(L.apply(op, x), parts)
    assert L.status() == 0


def test_mixed_packed_lanes_timeout_is_reported(R):
    L = R.Lanes(R.Base(1, 128), R.PREC_MIXED)
    x = np.random.default_rng(6).standard_normal((1100, 128))
    ref = L.apply(R.OP_FORWARD, x)
    R.set_gemm_wait_limit(0)
    try:
        L.apply(R.OP_FORWARD, x)
        assert L.status() & 2
    finally:
        R.set_gemm_wait_limit(-1)
    np.testing.assert_array_equal(L.apply(R.OP_FORWARD, x), ref)


def test_lanes_on_the_streams_of_two_threads_share_the_scratch_in_order(R):
    # cudaStreamPerThread: one handle value, a stream of its own in each thread
    import threading
    import ctypes
    n, lanes, per_thread = 130, 4096, ctypes.c_void_p(2)
    L = R.Lanes(R.Base(1, n))
    rng = np.random.default_rng(9)
    a, b = rng.standard_normal((2, lanes, n))
    ref = [L.apply(R.OP_FORWARD, x) for x in (a, b)]
    ins = [R.DeviceArray.from_host(x) for x in (a, b)]
    outs = [[R.DeviceArray((lanes, L.m)) for _ in range(8)] for _ in range(2)]
    R._check(R.lib().rbc_device_synchronize())
    gate, errors = threading.Barrier(2), []

    def work(k):
        try:
            gate.wait(60)
            for o in outs[k]:
                L.apply_dev(R.OP_FORWARD, ins[k], o, lanes, per_thread)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    R._check(R.lib().rbc_device_synchronize())
    for k in range(2):
        for o in outs[k]:
            np.testing.assert_array_equal(o.to_host(), ref[k])


@pytest.mark.parametrize("k0,n0,k1,n1", [(0, 512, 0, 257), (5, 1000, 1, 300), (1, 264, 2, 265)])
def test_noalloc_forward_beside_other_calls_of_the_space(R, k0, n0, k1, n1):
    # the documented shared state of fs_forward_noalloc is the library's buffer
    # alone: calls of the same space on another stream may overlap it
    torch = pytest.importorskip("torch")
    s = R.Space2(R.Base(k0, n0), R.Base(k1, n1))
    rng = np.random.default_rng(n0)
    v = rng.standard_normal((n0, n1))
    spec = s.forward(rng.standard_normal((n0, n1)))
    want, back = s.forward(v), s.backward(spec)
    d_v, d_spec = R.DeviceArray.from_host(v), R.DeviceArray.from_host(spec)
    outs = [R.DeviceArray(s.spectral, s.is_complex) for _ in range(10)]
    backs = [R.DeviceArray(s.physical, False) for _ in range(10)]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    R._check(R.lib().rbc_device_synchronize())
    for o, p in zip(outs, backs):
        s.forward_noalloc_dev(d_v, o, a.cuda_stream)
        s.backward_dev(d_spec, p, b.cuda_stream)
    torch.cuda.synchronize()
    for o, p in zip(outs, backs):
        np.testing.assert_array_equal(o.to_host(), want)
        np.testing.assert_array_equal(p.to_host(), back)


@pytest.mark.parametrize("n", [17, 129, 257, 46, 130])
def test_lanes_do_not_see_their_neighbours(R, n):
    # a lane's result is the same bits whatever the lane beside it holds: lanes
    # eight decades apart, a lane of zeros, a NaN, an infinity
    lanes = 700
    L = R.Lanes(R.Base(1, n), R.PREC_FP64, hholtz_c=5e-4)
    rng = np.random.default_rng(n)
    for op in (R.OP_FORWARD, R.OP_BACKWARD, R.OP_TO_ORTHO, R.OP_FROM_ORTHO, R.OP_HHOLTZ):
        x = rng.standard_normal((lanes, L.m if op in (R.OP_BACKWARD, R.OP_TO_ORTHO) else n))
        ref = L.apply(op, x)
        for first in (0, 1):
            y = x.copy()
            y[first::2] *= 1e8
            y[first + 10] = 0.0
            y[first + 20, 3] = np.nan
            y[first + 30, 2] = np.inf
            got = L.apply(op, y)
            np.testing.assert_array_equal(got[1 - first::2], ref[1 - first::2])
            assert (got[first + 10] == 0).all()


@pytest.mark.parametrize("k0,n0,k1,n1", [(5, 2048, 1, 200), (1, 264, 2, 2200), (1, 2049, 1, 100), (0, 3626, 2, 640)])
def test_space_with_one_long_axis(R, O, k0, n0, k1, n1):
    # a dense length beside an axis of more than 2044 points
    test_space_transforms_match_oracle(R, O, k0, n0, k1, n1)


def test_poisson_with_one_long_axis(R, O):
    # 198 modes as digit products over 2100 lanes
    test_poisson_with_split_eigenbasis_matches_oracle(R, O, 200, 2100)


@pytest.mark.parametrize("op", ["OP_FORWARD", "OP_BACKWARD"])
def test_fp64_lanes_timeout_leaves_nan_and_is_reported(R, op):
    n, lanes = 130, 700
    op = getattr(R, op)
    L = R.Lanes(R.Base(1, n))
    x = np.random.default_rng(7).standard_normal((lanes, n if op == R.OP_FORWARD else L.m))
    ref = L.apply(op, x)
    assert L.status() == 0
    d_in, d_out = R.DeviceArray.from_host(x), R.DeviceArray.from_host(ref)
    R.set_gemm_wait_limit(0)
    try:
        L.apply_dev(op, d_in, d_out, lanes)
        assert L.status() & 2
    finally:
        R.set_gemm_wait_limit(-1)
    assert np.isnan(d_out.to_host()).all()
    np.testing.assert_array_equal(L.apply(op, x), ref)
    assert L.status() == 0


def test_tables_of_sizes_no_longer_in_use_are_given_back(R):
    # digit operators and transform tables are shared by size and go with their
    # last user, up to 64 MB of the most recent ones
    torch = pytest.importorskip("torch")

    def free():
        R._check(R.lib().rbc_device_synchronize())
        return torch.cuda.mem_get_info()[0]

    def use(n):
        L = R.Lanes(R.Base(1, n))
        s = R.Space2(R.Base(1, n), R.Base(2, n + 1))
        c = R.Navier2D(16, n, 1e5, 1.0, 1e-3, 1.0, 0)
        c.set_temperature(0.2, 1, 1)
        del L, s, c

    use(480)
    before = free()
    for n in range(482, 522, 2):  # 20 sizes; 15 MB of tables each
        use(n)
    assert before - free() <= 80 * 2**20


@pytest.mark.parametrize("precision", [0, 1])
def test_lane_scratch_is_made_by_the_calls_that_use_it(R, precision):
    torch = pytest.importorskip("torch")

    def free():
        R._check(R.lib().rbc_device_synchronize())
        return torch.cuda.mem_get_info()[0]

    n, ops = 500, (R.OP_FORWARD, R.OP_BACKWARD)
    first = R.Lanes(R.Base(1, n), precision)  # operators that handles share, and kernels
    rng = np.random.default_rng(12)
    x = {op: rng.standard_normal((5000, n if op == R.OP_FORWARD else first.m)) for op in ops}
    ref = {op: first.apply(op, x[op]) for op in ops}
    before = free()
    handles = [R.Lanes(R.Base(1, n), precision) for _ in range(4)]
    for L in handles:  # too few lanes for it
        L.apply(R.OP_FORWARD, x[R.OP_FORWARD][:8])
    # tables of a handle: the dense transforms (2 MB), mixed the five operators of 4 n^2 bytes in two parts
    assert before - free() <= 4 * (16 if precision else 6) * 2**20
    for L, lanes in zip(handles, (1100, 4097, 128, 3000)):
        for k in (lanes, 5000, lanes):  # grown, then used for fewer lanes
            for op in ops:
                got = L.apply(op, x[op][:k])
                if k >= 1024:  # (fewer lanes may take the pass: another rounding)
                    np.testing.assert_array_equal(got, ref[op][:k])
        assert L.status() == 0


@pytest.mark.parametrize("n", [20, 127, 200])
def test_mixed_lanes_in_any_number_have_the_same_bits(R, n):
    # lane blocks of 128 with rows past the last lane, unpacked and packed
    L = R.Lanes(R.Base(1, n), R.PREC_MIXED)
    x = np.random.default_rng(n).standard_normal((1200, n))
    ref = L.apply(R.OP_FORWARD, x)
    for lanes in (1, 2, 31, 127, 128, 129, 1023, 1025):
        np.testing.assert_array_equal(L.apply(R.OP_FORWARD, x[:lanes]), ref[:lanes])
    assert L.status() == 0
