"""Objects made where the device has the memory for them but not for the scratch
of their faster forms (digit GEMMs, packed GEMM input): they are made, and give
the results of the other form within the bounds of the parity tests."""
import contextlib
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 2**20


@pytest.fixture(scope="module")
def R():
    from rustpde_gb300 import build
    build.build()
    import rustpde_gb300
    return rustpde_gb300


def _free(torch, R):
    R._check(R.lib().rbc_device_synchronize())
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _leave(torch, R, nbytes):
    """All device memory but nbytes is taken for the body's time."""
    gc.collect()
    torch.cuda.empty_cache()
    fill = torch.empty((_free(torch, R) - nbytes) // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del fill
        torch.cuda.empty_cache()


def test_space_without_room_for_its_digits(R):
    torch = pytest.importorskip("torch")
    shape = (640, 1200)
    scratch = 10 * 40 * 28672 + 8 * shape[0] * shape[1]  # digits of 1200 lanes of 640, products
    make = lambda: R.Space2(R.Base(0, shape[0]), R.Base(0, shape[1]))  # noqa: E731
    v = np.random.default_rng(1).standard_normal(shape)
    s = make()
    want = s.forward(v)
    before = _free(torch, R)
    del s
    gc.collect()
    full = _free(torch, R) - before
    d_v, d_o = R.DeviceArray.from_host(v), R.DeviceArray(shape)
    with _leave(torch, R, full - scratch // 2):
        s = make()
        s.forward_dev(d_v, d_o)
        R._check(R.lib().rbc_device_synchronize())
    got = d_o.to_host()
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("batch", [False, True])
def test_case_without_room_for_its_digits(R, batch):
    torch = pytest.importorskip("torch")
    p = (400, 400, 1e6, 1.0, 1e-3, 1.0, 0)

    def make():
        c = R.Batch([p]) if batch else R.Navier2D(*p)
        return c, (c.cases[0] if batch else c)

    def run(c, one):
        one.set_velocity(0.2, 1, 1)
        one.set_temperature(0.2, 1, 2)
        c.update(3)
        c.synchronize()
        assert one.status() == 0
        return [one.get(f) for f in (R.TEMP, R.UX, R.UY)]

    run(*make())  # kernels and graphs loaded
    gc.collect()
    before = _free(torch, R)
    c, one = make()
    want = run(c, one)
    full = before - _free(torch, R)
    del c, one
    gc.collect()
    # the digits, the y- and the x-transformed fields: 6 and 8 values per point and more
    scratch = 8 * 14 * 400 * 400
    with _leave(torch, R, full - scratch // 2):
        c, one = make()
        got = run(c, one)
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("precision", [0, 1])
def test_served_request_without_room_for_its_digits(R, precision):
    # a budget just below the case with everything
    p = (512, 257, 1e6, 1.0, 1e-3, 1.0, R.PERIODIC, precision)
    full = R.Navier2D(*p).device_bytes()
    res = []
    for budget in (full - 10**6, 8 * 10**9):
        srv = R.Server(hbm_budget_bytes=budget, max_active=4, chunk_steps=2)
        srv.submit(p, 0.01, 3)
        assert srv.wait_idle(60.0)
        res += srv.poll()
        srv.close()
    assert [r["status"] for r in res] == [0, 0]
    assert abs(res[0]["nu"] - res[1]["nu"]) <= 1e-10 * abs(res[1]["nu"])
