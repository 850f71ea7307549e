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
