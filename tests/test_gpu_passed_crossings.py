"""Where two crossings have passed each other along a yarn (du < 0 on an
edge): the device's system against the CPU oracle, every row to 1e-11 of its
largest entry (the tolerance of the other comparisons with the reference's
system), and the reverse step against forward tangents,
g . (J d) = (J^T g) . d, at the tolerance of the identity in other states."""
import numpy as np
import pytest

import passed_cases
from pkg import gpu_available, ys
from test_gpu_adjoint import COMPS, REL, TOL, _dot, _forward_tangent, _random_direction

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.skip("no CUDA device")


def _batch(kw, k, **how):
    spec = ys.ClothSpec(**kw)
    b = ys.ClothBatch([spec])
    st = passed_cases.state(b.get_state(), kw, k, **how)
    b.set_state(**st)
    return spec, st, b


@pytest.mark.parametrize("weave,k,kf", passed_cases.CASES)
def test_system_matches_oracle(weave, k, kf):
    from oracle.oracle import ClothSpec, OracleCloth
    kw = passed_cases.kwargs(weave, kf)
    _, st, b = _batch(kw, k)
    b.assemble(1e-3)
    A, rhs = b.export_system(0)
    b.close()
    oc = OracleCloth(ClothSpec(**kw))
    oc.set_state(st)
    oc.fill()
    A_ref, b_ref = oc.system(1e-3)
    assert (np.abs(A - A_ref).max(1) / np.abs(A_ref).max(1)).max() <= 1e-11
    assert np.abs(rhs - b_ref).max() <= 1e-11 * np.abs(b_ref).max()


@pytest.mark.parametrize("mode", ["exact", "reference"])
@pytest.mark.parametrize("k", [0, 1])
def test_adjoint_identity(k, mode):
    kw = passed_cases.kwargs(1, 1000.0, base=(1e-3, 1e3, 1e-5))
    spec, st, b = _batch(kw, k, amp=1e-5)
    rng = np.random.default_rng(3)
    g = {key: rng.standard_normal((spec.num_nodes, c)) for key, c in COMPS.items()}
    adj = ys.Adjoint(b, mode)
    gs, gp, _ = adj.step_back(1e-3, g, tol=TOL, maxiter=100000)
    adj.close()
    b.close()
    d = _random_direction(spec, rng, ext=False)
    tan = _forward_tangent(spec, st, d, mode, 1e-3, 1)[0]
    lhs = [_dot(g[key], tan[key]) for key in COMPS]
    rhs = [_dot(gs[key], d[key]) for key in COMPS] + [_dot(gp[key], d[key]) for key in ("rho", "Y", "B", "S", "mu")]
    assert abs(sum(lhs) - sum(rhs)) <= REL * sum(abs(x) for x in lhs + rhs)
