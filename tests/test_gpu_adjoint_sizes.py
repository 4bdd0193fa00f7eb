"""The reverse step at sizes around its kernels' tiles (32 crossings a block
for friction, warps over a line's elements, cloths without an inner bend
segment): dL/d(state, materials) against forward tangents, g . (J d) = (J^T g) . d.

Both solves run to 1e-14 of their right-hand sides; their errors enter with
the systems' condition, below 1e5 here, so 1e-9 of the sum of the terms.
"""
import numpy as np
import pytest

from pkg import gpu_available, ys
from test_gpu_adjoint import COMPS, REL, TOL, _dot, _forward_tangent, _random_direction

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.skip("no CUDA device")


def _cloth(W, H, weave, rng):
    line = lambda n: np.array([2e-3, 170000.0, 1e-4]) * rng.uniform(0.7, 1.3, (n, 3))  # noqa: E731
    return ys.ClothSpec(width=W, length=H, weave=weave, warp=line(H), weft=line(W), handles=[(0, 0)],
                        wind_vel=(0.3, -0.2, 1.0), wind_density=1.2, wind_drag=0.5)


def _state(spec, rng):
    b = ys.ClothBatch([spec])
    st = b.get_state()
    b.close()
    N = spec.num_nodes
    st["LPos"] = st["LPos"] + 1e-5 * rng.standard_normal((N, 3))
    st["LVel"] = 1e-2 * rng.standard_normal((N, 3))
    st["EPos"] = st["EPos"] + 2e-6 * rng.standard_normal((N, 2))
    return st


@pytest.mark.parametrize("mode", ["exact", "reference"])
@pytest.mark.parametrize("sizes", [[(3, 3, 0)], [(4, 3, 1), (3, 5, 0)], [(31, 4, 2)], [(33, 3, 0), (8, 4, 1)],
                                   [(5, 40, 1)]])
def test_adjoint_identity_by_size(sizes, mode):
    rng = np.random.default_rng(11)
    specs = [_cloth(*s, rng) for s in sizes]
    states = [_state(s, rng) for s in specs]
    b = ys.ClothBatch(specs)
    b.set_state(**{k: np.concatenate([np.asarray(s[k]) for s in states]) for k in states[0]})
    g = {k: rng.standard_normal((sum(s.num_nodes for s in specs), c)) for k, c in COMPS.items()}
    adj = ys.Adjoint(b, mode)
    gs, gp, _ = adj.step_back(1e-3, g, tol=TOL, maxiter=100000)
    adj.close()
    b.close()
    n0 = l0 = 0
    for c, (spec, st) in enumerate(zip(specs, states)):
        n, nl = slice(n0, n0 + spec.num_nodes), slice(l0, l0 + spec.width + spec.length)
        n0, l0 = n.stop, nl.stop
        d = _random_direction(spec, rng, ext=False)
        tan = _forward_tangent(spec, st, d, mode, 1e-3, 1)[0]
        lhs = [_dot(g[k][n], tan[k]) for k in COMPS]
        rhs = [_dot(gs[k][n], d[k]) for k in COMPS] + [_dot(gp[k][nl], d[k]) for k in ("rho", "Y", "B")]
        rhs += [_dot(gp[k][c], d[k]) for k in ("S", "mu")]
        scale = sum(abs(x) for x in lhs + rhs)
        assert abs(sum(lhs) - sum(rhs)) <= REL * scale, (sizes[c], sum(lhs), sum(rhs), scale)
