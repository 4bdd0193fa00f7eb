"""Forward tangents at sizes around the tangent kernels' tiles (32 crossings a
block for friction, 64 elements a block elsewhere, cloths without an inner
bend segment) against the host emulation, whose tangents carry the whole
system's derivatives (A and b) instead of the residual's.

Both solve to 1e-14; 1e-8 of the largest tangent covers the systems' condition
(below 1e5) with the solves' and the records' rounding, as for the emulation's
other comparisons.
"""
import numpy as np
import pytest

import goldens
from emu_py import EmuCloth
from pkg import gpu_available, ys
from test_gpu_adjoint_sizes import _cloth, _state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("size", [(3, 3, 0), (3, 5, 1), (33, 3, 2), (8, 4, 0), (5, 40, 1)])
def test_tangents_by_size(size, mode):
    rng = np.random.default_rng(5)
    spec = _cloth(*size, rng)
    st = _state(spec, rng)
    N, nl = spec.num_nodes, spec.width + spec.length
    b = ys.ClothBatch([spec])
    b.set_state(**st)
    b.tangent_enable(mode)
    K = b.n_tangents
    al = np.concatenate([np.asarray(spec.warp), np.asarray(spec.weft)])
    seed = [al[:, i] * rng.standard_normal((K, nl)) for i in range(3)]
    seed += [spec.S * rng.standard_normal((K, 1)), spec.mu * rng.standard_normal((K, 1))]
    tan = dict(dlpos=1e-5 * rng.standard_normal((K, N, 3)), dlvel=1e-3 * rng.standard_normal((K, N, 3)),
               depos=1e-6 * rng.standard_normal((K, N, 2)), deposbar=1e-6 * rng.standard_normal((K, N, 2)),
               devel=1e-4 * rng.standard_normal((K, N, 2)))
    b.tangent_seed(*seed)
    b.tangent_set_state(**tan)
    assert b.step_tangent(1e-3, tol=1e-14, maxiter=100000)[0]["ok"]
    got = b.tangent_get_state()
    b.close()
    kw = {k: getattr(spec, k) for k in ("width", "length", "height", "L", "R", "pose", "weave", "warp", "weft", "kc", "kf",
                                        "df", "mu", "S", "handle_stiffness", "G", "wind_vel", "wind_density",
                                        "wind_drag", "handles")}
    em = EmuCloth(**kw)
    em.set_state(st)
    em.tangent_init(mode)
    em.tangent_seed(seed[0], seed[1], seed[2], seed[3][:, 0], seed[4][:, 0])
    em.tangent_set_state(**tan)
    assert em.step_tangent(1e-3, tol=1e-14) == 0
    want = em.tangent_get_state()
    for key in ("LPos", "LVel", "EPos", "EVel", "EPosBar"):
        for k in range(K):
            assert goldens.rel(got[key][k], want[key][k]) <= 1e-8, (key, k)
