"""The two PCG schedules against each other with each one selected by name: a
batch's default is the persistent PCG wherever it is expected to be faster, so
a comparison with the default may compare it with itself. Same arithmetic and
order, hence the same bits, over several steps with h and the external force
changing, launch by launch and as a graph (the phases' graph holds the
conditional while node), at cluster splits of one to eight groups of 32 nodes a
CTA, and in the reference mode's reverse solve. Then the element producers'
block sizes where each kernel is launched on its own."""
import numpy as np
import pytest

from pkg import gpu_available, ys
from test_gpu_pcg_persistent import MIXED, SMALL, _same, _specs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.skip("no CUDA device")


def _batch(sides, seed, persistent):
    b = ys.ClothBatch(_specs(sides, seed))
    b.set_pcg_schedule(persistent, 1024, 16)
    assert b.pcg_schedule()["pcg"] == ("persistent" if persistent else "phases")
    return b


def _steps(sides, persistent, graphed, every=4):
    b = _batch(sides, 3, persistent)
    b.use_graphs(graphed)
    ext = 1e-4 * np.random.default_rng(4).standard_normal((b.total_nodes, 5))
    out = []
    for k, h in enumerate([1e-3] * 4 + [5e-4] * 2):
        stats = b.step(h, ext if k % 2 else None, tol=1e-10, check_every=every)
        assert all(s["ok"] for s in stats)
        out.append((b.get_state(), [(s["cg_iterations"], s["cg_error"]) for s in stats]))
    shape = b.pcg_schedule()
    b.close()
    return out, shape


@pytest.mark.parametrize("sides", [SMALL, MIXED])
def test_steps_in_both_schedules(sides):
    ref, _ = _steps(sides, False, False)
    for persistent, graphed, every in ((False, True, 4), (False, True, 2), (False, False, 7), (True, False, 4), (True, True, 4)):
        _same(ref, _steps(sides, persistent, graphed, every)[0])


@pytest.mark.parametrize("side,groups", [(22, 1), (31, 2), (39, 3), (45, 4), (50, 5), (54, 6), (57, 7), (64, 8)])
def test_cluster_splits(side, groups):
    """One cloth of side^2 nodes on 16 CTAs of `groups` groups."""
    ref, _ = _steps([(side, side)], False, False)
    got, shape = _steps([(side, side)], True, False)
    assert shape == dict(pcg="persistent", threads=128 * groups, cluster=16)
    _same(ref, got)


@pytest.mark.parametrize("mode", ["exact", "reference"])
def test_reverse_solves(mode):
    outs = []
    for persistent in (False, True):
        b = _batch([(12, 13), (5, 9)], 7, persistent)
        rng = np.random.default_rng(4)
        g = {k: rng.standard_normal((b.total_nodes, c))
             for k, c in dict(LPos=3, LVel=3, EPos=2, EVel=2, EPosBar=2).items()}
        adj = ys.Adjoint(b, mode)
        gs, gp, ge = adj.step_back(1e-3, g, None, tol=1e-12, maxiter=100000, want_ext=True)
        outs.append({**gs, **gp, "ext": ge})
        adj.close()
        b.close()
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k]), k


@pytest.mark.parametrize("threads", [32, 64, 256])
@pytest.mark.parametrize("sides,graphed", [(MIXED, True), ([(3, 5), (12, 11)] * 160, False)])
def test_producer_block_sizes_launched_apart(sides, graphed, threads):
    """A graph launches edges, bends, faces and shear by themselves, and so does
    a batch of more 128-node blocks (480) than two an SM."""
    def run(t):
        b = ys.ClothBatch(_specs(sides, 9))
        b.use_graphs(graphed)
        if t:
            b.set_producer_threads(t)
        out = []
        for _ in range(2):
            assert all(s["ok"] for s in b.step(1e-3, tol=1e-10))
            out.append(b.get_state())
        b.close()
        return out
    for a, c in zip(run(None), run(threads)):
        for k in a:
            assert np.array_equal(a[k], c[k]), k
