"""ClothBatch.pcg_schedule: the schedule that a batch's solves run, whatever
arguments selected it."""
import pytest

from pkg import gpu_available, ys
from test_gpu_pcg_persistent import MIXED, SMALL, _specs

pytestmark = pytest.mark.gpu
PHASES = dict(pcg="phases", threads=0, cluster=0)


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("sides", [SMALL, MIXED, [(50, 50)], [(64, 64)]])
def test_persistent_shape(sides):
    b = ys.ClothBatch(_specs(sides, 1))
    b.set_pcg_schedule(False)
    assert b.pcg_schedule() == PHASES
    b.set_pcg_schedule(True, 1024, 16)
    run = b.pcg_schedule()
    assert run["pcg"] == "persistent"
    # four warps per 32 nodes, on at most eight such groups a CTA
    assert run["threads"] % 128 == 0 and 128 <= run["threads"] <= 1024
    assert run["cluster"] in (1, 2, 4, 8, 16)
    assert run["threads"] // 4 * run["cluster"] >= max(w * h for w, h in sides)
    b.set_pcg_schedule(True, 1024, 8)
    assert b.pcg_schedule() == run
    with pytest.raises(ys.YarnSimError):
        b.set_pcg_schedule(True, 384, 8)
    assert b.pcg_schedule() == run
    b.close()


def test_largest_cloth_of_a_cluster_and_one_row_more():
    b = ys.ClothBatch(_specs([(64, 65)], 1))
    assert b.pcg_schedule() == PHASES
    b.set_pcg_schedule(True, 1024, 16)  # 4,160 nodes: accepted, the phases run
    assert b.pcg_schedule() == PHASES
    b.close()


def test_after_the_tuner():
    b = ys.ClothBatch(_specs(SMALL, 1))
    assert b.pcg_schedule()["pcg"] == b.autotune(1e-3, steps=1)["pcg"]
    b.close()
