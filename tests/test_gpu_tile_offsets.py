"""Many short tiles on one CTA, C along its rows and not read: each tile's output offsets replace
the ones before only once every lane has stored with those.  Whole numbers, so results are exact."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["split_bf16", "fp64"])
def test_short_tiles_one_after_another(precision):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300 as eg
    rng = np.random.default_rng(7)
    As, Bs = [], []
    for q in range(1200):  # items of other extents than their neighbours on a CTA
        i, a, b = int(rng.integers(33, 70)), int(rng.integers(20, 129)), int(rng.integers(5, 129))
        As.append(torch.from_numpy(rng.integers(-9, 10, (i, a)).astype(float)).cuda())
        Bs.append(torch.from_numpy(rng.integers(-9, 10, (i, b)).astype(float)).cuda())
    Cs = [torch.full((B.shape[1], A.shape[1]), float("nan"), dtype=torch.float64, device="cuda") for A, B in zip(As, Bs)]
    plan = eg.GroupedPlan(0.0, "ba", Cs, 1.0, "ia", As, "ib", Bs, precision=precision)
    for _ in range(4):
        plan.execute()
    torch.cuda.synchronize()
    for A, B, C in zip(As, Bs, Cs):
        assert torch.equal(C, (A.T @ B).T)
    plan.close()
