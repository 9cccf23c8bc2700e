"""FP64 contractions of operands that meet in few summed indices, at sizes that go to the tensor
cores: sums of one product have the bits of that product rounded once, and the others are off by
no more than a chain of FMAs; whether tiles are cut along K or not, and in lists."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(scope="module")
def eg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300
    from einsums_gb300 import build
    build.build()
    return einsums_gb300


def cu(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def operands(rng, m, n, k, common):
    """Rows whose largest elements (columns 0 and 1 of K) meet zeros, and `common` products."""
    A, B = np.zeros((m, k)), np.zeros((k, n))
    A[:, 0], B[1] = 0.97, 0.97
    groups = rng.integers(0, 6, m)
    at = 2 + np.sort(rng.choice(k - 2, 6 * common, replace=False)).reshape(6, common)
    size = lambda *s: rng.uniform(0.04, 0.25, s) * rng.choice([-1, 1], s)
    for i in range(m):
        A[i, at[groups[i]]] = size(common)
    B[at.reshape(-1)] = size(6 * common, n)
    return A, B, at[groups]


@pytest.mark.parametrize("m,n,k", [(500, 450, 600), (300, 260, 4100), (2000, 75, 700)])
@pytest.mark.parametrize("common", [1, 2, 5])
def test_sums_of_few_products(eg, m, n, k, common):
    rng = np.random.default_rng(m + common)
    A, B, at = operands(rng, m, n, k, common)
    C = torch.full((m, n), float("nan"), dtype=torch.float64, device="cuda")
    eg.einsum(0.0, "ij", C, 1.0, "ik", cu(A), "kj", cu(B))
    got = C.cpu().numpy()
    a = np.take_along_axis(A, at, 1)  # [m, common]
    terms = a[:, :, None].astype(np.longdouble) * B[at].astype(np.longdouble)
    exact, mag = terms.sum(1), np.abs(terms).sum(1)
    if common == 1:
        assert np.array_equal(got, a * B[at[:, 0]])
    else:  # an output's sum is rounded `common` times by a chain, once here after half a rounding left out
        assert np.all(np.abs(got - exact) <= max(common, 2) * U * mag)


def test_lists(eg):
    rng = np.random.default_rng(9)
    As, Bs, want = [], [], []
    for q in range(400):
        m, n, k = int(rng.integers(40, 121)), int(rng.integers(40, 121)), int(rng.integers(300, 900))
        A, B, at = operands(rng, m, n, k, 1)
        As.append(cu(A)), Bs.append(cu(B))
        want.append(np.take_along_axis(A, at, 1) * B[at[:, 0]])
    Cs = [torch.full(w.shape, float("nan"), dtype=torch.float64, device="cuda") for w in want]
    plan = eg.GroupedPlan(0.0, "ij", Cs, 1.0, "ik", As, "kj", Bs)
    plan.execute()
    torch.cuda.synchronize()
    for C, w in zip(Cs, want):
        assert np.array_equal(C.cpu().numpy(), w)
    plan.close()
