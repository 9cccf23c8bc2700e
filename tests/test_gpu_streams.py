"""Memory-bound FP64 passes at the edges of their routes: rows and tiles of the permutation
(odd, even, short and long rows, C_prefactor, bases off a 16-byte boundary), elementwise
products over contiguous ranges, sums of one launch and of two, and matrix-vector products
whose summed modes are one run, two nested runs or neither.

Permutations are compared bit for bit with the oracle.  An elementwise product rounds at most
four times; a sum over K has at most K / 256 + 24 additions on a path, each with an error of at
most 2^-53 of the sum of the magnitudes."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def eg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300
    from einsums_gb300 import build
    build.build()
    return einsums_gb300


def cu(x, off=0):
    """x on the device, `off` doubles past an aligned address."""
    x = np.ascontiguousarray(x, dtype=np.float64)
    t = torch.empty(x.size + off, dtype=torch.float64, device="cuda")[off:].view(x.shape)
    t.copy_(torch.from_numpy(x))
    return t


@pytest.mark.parametrize("L", [2, 7, 64, 65, 127, 128, 129, 256, 257, 4098])
@pytest.mark.parametrize("cp,ap", [(0.0, 1.0), (0.0, -2.5), (0.75, 1.5), (1.0, 1.0), (1.0, -1.0), (1.0, 0.5)])
def test_permute_rows(eg, L, cp, ap):
    rng = np.random.default_rng(L)
    for shape, off in [((5, 9, L), 0), ((5, 9, L), 1), ((67, 33, L), 0)]:
        A, C0 = rng.standard_normal(shape), rng.standard_normal((shape[1], shape[0], L))
        C = cu(C0, off)
        eg.permute(cp, "jis", C, ap, "ijs", cu(A, off))
        oracle.permute("jis", C0, cp, ap, "ijs", A)
        assert np.array_equal(C.cpu().numpy().view(np.uint64), C0.view(np.uint64)), (shape, off)


@pytest.mark.parametrize("m,n", [(1, 33), (31, 32), (33, 257), (65, 300), (129, 31)])
@pytest.mark.parametrize("cp,ap", [(0.0, 1.0), (0.0, 3.0), (-0.5, 1.5), (1.0, 1.0), (1.0, -1.0), (-1.0, 1.0)])
def test_permute_tiles(eg, m, n, cp, ap):
    rng = np.random.default_rng(m + n)
    for off in (0, 1):
        A, C0 = rng.standard_normal((m, 3, n)), rng.standard_normal((n, 3, m))
        C = cu(C0, off)
        eg.permute(cp, "nkm", C, ap, "mkn", cu(A, off))
        oracle.permute("nkm", C0, cp, ap, "mkn", A)
        assert np.array_equal(C.cpu().numpy().view(np.uint64), C0.view(np.uint64)), off


@pytest.mark.parametrize("shape", [(1, 1), (1, 3), (32, 64), (33, 65), (700, 801)])
@pytest.mark.parametrize("cp,ab", [(0.0, 1.0), (0.0, -1.5), (1.0, 1.0), (0.3, 2.0)])
def test_elementwise(eg, shape, cp, ab):
    rng = np.random.default_rng(shape[0])
    A, B, C0 = (rng.standard_normal(shape) for _ in range(3))
    want = cp * C0 + ab * (A * B)
    bound = 4 * EPS * (np.abs(cp * C0) + np.abs(ab * A * B))
    for off in (0, 1):
        C = cu(C0, off)
        eg.einsum(cp, "ij", C, ab, "ij", cu(A), "ij", cu(B, off))
        assert np.all(np.abs(C.cpu().numpy() - want) <= bound), off
    C = cu(C0.T)  # C in another order: not one run
    eg.einsum(cp, "ji", C, ab, "ij", cu(A), "ij", cu(B))
    assert np.all(np.abs(C.cpu().numpy().T - want) <= bound)
    old = cu(np.where(cp == 0.0, np.nan, C0))  # zero times an old NaN does not reach the result
    eg.einsum(cp, "ij", old, ab, "ij", cu(A), "ij", cu(B))
    assert np.all(np.abs(old.cpu().numpy() - want) <= bound)


def sums(A, B):
    """Exact products' sums over the last axis, to more than 64 bits, and the sums of magnitudes."""
    p = A.astype(np.longdouble) * B.astype(np.longdouble)
    return p.sum(-1), np.abs(p).sum(-1).astype(np.float64)


@pytest.mark.parametrize("K", [1, 31, 511, 4097, 16384, 16385, 50001, 400002])
def test_dot(eg, K):
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal(K), rng.standard_normal(K)
    want, mag = sums(A, B)
    for cp, ab, off in [(0.0, 1.0, 0), (0.0, 1.0, 1), (0.5, -2.0, 0)]:
        C = torch.tensor(3.0, dtype=torch.float64, device="cuda")
        eg.einsum(cp, "", C, ab, "i", cu(A, off), "i", cu(B))
        ref = float(cp * 3.0 + ab * want)
        assert abs(float(C) - ref) <= EPS * ((K / 256 + 24) * abs(ab) * mag + 3 * abs(cp)), (cp, off)
    strided = cu(np.repeat(A, 2))[::2]
    C = torch.tensor(3.0, dtype=torch.float64, device="cuda")
    eg.einsum(0.0, "", C, 1.0, "i", strided, "i", cu(B))
    assert abs(float(C) - float(want)) <= EPS * (K / 256 + 24) * mag
    for a in (cu(A), strided):  # a dot product scales C even by zero, as the reference does
        C = torch.tensor(float("nan"), dtype=torch.float64, device="cuda")
        eg.einsum(0.0, "", C, 1.0, "i", a, "i", cu(B))
        assert np.isnan(float(C))


@pytest.mark.parametrize("k,l", [(50, 42), (51, 43), (1, 2100), (300, 7), (3, 1024), (64, 33)])
@pytest.mark.parametrize("rows", [2, 5, 161])
def test_matrix_vector(eg, k, l, rows):
    rng = np.random.default_rng(k * l + rows)
    A, B = rng.standard_normal((rows, k, l)), rng.standard_normal((k, l))
    want, mag = sums(A.reshape(rows, -1), B.reshape(1, -1))
    bound = EPS * ((k * l / 256 + 24) * mag)
    ok = lambda C: np.all(np.abs(C.cpu().numpy() - want.astype(np.float64)) <= bound)
    for off in (0, 1):
        C = cu(np.full(rows, np.nan))
        eg.einsum(0.0, "i", C, 1.0, "ikl", cu(A, off), "kl", cu(B, off))  # one run
        assert ok(C), off
        C = cu(np.full(rows, np.nan))
        eg.einsum(0.0, "i", C, 1.0, "kil", cu(A.transpose(1, 0, 2), off), "kl", cu(B))  # nested runs
        assert ok(C), off
        C = cu(np.full(rows, np.nan))
        eg.einsum(0.0, "i", C, 1.0, "kl", cu(B, off), "kil", cu(A.transpose(1, 0, 2)))  # the vector first
        assert ok(C), off
    C = cu(np.full(rows, np.nan))
    eg.einsum(0.0, "i", C, 1.0, "lki", cu(A.transpose(2, 1, 0)), "kl", cu(B))  # neither
    assert ok(C)
