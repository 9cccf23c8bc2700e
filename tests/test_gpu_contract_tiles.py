"""The plain FP64 contraction at the edges of its tiles: extents around the 8, 16
and 32 tile edges and the k chunks, K cut over clusters of 2, 4 and 8 CTAs,
operands read along rows, along k, and through several k modes, with batches."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300
    from einsums_gb300 import build
    build.build()
    return einsums_gb300


def cu(x):
    return torch.from_numpy(np.array(x, dtype=np.float64, order="C", copy=True)).cuda()


def check(got, want, scale, K):
    # K products and K - 1 additions, each rounded once, then the prefactors: (K + 4) 2^-53 of the sum of magnitudes
    assert np.all(np.abs(got - want) <= (K + 4) * 2.0 ** -53 * scale * 1.0001)


@pytest.mark.parametrize("m,n,k", [(1, 2, 3), (2, 2, 1), (7, 9, 31), (8, 8, 32), (9, 7, 33), (16, 17, 64),
                                   (15, 33, 65), (31, 65, 127), (40, 60, 50), (64, 64, 64), (96, 100, 16),
                                   (5, 6, 5000), (33, 18, 1030), (200, 130, 77), (700, 500, 24)])
@pytest.mark.parametrize("layout", ["ik,kj", "ki,jk", "ki,kj", "ik,jk"])
def test_tile_edges(eg, m, n, k, layout):
    rng = np.random.default_rng(m * 1000 + n * 10 + k)
    Al, Bl = layout.split(",")
    d = {"i": m, "j": n, "k": k}
    A, B = rng.standard_normal([d[c] for c in Al]), rng.standard_normal([d[c] for c in Bl])
    C0 = rng.standard_normal((m, n))
    A2, B2 = (A if Al == "ik" else A.T), (B if Bl == "kj" else B.T)
    want = (0.5 * C0.astype(np.longdouble) - 1.25 * (A2.astype(np.longdouble) @ B2.astype(np.longdouble))).astype(float)
    C = cu(C0)
    eg.einsum(0.5, "ij", C, -1.25, Al, cu(A), Bl, cu(B))
    check(C.cpu().numpy(), want, 0.5 * np.abs(C0) + 1.25 * (np.abs(A2) @ np.abs(B2)), k)


@pytest.mark.parametrize("d", [dict(b=3, i=9, j=7, m=5, n=11), dict(b=1, i=40, j=8, m=17, n=40),
                               dict(b=2, i=33, j=2, m=3, n=700)])
def test_modes_batches_and_views(eg, d):
    rng = np.random.default_rng(sum(d.values()))
    A = rng.standard_normal([d[c] for c in "bminx".replace("x", "")])
    big = rng.standard_normal((d["n"], d["b"], d["j"], 2 * d["m"]))
    B = big[..., ::2]
    C = torch.full((d["b"], d["i"], d["j"]), float("nan"), dtype=torch.float64, device="cuda")
    want = np.zeros(tuple(C.shape))
    oracle.einsum("bij", want, 0.0, 1.0, "bmin", A, "nbjm", B)
    eg.einsum(0.0, "bij", C, 1.0, "bmin", cu(A), "nbjm", cu(big)[..., ::2])
    scale = np.einsum("bmin,nbjm->bij", np.abs(A), np.abs(B))
    check(C.cpu().numpy(), want, 2 * scale, d["m"] * d["n"])
