"""The tensor kernel's tiles and schedules, bit for bit against the CPU restatement of the split
product: single CTAs and CTA pairs (chosen by estimate, or forced through the environment in
child processes), rows around the 128- and 256-row tiles, K of one and of many K blocks, tiles of
the last round cut along K, every slice count, C along its rows, along its columns and strided,
and the FP64 form under both kinds of tiles."""
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [(5, 7, 5, 64), (128, 128, 5, 64), (129, 65, 5, 130), (255, 130, 2, 200), (256, 5, 3, 1088), (257, 257, 4, 640),
         (300, 200, 6, 128), (700, 900, 5, 4100), (1300, 1300, 5, 330), (2600, 1300, 4, 200)]


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


def run_split(eg, M, N, S, K):
    from test_split_math import split_product_fast
    rng = np.random.default_rng(M + 3 * N + 7 * K + S)
    A = rng.standard_normal((M, K)) * np.exp2(rng.integers(-30, 30, size=(M, 1)))
    B = rng.standard_normal((N, K))
    rows = np.unique(np.concatenate([rng.choice(M, min(M, 40), replace=False), [0, M - 1, min(127, M - 1), min(128, M - 1)]]))
    ref = split_product_fast(A[rows], B, S)
    C0 = rng.standard_normal((M, N))
    same = lambda got, want: np.array_equal(got.view(np.uint64), np.ascontiguousarray(want).view(np.uint64))
    # along C's columns, and scaled by -1/2 into old values
    C = cu(C0)
    eg.einsum(1.0, "ij", C, -0.5, "ik", cu(A), "jk", cu(B), precision="split_bf16", slices=S)
    assert same(np.ascontiguousarray(C.cpu().numpy()[rows]), C0[rows] + -0.5 * ref), "columns"
    # along C's rows
    Ct = torch.full((N, M), float("nan"), dtype=torch.float64, device="cuda")
    eg.einsum(0.0, "ji", Ct, 1.0, "ik", cu(A), "jk", cu(B), precision="split_bf16", slices=S)
    assert same(np.ascontiguousarray(Ct.cpu().numpy()[:, rows].T), ref), "rows"
    # a strided C with another prefactor
    big = torch.zeros((M, 2 * N), dtype=torch.float64, device="cuda")
    eg.einsum(0.0, "ij", big[:, ::2], 3.0, "ik", cu(A), "jk", cu(B), precision="split_bf16", slices=S)
    assert same(np.ascontiguousarray(big[:, ::2].cpu().numpy()[rows]), 3.0 * ref), "strided"
    assert not torch.any(big[:, 1::2])


def run_f64(eg, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A, B, C0 = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    A[m // 2] *= 10.0 ** np.linspace(-9, 9, k)  # a few blocks fail the check
    B[:, n // 3] /= 10.0 ** np.linspace(-9, 9, k)
    C = cu(C0)
    eg.einsum(1.0, "ij", C, 0.25, "ik", cu(A), "kj", cu(B))
    rows = np.unique(np.concatenate([rng.choice(m, 10, replace=False), [m // 2, m - 1, min(m - 1, 128)]]))
    want = (C0[rows].astype(np.longdouble) + 0.25 * (A[rows].astype(np.longdouble) @ B.astype(np.longdouble))).astype(float)
    scale = np.abs(C0[rows]) + 0.25 * (np.abs(A[rows]) @ np.abs(B))
    assert np.all(np.abs(C.cpu().numpy()[rows] - want) <= (k + 4) * 2.0 ** -53 * scale)


F64_CASES = [(600, 500, 700), (129, 1500, 640), (1300, 1300, 130), (90000, 75, 75)]


@pytest.mark.parametrize("M,N,S,K", CASES)
def test_tiles_by_estimate(eg, M, N, S, K):
    run_split(eg, M, N, S, K)


def forced():
    import einsums_gb300 as eg
    for c in CASES:
        run_split(eg, *c)
    for c in F64_CASES:
        run_f64(eg, *c)
    print("ran", len(CASES) + len(F64_CASES))


@pytest.mark.parametrize("pairs", ["0", "1"])
def test_tiles_forced(eg, pairs):
    here = os.path.dirname(os.path.abspath(__file__))
    root = os.path.dirname(here)
    path = os.pathsep.join([root, os.path.join(root, "oracle"), here, os.environ.get("PYTHONPATH", "")])
    env = dict(os.environ, EINSUMS_GB300_TC_PAIRS=pairs, PYTHONPATH=path)
    r = subprocess.run([sys.executable, "-c", "import test_gpu_tensor_tiles as t; t.forced()"], cwd=here, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "ran 14" in r.stdout, r.stdout + r.stderr


def test_subnormal_and_huge_results(eg):
    """Results at both ends of the range take the conversion that is not the fast one."""
    from test_split_math import split_product_fast
    rng = np.random.default_rng(9)
    A, B = rng.standard_normal((70, 100)), rng.standard_normal((90, 100))
    ref = split_product_fast(A, B, 5)
    for e in (-1060, -1022, 1015):
        C = torch.zeros((70, 90), dtype=torch.float64, device="cuda")
        eg.einsum(0.0, "ij", C, 1.0, "ik", cu(np.ldexp(A, e // 2)), "jk", cu(np.ldexp(B, e - e // 2)),
                  precision="split_bf16", slices=5)
        with np.errstate(over="ignore", under="ignore"):
            want = np.ldexp(ref, e)
        # one rounding of the exact sum against two: at most one unit of the last place apart
        ok = np.abs(C.cpu().numpy() - want) <= np.maximum(np.abs(np.spacing(want)), 5e-324)
        assert np.all(ok | (C.cpu().numpy() == want))


@pytest.mark.parametrize("K", [65, 130, 1111, 5000, 20000, 26000])
@pytest.mark.parametrize("layout", ["k", "k odd base", "k odd stride", "rows", "both strided", "two k modes"])
def test_operand_splitting(eg, K, layout):
    """The splitting launch: K of one CTA and of clusters, 32 and 8 rows, and beyond (the passes);
    operands read along k (in pairs when aligned), along rows, or strided both ways."""
    from test_split_math import split_product_fast
    M, N, S = 45, 6, 3
    rng = np.random.default_rng(K + len(layout))
    A = rng.standard_normal((M, K)) * np.exp2(rng.integers(-9, 9, size=(M, 1)))
    B = rng.standard_normal((N, K))
    A[7] = 0.0
    labels = "ik"
    if layout == "k":
        tA = cu(A)
    elif layout == "k odd base":
        tA = cu(np.concatenate([np.zeros(1), A.ravel()]))[1:].view(M, K)
    elif layout == "k odd stride":
        tA = cu(np.concatenate([A, np.zeros((M, 1 + K % 2))], 1))[:, :K]
    elif layout == "rows":
        tA = cu(A.T).T
    elif layout == "both strided":
        big = torch.zeros((M, 2 * K), dtype=torch.float64, device="cuda")
        big[:, ::2] = cu(A)
        tA = big[:, ::2]
    else:
        q = next(d for d in (13, 11, 5, 2) if K % d == 0)
        tA, labels = cu(A.reshape(M, q, K // q).transpose(1, 0, 2)), "kil"
    tB = cu(B)
    C = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    if labels == "ik":
        eg.einsum(0.0, "ij", C, 1.0, "ik", tA, "jk", tB, precision="split_bf16", slices=S)
    else:
        eg.einsum(0.0, "ij", C, 1.0, "kil", tA, "jkl", tB.view(N, q, K // q), precision="split_bf16", slices=S)
    want = split_product_fast(A, B, S)
    assert np.array_equal(C.cpu().numpy().view(np.uint64), np.ascontiguousarray(want).view(np.uint64))
