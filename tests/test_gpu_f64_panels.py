"""FP64 contractions on the tensor cores whose digit planes go through the scratch in panels -- of
batch indices, of A's rows with B's planes kept, of both -- with blocks in later panels that fail the
accuracy check, and batched and strided operands.  Inputs are whole numbers, in part graded by powers
of two that cancel in every product, so results are exact whatever computes them."""
import ctypes

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
    yield einsums_gb300
    einsums_gb300.trim_memory()


def launched(eg, *args, **kw):
    """einsum, and {kernel: launches}."""
    from einsums_gb300 import _lib
    lib = _lib.load()
    buf = ctypes.create_string_buffer(1 << 16)
    lib.eg_profile_enable(1)
    lib.eg_profile_reset()
    try:
        eg.einsum(*args, **kw)
        torch.cuda.synchronize()
        _lib.check(lib.eg_profile_summary(buf, len(buf)))
    finally:
        lib.eg_profile_enable(0)
    return {line.split(",")[0]: int(line.split(",")[1]) for line in buf.value.decode().split()}


def whole(gen, *shape):
    return torch.randint(-40, 41, shape, generator=gen, device="cuda").to(torch.float64)


@pytest.fixture
def gen():
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    return g


def test_batch_indices_in_panels(eg, gen):
    # 81920 bytes of planes a row: 26112 rows of both operands at a time, four of nine indices
    nb, m, n, k = 9, 3000, 3100, 4096
    A, B = whole(gen, nb, m, k), whole(gen, nb, k, n)
    C0 = whole(gen, nb, m, n)
    want = C0 + 2 * torch.bmm(A, B)
    grade = torch.exp2(torch.linspace(-30, 30, k, dtype=torch.float64, device="cuda").round())
    for b, rows in ((2, slice(0, 40)), (5, slice(2900, 3000)), (8, slice(1000, 1400))):  # graded against each other
        A[b, rows] *= grade
        B[b, :, 1500:1700] /= grade[:, None]
        A[b, rows.stop:] = 0.0
        A[b, :rows.start] = 0.0
        want[b] = C0[b]
        keep = torch.zeros(n, dtype=torch.bool, device="cuda")
        keep[1500:1700] = True
        B[b, :, ~keep] = 0.0
        want[b, rows, 1500:1700] += 2 * ((A[b, rows] / grade) @ (B[b, :, 1500:1700] * grade[:, None]))
    C = C0.clone()
    kernels = launched(eg, 1.0, "bij", C, 2.0, "bik", A, "bkj", B)
    assert kernels["k_tc_split_gemm_f64"] == 3 and kernels["k_contract_f64_listed"] == 1
    assert torch.equal(C, want)


@pytest.mark.parametrize("m,n,k,tensor", [(30000, 1000, 8192, 3), (9000, 8000, 8192, 4)])
def test_rows_in_panels(eg, gen, m, n, k, tensor):
    # 163872 bytes of planes a row, 13056 rows at a time: B's planes stay, or both operands in halves
    A, B = whole(gen, m, k), whole(gen, k, n)
    want = A @ B
    grade = torch.exp2(torch.linspace(-30, 30, k, dtype=torch.float64, device="cuda").round())
    A[m - 700:] *= grade  # in the last panel, against every column: those that match it by 1 / grade
    B[:, 300:500] /= grade[:, None]
    want[m - 700:] = float("nan")
    want[:, 300:500] = float("nan")
    want[m - 700:, 300:500] = (A[m - 700:] / grade) @ (B[:, 300:500] * grade[:, None])
    exact = ~torch.isnan(want)
    C = torch.full((m, n), float("nan"), dtype=torch.float64, device="cuda")
    kernels = launched(eg, 0.0, "ij", C, 1.0, "ik", A, "kj", B)
    assert kernels["k_tc_split_gemm_f64"] == tensor and kernels["k_contract_f64_listed"] == 1
    assert torch.equal(C[exact], want[exact])
    assert not torch.isnan(C).any()
    rows, cols = [m - 1, m - 700, 5], [300, 499, 0, n - 1]  # and where one side alone is graded
    a, b = A[rows].cpu().numpy(), B[:, cols].cpu().numpy()
    ref = (a.astype(np.longdouble) @ b.astype(np.longdouble)).astype(float)
    assert np.all(np.abs(C[rows][:, cols].cpu().numpy() - ref) <= (k + 4) * U * (np.abs(a) @ np.abs(b)))


def test_batched_and_strided_operands(eg, gen):
    A, B = whole(gen, 3, 40, 15, 30, 22), whole(gen, 22, 3, 50, 15, 34)
    big = torch.zeros((30, 50, 3, 40, 68), dtype=torch.float64, device="cuda")
    C = big[..., ::2]
    kernels = launched(eg, 0.0, "enbij", C, 1.0, "bikel", A, "lbnkj", B)
    assert "k_tc_split_gemm_f64" in kernels and "k_contract_f64" not in kernels
    assert torch.equal(C, torch.einsum("bikel,lbnkj->enbij", A, B))
    assert torch.all(big[..., 1::2] == 0)


@pytest.mark.parametrize("conj", [False, True])
def test_complex_bound(eg, conj):
    """Every part of a complex output within eight roundings of its products' magnitudes."""
    rng = np.random.default_rng(3)
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    A, B = z(400, 300), z(300, 260)
    C = torch.full((400, 260), float("nan"), dtype=torch.complex128, device="cuda")
    kernels = launched(eg, 0.0, "ij", C, 1.0, "ik", torch.from_numpy(A).cuda(), "kj", torch.from_numpy(B).cuda(), conj_A=conj)
    assert "k_tc_split_gemm_f64" in kernels
    rows = [0, 31, 32, 127, 128, 255, 399]
    a, b, got = (A.conj() if conj else A)[rows], B, C[rows].cpu().numpy()
    mm = lambda x, y: x.astype(np.longdouble) @ y.astype(np.longdouble)
    for part, want, mag in ((got.real, mm(a.real, b.real) - mm(a.imag, b.imag),
                             np.abs(a.real) @ np.abs(b.real) + np.abs(a.imag) @ np.abs(b.imag)),
                            (got.imag, mm(a.real, b.imag) + mm(a.imag, b.real),
                             np.abs(a.real) @ np.abs(b.imag) + np.abs(a.imag) @ np.abs(b.real))):
        assert np.all(np.abs(part - want.astype(float)) <= 8 * U * mag)
