"""The FP64 contraction on the tensor cores against exact products: every output within the
bound the path promises, blocks that fail its accuracy check recomputed by the FMA kernel,
and the calls that keep to the FMA kernel (capture, a memory budget)."""
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
    return einsums_gb300


def cu(x):
    return torch.from_numpy(np.array(x, dtype=np.float64, order="C", copy=True)).cuda()


def run(eg, *args, **kw):
    """einsum, and the kernels it launched."""
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
    return buf.value.decode()


def dd_matmul(A, B):
    """A @ B in extended precision (numpy long double; on the GPU machine this is 113-bit software)."""
    return A.astype(np.longdouble) @ B.astype(np.longdouble)


@pytest.mark.parametrize("m,n,k,cp,ab", [(512, 512, 256, 0.0, 1.0), (513, 385, 129, 1.0, -0.5), (127, 1100, 500, 0.5, 3.0),
                                         (640, 300, 1000, 1.0, 1.0), (128, 129, 4100, -1.0, 0.25), (2000, 75, 75, 0.0, 1.0),
                                         (1025, 897, 129, 1.0, -0.5), (90000, 75, 75, 0.0, 1.0)])
def test_ordinary_data_within_bound(eg, m, n, k, cp, ab):
    rng = np.random.default_rng(m + n + k)
    A, B, C0 = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    rows = rng.choice(m, 24, replace=False)
    C = cu(C0)
    kernels = run(eg, cp, "ij", C, ab, "ik", cu(A), "kj", cu(B))
    assert "k_tc_split_gemm_f64" in kernels or m * n * k < 4e7 # the FMA kernel's
    got = C.cpu().numpy()
    want = (np.longdouble(cp) * C0[rows] + np.longdouble(ab) * dd_matmul(A[rows], B)).astype(float)
    scale = np.abs(cp * C0[rows]) + np.abs(ab) * (np.abs(A[rows]) @ np.abs(B))
    # four roundings' worth of truncation, then at most four roundings (sum, ab, cp, addition)
    assert np.all(np.abs(got[rows] - want) <= 8 * U * scale)
    # and off by no more, over all, than a chain of FMAs
    chain = np.zeros((len(rows), n))
    for q in range(k):
        chain += A[rows][:, q:q + 1] * B[q]
    err = lambda x: np.linalg.norm(x - (dd_matmul(A[rows], B)).astype(float))
    if cp == 0.0 and ab == 1.0:
        assert err(got[rows]) <= err(chain)


@pytest.mark.parametrize("case", ["graded", "one block", "inf", "nan", "zeros", "sparse", "tiny", "huge"])
def test_hard_data(eg, case):
    m, n, k = 500, 450, 600
    rng = np.random.default_rng(len(case))
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if case == "graded":
        d = 10.0 ** np.linspace(-9, 9, k)
        A, B = A * d, B / d[:, None]
    elif case == "one block":  # one row of A graded against every column of B
        d = 10.0 ** np.linspace(-9, 9, k)
        A[131] *= d
        B[:, 70] /= d
    elif case == "inf":
        A[5, 7], B[9, 200] = np.inf, -np.inf
        A[300] = 0.0
    elif case == "nan":
        A[450, 599] = np.nan
    elif case == "zeros":
        A[:, ::3], B[1::3] = 0.0, 0.0
        A[17], B[:, 33] = 0.0, 0.0
    elif case == "sparse":
        A *= rng.random(A.shape) < 0.02
        B *= rng.random(B.shape) < 0.02
    elif case == "tiny":
        A, B = A * 1e-290, B * 1e-5
    elif case == "huge":
        A, B = A * 1e200, B * 1e100
    C = torch.full((m, n), 7.0, dtype=torch.float64, device="cuda")
    kernels = run(eg, 0.0, "ij", C, 1.0, "ik", cu(A), "kj", cu(B))
    assert "k_tc_split_gemm_f64" in kernels
    got = C.cpu().numpy()
    with np.errstate(all="ignore"):
        rows = np.unique(np.concatenate([rng.choice(m, 12, replace=False), [5, 17, 131, 300, 450]]))
        want = dd_matmul(A[rows], B).astype(float)
        scale = np.abs(A[rows]) @ np.abs(B)
        fin = np.isfinite(scale)
        assert np.all(np.abs(got[rows] - want)[fin] <= (k + 4) * U * scale[fin] + 1e-322)
        # infinities and NaN where the FMA chain has them
        plain = np.where(np.isfinite(want), 0.0, want)
        have = np.where(np.isfinite(got[rows]), 0.0, got[rows])
        assert np.array_equal(np.isnan(plain), np.isnan(have))
        assert np.array_equal(plain[~np.isnan(plain)], have[~np.isnan(have)])
    if case in ("graded", "one block", "sparse"):  # graded: nearly every output would have failed the bound
        assert np.all(np.abs(got[rows] - want) <= (k + 4) * U * scale)


def test_modes_and_batches(eg):
    rng = np.random.default_rng(3)
    # both operands' summed modes strided, a batch index, C strided
    A, B = rng.standard_normal((3, 20, 15, 18, 22)), rng.standard_normal((22, 3, 25, 15, 17))
    big = torch.zeros((18, 25, 3, 20, 34), dtype=torch.float64, device="cuda")
    C = big[..., ::2]
    kernels = run(eg, 0.0, "enbij", C, 1.0, "bikel", cu(A), "lbnkj", cu(B))
    want = np.einsum("bikel,lbnkj->enbij", A, B)
    scale = np.einsum("bikel,lbnkj->enbij", np.abs(A), np.abs(B))
    assert np.all(np.abs(C.cpu().numpy() - want) <= 2 * (330 + 4) * U * scale)
    assert torch.all(big[..., 1::2] == 0)
    assert "k_" in kernels


def test_panels_of_a_long_summed_extent(eg):
    # K = 60000: ten planes of 1.2 MB a row, so both operands go through the scratch in panels
    m, n, k = 1000, 900, 60000
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    A = torch.randn((m, k), generator=gen, dtype=torch.float64, device="cuda")
    B = torch.randn((k, n), generator=gen, dtype=torch.float64, device="cuda")
    C = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    kernels = run(eg, 0.0, "ij", C, 1.0, "ik", A, "kj", B)
    assert "k_tc_split_gemm_f64" in kernels
    rows, cols = [0, 127, 128, 700, 895, 896, 999], [0, 1, 127, 128, 450, 899]
    want = dd_matmul(A[rows].cpu().numpy(), B[:, cols].cpu().numpy()).astype(float)
    scale = np.abs(A[rows].cpu().numpy()) @ np.abs(B[:, cols].cpu().numpy())
    assert np.all(np.abs(C.cpu().numpy()[np.ix_(rows, cols)] - want) <= 8 * U * scale)


def test_capture_and_budget_keep_the_fma_kernel(eg):
    from einsums_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(4)
    A, B = cu(rng.standard_normal((512, 300))), cu(rng.standard_normal((300, 512)))
    want = A.cpu().numpy() @ B.cpu().numpy()
    C = torch.zeros((512, 512), dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B)
    g.replay()
    torch.cuda.synchronize()
    assert np.allclose(C.cpu().numpy(), want, rtol=0, atol=1e-11)
    # a budget that leaves no scratch: the call still runs, and the library's other
    # allocations get back what the scratch held
    used = ctypes.c_size_t()
    _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
    try:
        run(eg, 0.0, "ij", C, 1.0, "ik", A, "kj", B)
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        _lib.check(lib.eg_set_memory_budget(used.value + (1 << 20)))
        p = ctypes.c_void_p()
        _lib.check(lib.eg_device_alloc(16 << 20, ctypes.byref(p)))  # fits only without the scratch
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        _lib.check(lib.eg_set_memory_budget(used.value + (1 << 20)))
        C.zero_()
        kernels = run(eg, 0.0, "ij", C, 1.0, "ik", A, "kj", B)
        assert "k_tc_split_gemm_f64" not in kernels and "k_contract_f64" in kernels
        assert np.allclose(C.cpu().numpy(), want, rtol=0, atol=1e-11)
        _lib.check(lib.eg_device_free(p))
    finally:
        _lib.check(lib.eg_set_memory_budget(0))


def test_streams_and_threads_share_the_scratch(eg):
    import threading
    rng = np.random.default_rng(6)
    sets = []
    for q in range(4):
        m, n, k = 500 + 13 * q, 520 - 7 * q, 256 + 31 * q
        A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
        sets.append((cu(A), cu(B), [torch.zeros((m, n), dtype=torch.float64, device="cuda") for _ in range(8)], A @ B))
    torch.cuda.synchronize()
    fails = []

    def work(q, stream):
        try:
            A, B, Cs, _ = sets[q]
            for C in Cs:
                eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B, stream=stream)
        except Exception as e:  # noqa: BLE001
            fails.append(e)

    streams = [torch.cuda.Stream(), torch.cuda.Stream(), None, None]  # two on the default stream
    ts = [threading.Thread(target=work, args=(q, streams[q])) for q in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    torch.cuda.synchronize()
    assert not fails
    for A, B, Cs, want in sets:
        for C in Cs:
            assert np.allclose(C.cpu().numpy(), want, rtol=0, atol=1e-11)


def launches():
    from einsums_gb300 import _lib
    n = ctypes.c_uint64()
    _lib.check(_lib.load().eg_kernel_launches(ctypes.byref(n)))
    return n.value


@pytest.mark.parametrize("pattern", [("ab", "ija", "ijb"), ("zab", "zai", "zbi")])
def test_lists(eg, pattern):
    """A list long enough for the tensor cores (three kernels a replay): items of one and of several
    tiles, hard items among them, replays on changed inputs and on two streams; the FMA plan under a
    memory budget."""
    from einsums_gb300 import _lib
    Cl, Al, Bl = pattern
    rng = np.random.default_rng(len(Cl))
    As, Bs = [], []
    for q in range(300):
        d = dict(i=int(rng.integers(9, 33)), j=int(rng.integers(9, 33)), a=int(rng.integers(40, 130)),
                 b=int(rng.integers(40, 130)), z=1 + q % 2)
        if q == 0:
            d = dict(i=32, j=34, a=300, b=7, z=3)
        As.append(rng.standard_normal([d[c] for c in Al]))
        Bs.append(rng.standard_normal([d[c] for c in Bl]))
    if Cl == "ab":  # graded against each other over the summed indices, an infinity, a row of zeros
        g = 10.0 ** np.linspace(-9, 9, As[5].shape[0])[:, None, None]
        As[5], Bs[5] = As[5] * g, Bs[5] / g
        As[6][0, 0, 3] = np.inf
        Bs[7][:, :, 2] = 0.0
    tA, tB = [cu(x) for x in As], [cu(x) for x in Bs]
    want = lambda k: np.einsum(f"{Al},{Bl}->{Cl}", As[k], Bs[k])
    scale = lambda k: np.einsum(f"{Al},{Bl}->{Cl}", np.abs(As[k]), np.abs(Bs[k]))

    def check(tC, factor=1.0):
        for k in range(len(As)):
            K = As[k].size // tC[k].shape[-2] // (As[k].shape[0] if Cl == "zab" else 1)
            with np.errstate(invalid="ignore"):
                w, s, got = want(k) * factor, scale(k), tC[k].cpu().numpy()
                off = np.abs(got - w)
            fin = np.isfinite(s)
            assert np.all(off[fin] <= 2 * (K + 4) * U * s[fin] * abs(factor)), k
            assert np.array_equal(np.isfinite(got), np.isfinite(w)), k

    empty = lambda: [torch.full(want(k).shape, float("nan"), dtype=torch.float64, device="cuda") for k in range(len(As))]
    tC = empty()
    plan = eg.GroupedPlan(0.0, Cl, tC, 1.0, Al, tA, Bl, tB)
    n = launches()
    plan.execute()
    assert launches() - n == 3
    torch.cuda.synchronize()
    check(tC)
    for t in tA:
        t.mul_(-2.0)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):  # each replay writes all of C; they share the plan's scratch
        plan.execute(stream=s1)
        plan.execute(stream=s2)
    torch.cuda.synchronize()
    check(tC, -2.0)
    plan.close()
    for t in tA:
        t.mul_(-0.5)
    used = ctypes.c_size_t()
    _lib.check(_lib.load().eg_memory_in_use(ctypes.byref(used)))
    try:
        _lib.check(_lib.load().eg_set_memory_budget(used.value + (64 << 20)))
        tC = empty()
        plan = eg.GroupedPlan(0.0, Cl, tC, 1.0, Al, tA, Bl, tB)
        n = launches()
        plan.execute()
        assert launches() - n == 1
        torch.cuda.synchronize()
        check(tC)
        plan.close()
    finally:
        _lib.check(_lib.load().eg_set_memory_budget(0))
