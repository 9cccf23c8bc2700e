"""Complex FP64 contractions as one real contraction: against NumPy and against the four
real contractions (which a captured call still runs), over the orders and strides of both
operands, conjugations, prefactors, batches and tile edges.  A part of the result sums 2 K
products, exact in 64 bits up to 2 K + 8 roundings of at most 2^-53 of the magnitudes."""
import ctypes

import numpy as np
import pytest

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


def launches(f):
    from einsums_gb300 import _lib
    lib = _lib.load()
    lib.eg_profile_enable(1)
    lib.eg_profile_reset()
    try:
        f()
        torch.cuda.synchronize()
        buf = ctypes.create_string_buffer(1 << 16)
        _lib.check(lib.eg_profile_summary(buf, len(buf)))
    finally:
        lib.eg_profile_enable(0)
    return {l.split(",")[0]: int(l.split(",")[1]) for l in buf.value.decode().strip().split("\n") if l}


def rand(rng, dims, labels, wide):
    """A complex tensor with the labels' extents; `wide`: a view with gaps along every index."""
    shape = [dims[l] for l in labels]
    big = [2 * n + 1 for n in shape] if wide else shape
    x = rng.standard_normal(big) + 1j * rng.standard_normal(big)
    t = torch.tensor(x, device="cuda")
    return (t[tuple(slice(1, None, 2) for _ in shape)] if wide else t)


CASES = [("ij", "ik", "kj"), ("ij", "ki", "kj"), ("ji", "ik", "jk"), ("ij", "ki", "jk"),
         ("bij", "bik", "bkj"), ("iajb", "klia", "jkbl"), ("ij", "iak", "kja")]
DIMS = [dict(i=1, j=1, k=3, l=1, a=2, b=1), dict(i=9, j=5, k=7, l=2, a=3, b=4),
        dict(i=33, j=31, k=65, l=2, a=2, b=3), dict(i=40, j=64, k=16, l=3, a=2, b=2)]


@pytest.mark.parametrize("Cl,Al,Bl", CASES)
@pytest.mark.parametrize("dims", DIMS, ids=lambda d: str(d["i"]))
@pytest.mark.parametrize("conj", [(False, False), (True, False), (False, True), (True, True)])
def test_one_contraction(eg, Cl, Al, Bl, dims, conj):
    rng = np.random.default_rng(dims["i"] + 2 * conj[0] + conj[1])
    K = int(np.prod([dims[l] for l in set(Al) & set(Bl) - set(Cl)]))
    for wide in (False, True):
        A, B, C0 = (rand(rng, dims, l, wide) for l in (Al, Bl, Cl))
        a, b, c = A.cpu().numpy(), B.cpu().numpy(), C0.cpu().numpy()
        ax, bx = a.conj() if conj[0] else a, b.conj() if conj[1] else b
        spec = f"{Al},{Bl}->{Cl}"
        for cp, ab in [(0.0, 1.0), (0.5, -2.0), (1.0 - 0.5j, 1.0)]:
            want = cp * c + ab * np.einsum(spec, ax, bx)
            mag = abs(cp) * np.abs(c) + abs(ab) * np.einsum(spec, np.abs(a), np.abs(b))
            bound = 2 * EPS * (2 * K + 8) * mag
            C = C0.clone() if not wide else rand(rng, dims, Cl, True)
            C.copy_(C0)
            run = lambda: eg.einsum(cp, Cl, C, ab, Al, A, Bl, B, conj_A=conj[0], conj_B=conj[1])
            seen = launches(run)
            if dims["i"] > 1:
                assert seen.get("k_complex_blocks") == 1 and seen.get("k_contract_f64") == 1, seen
            got = C.cpu().numpy()
            assert np.all(np.abs(got.real - want.real) <= bound) and np.all(np.abs(got.imag - want.imag) <= bound)
            if dims["i"] == 1:  # products by vectors need scratch of their own: refused under capture as before
                continue
            C.copy_(C0)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                run()
            graph.replay()
            four = C.cpu().numpy()
            assert np.all(np.abs(four - got) <= 2 * bound)


@pytest.mark.parametrize("Cl,Al,Bl", [("ij", "ik", "kj"), ("ji", "ki", "jk"), ("bij", "bik", "bkj")])
@pytest.mark.parametrize("i,j,k", [(300, 170, 257), (129, 400, 300), (640, 640, 130)])
def test_on_the_tensor_cores(eg, Cl, Al, Bl, i, j, k):
    """Above the FMA kernel's sizes: no more than four roundings' worth of the magnitudes a part."""
    rng = np.random.default_rng(i + j)
    dims = dict(i=i, j=j, k=k, b=2)
    A, B, C = (rand(rng, dims, l, False) for l in (Al, Bl, Cl))
    a, b, c = A.cpu().numpy().conj(), B.cpu().numpy(), C.cpu().numpy()
    spec = f"{Al},{Bl}->{Cl}"
    want = 0.5 * c - 2.0 * np.einsum(spec, a, b, optimize=True)
    mag = 0.5 * np.abs(c) + 2.0 * np.einsum(spec, np.abs(a), np.abs(b), optimize=True)
    seen = launches(lambda: eg.einsum(0.5, Cl, C, -2.0, Al, A, Bl, B, conj_A=True))
    assert seen.get("k_tc_split_gemm_f64") == 1 and seen.get("k_complex_blocks") == 1, seen
    got = C.cpu().numpy()
    # numpy's own sums of 2 K products may be as far off as theirs
    bound = EPS * (8 + 2 * k + 8) * mag
    assert np.all(np.abs(got.real - want.real) <= bound) and np.all(np.abs(got.imag - want.imag) <= bound)
