"""What this framework's speed is measured on: contractions, permutes and Fock builds as a
quantum-chemistry program issues them, each through the public Python entry points.

The listed cases are the methods such a program runs, from the small matrix products of an
SCF iteration to the W intermediates of a coupled-cluster step with 160 virtual orbitals;
``draw`` gives more of the same methods over the sizes between.  Inputs are seeded and made
on the GPU with the distributions of ``einsums_gb300.workloads``.

``exact`` computes the same results with torch in 64 bits.  Its matrix products cut each
operand row into pieces short enough that every partial product sums without rounding, so
that what it returns is off by about one rounding, whatever the number of terms.
"""
import math

import torch

import einsums_gb300 as eg
from einsums_gb300 import workloads


def listed():
    return [
        # SCF: one of the many small products (orthogonalisation, density) of an iteration; latency
        {"name": "gemm_small", "kind": "gemm", "m": 40, "n": 60, "k": 50, "dtype": "float64"},
        # the same on complex orbitals (periodic or relativistic codes), A conjugated
        {"name": "gemm_complex", "kind": "gemm", "m": 300, "n": 170, "k": 257, "dtype": "complex128"},
        # particle-particle ladder of a small coupled-cluster iteration, FP64: an ordinary contraction
        {"name": "ladder", "kind": "ladder", "o": 12, "v": 48},
        # ring intermediate W_mbej in FP64: both operands' summed indices strided, the large FP64 case
        {"name": "ring", "kind": "ring", "o": 24, "v": 96},
        # the four quarter transformations of the two-electron integrals to the orbital basis, odd n
        {"name": "ao2mo", "kind": "ao2mo", "n": 75},
        # W intermediates and energy of a large coupled-cluster step on the split-BF16 form: the largest
        {"name": "ccd_split", "kind": "ccd", "o": 32, "v": 160, "slices": 5},
        # differentiated ring contraction: forward and both adjoints, split-BF16
        {"name": "ring_grad", "kind": "grad", "o": 24, "v": 96, "precision": "split_bf16"},
        # uneven small contractions of a pair-local method, one grouped plan, FP64
        {"name": "pairs", "kind": "pairs", "count": 512, "precision": "fp64"},
        # a larger batch of them on the split-BF16 form
        {"name": "pairs_split", "kind": "pairs", "count": 2048, "precision": "split_bf16"},
        # Fock build from integrals with 8-fold symmetry
        {"name": "fock_sym", "kind": "fock_sym", "n": 100},
        # Fock build for general integrals (Coulomb and exchange einsums) and the energy
        {"name": "fock", "kind": "fock", "n": 100},
        # MP2: amplitudes, antisymmetrised integrals (permutes), energy; memory-bound
        {"name": "mp2", "kind": "mp2", "o": 31, "v": 126},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "ladder", "ring", "ao2mo", "ccd", "grad", "pairs", "fock_sym", "fock", "mp2"])
    if kind == "gemm":
        if rng.random() < 0.5:
            return {"kind": kind, "m": _log(rng, 8, 200), "n": _log(rng, 8, 200), "k": _log(rng, 8, 200),
                    "dtype": "float64"}
        return {"kind": kind, "m": _log(rng, 24, 320), "n": _log(rng, 24, 320), "k": _log(rng, 24, 320),
                "dtype": "complex128"}
    if kind == "ladder":
        return {"kind": kind, "o": _log(rng, 4, 14), "v": _log(rng, 14, 60)}
    if kind == "ring":
        return {"kind": kind, "o": _log(rng, 6, 24), "v": _log(rng, 20, 96)}
    if kind == "ao2mo":
        return {"kind": kind, "n": rng.randint(18, 75)}
    if kind == "ccd":
        return {"kind": kind, "o": _log(rng, 8, 31), "v": _log(rng, 40, 158), "slices": rng.choice([4, 5])}
    if kind == "grad":
        return {"kind": kind, "o": _log(rng, 8, 24), "v": _log(rng, 30, 96), "precision": "split_bf16"}
    if kind == "pairs":
        return {"kind": kind, "count": _log(rng, 64, 2048), "precision": rng.choice(["fp64", "split_bf16"])}
    if kind == "mp2":
        return {"kind": kind, "o": _log(rng, 6, 32), "v": _log(rng, 20, 126)}
    return {"kind": kind, "n": rng.randint(24, 100)}


# ------------------------------------------------------------------ inputs --
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _normal(gen, *shape, dtype=torch.float64):
    return torch.randn(shape, generator=gen, dtype=dtype, device="cuda")


def _empty(*shape):
    return torch.empty(shape, dtype=torch.float64, device="cuda")



def _inputs(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    if kind == "gemm":
        dt = getattr(torch, case["dtype"])
        return {"A": _normal(gen, case["m"], case["k"], dtype=dt), "B": _normal(gen, case["k"], case["n"], dtype=dt)}
    if kind == "ladder":
        o, v = case["o"], case["v"]
        t = _normal(gen, o, o, v, v) * 0.01
        g = torch.rand((v, v, v, v), generator=gen, dtype=torch.float64, device="cuda") * 2.0 - 1.0
        return {"t": t, "g": g, "r": _normal(gen, o, o, v, v)}
    if kind in ("ring", "grad"):
        x = workloads.ccd_inputs(case["o"], case["v"], seed=seed, backend="cuda", with_vvvv=False)
        o, v = case["o"], case["v"]
        return {"t": x["t"], "g": x["g_oovv"], "w": x["g_ovvo"], "R": _normal(gen, o, v, v, o)}
    if kind == "ccd":
        x = workloads.ccd_inputs(case["o"], case["v"], seed=seed, backend="cuda")
        return {"t": x["t"], "g": x["g_oovv"], "mnij": x["g_oooo"], "abef": x["g_vvvv"], "mbej": x["g_ovvo"]}
    if kind in ("ao2mo", "fock", "fock_sym"):
        n = case["n"]
        g, D = workloads.fock_inputs(n, seed=seed, backend="cuda", nocc=max(1, n // 5))
        Q, _ = torch.linalg.qr(_normal(gen, n, n))
        H = _normal(gen, n, n)
        return {"g": g, "D": D, "Q": Q.contiguous(), "H": (H + H.T).contiguous()}
    if kind == "pairs":
        # the shapes are the case's own, the values the seed's
        shapes = workloads.batched_shapes(case["count"], seed=case["count"])
        flat = lambda sizes: _normal(gen, sum(sizes))
        A = flat([i * j * a for i, j, a, b in shapes])
        B = flat([i * j * b for i, j, a, b in shapes])
        return {"shapes": shapes, "A": A, "B": B}
    o, v = case["o"], case["v"]
    g = _normal(gen, o, v, o, v) * 0.1
    e_o = -torch.rand((o,), generator=gen, dtype=torch.float64, device="cuda") - 0.5
    e_v = torch.rand((v,), generator=gen, dtype=torch.float64, device="cuda") * 3.0 + 0.1
    scale = 1.0 / (e_o[:, None, None, None] + e_o[None, None, :, None]
                   - e_v[None, :, None, None] - e_v[None, None, None, :])
    return {"g": g, "scale": scale}


def _views(flat, sizes):
    out, off = [], 0
    for s in sizes:
        n = math.prod(s)
        out.append(flat[off:off + n].view(s))
        off += n
    return out


def prepare(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    st = dict(x, kind=kind, case=dict(case))
    if kind == "gemm":
        st["plan"] = eg.compile_plan("ij", "ik", "kj")
        st["C"] = torch.empty((case["m"], case["n"]), dtype=x["A"].dtype, device="cuda")
    elif kind == "ao2mo":
        n = case["n"]
        st["t1"], st["t2"], st["mo"] = _empty(n, n, n, n), _empty(n, n, n, n), _empty(n, n, n, n)
    elif kind == "ccd":
        st["E"] = _empty()
    elif kind == "grad":
        st["t"].requires_grad_(True)
        st["g"].requires_grad_(True)
    elif kind == "pairs":
        sh = x["shapes"]
        st["C"] = _empty(sum(a * b for i, j, a, b in sh))
        st["plan"] = eg.GroupedPlan(0.0, "ab", _views(st["C"], [(a, b) for i, j, a, b in sh]), 1.0, "ija",
                                    _views(x["A"], [(i, j, a) for i, j, a, b in sh]), "ijb",
                                    _views(x["B"], [(i, j, b) for i, j, a, b in sh]), precision=case["precision"])
    elif kind in ("fock", "fock_sym"):
        st["F"] = _empty(case["n"], case["n"])
        st["E"] = _empty()
    elif kind == "mp2":
        o, v = case["o"], case["v"]
        st["amps"], st["K"], st["T"] = _empty(o, v, o, v), _empty(o, o, v, v), _empty(v, v, o, o)
        st["L"], st["E"] = _empty(o, v, o, v), _empty()
    return st


# --------------------------------------------------------------------- run --
def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "gemm":
        if case["dtype"] == "float64":
            st["plan"].execute(0.0, st["C"], 1.0, st["A"], st["B"])
        else:
            eg.einsum(0.0, "ij", st["C"], 1.0, "ik", st["A"], "kj", st["B"], conj_A=True)
        return st["C"]
    if kind == "ladder":
        eg.einsum(1.0, "ijab", st["r"], 0.5, "ijef", st["t"], "efab", st["g"])
        return st["r"]
    if kind == "ring":
        eg.einsum(1.0, "mbej", st["w"], -0.5, "jnfb", st["t"], "mnef", st["g"])
        return st["w"]
    if kind == "ao2mo":
        t1, t2, mo, Q = st["t1"], st["t2"], st["mo"], st["Q"]
        eg.einsum(0.0, "pqrs", t1, 1.0, "mqrs", st["g"], "mp", Q)
        eg.einsum(0.0, "pqrs", t2, 1.0, "pmrs", t1, "mq", Q)
        eg.einsum(0.0, "pqrs", t1, 1.0, "pqms", t2, "mr", Q)
        eg.einsum(0.0, "pqrs", mo, 1.0, "pqrm", t1, "ms", Q)
        return mo
    if kind == "ccd":
        t, g, kw = st["t"], st["g"], {"precision": "split_bf16", "slices": case["slices"]}
        eg.einsum(1.0, "mnij", st["mnij"], 0.25, "ijef", t, "mnef", g, **kw)
        eg.einsum(1.0, "abef", st["abef"], 0.25, "mnef", g, "mnab", t, **kw)
        eg.einsum(1.0, "mbej", st["mbej"], -0.5, "jnfb", t, "mnef", g, **kw)
        eg.compile_plan("", "ijab", "ijab").execute(0.0, st["E"], 0.25, t, g)
        return {"mnij": st["mnij"], "abef": st["abef"], "mbej": st["mbej"], "E": st["E"]}
    if kind == "grad":
        t, g = st["t"], st["g"]
        t.grad = g.grad = None
        C = eg.einsum_ag("mbej", "jnfb", "mnef", t, g, precision=case["precision"])
        C.backward(st["R"])
        return {"C": C, "dt": t.grad, "dg": g.grad}
    if kind == "pairs":
        st["plan"].execute()
        return st["C"]
    if kind == "fock_sym":
        F = st["F"]
        F.copy_(st["H"])
        eg.fock_jk_symmetric(F, st["g"], st["D"])
        return F
    if kind == "fock":
        F, g, D, E = st["F"], st["g"], st["D"], st["E"]
        F.copy_(st["H"])
        eg.einsum(1.0, "pq", F, 2.0, "pqrs", g, "rs", D)
        eg.einsum(1.0, "pq", F, -1.0, "prqs", g, "rs", D)
        eg.compile_plan("", "pq", "pq").execute(0.0, E, 1.0, D, F)
        return {"F": F, "E": E}
    g, amps, L, E = st["g"], st["amps"], st["L"], st["E"]
    eg.einsum(0.0, "iajb", amps, 1.0, "iajb", g, "iajb", st["scale"])
    eg.permute(0.0, "iajb", L, 2.0, "iajb", g)
    eg.permute(1.0, "iajb", L, -1.0, "ibja", g)
    eg.permute(0.0, "ijab", st["K"], 1.0, "iajb", amps)
    eg.permute(0.0, "abij", st["T"], 1.0, "ijab", st["K"])
    eg.compile_plan("", "iajb", "iajb").execute(0.0, E, 1.0, amps, L)
    return {"L": L, "K": st["K"], "T": st["T"], "E": E}


# -------------------------------------------------------------------- work --
def work(case):
    kind = case["kind"]
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        z = case["dtype"] == "complex128"
        return {"bytes": (m * k + k * n + m * n) * (16 if z else 8), "flops": 2.0 * m * n * k * (4 if z else 1)}
    if kind == "ladder":
        o, v = case["o"], case["v"]
        return {"bytes": 8.0 * (3 * o * o * v * v + v ** 4), "flops": 2.0 * o * o * v ** 4}
    if kind == "ring":
        ov = case["o"] * case["v"]
        return {"bytes": 8.0 * 4 * ov * ov, "flops": 2.0 * ov ** 3}
    if kind == "grad":
        ov = case["o"] * case["v"]
        return {"bytes": 8.0 * 6 * ov * ov, "flops": 6.0 * ov ** 3}
    if kind == "ao2mo":
        n = case["n"]
        return {"bytes": 8.0 * (2 * n ** 4 + n * n), "flops": 8.0 * n ** 5}
    if kind == "ccd":
        o, v = case["o"], case["v"]
        ov = o * v
        return {"bytes": 8.0 * (2 * ov * ov + 2 * (o ** 4 + v ** 4 + ov * ov)),
                "flops": 2.0 * (o ** 4 * v * v + v ** 4 * o * o + ov ** 3 + ov * ov)}
    if kind == "pairs":
        sh = workloads.batched_shapes(case["count"], seed=case["count"])
        return {"bytes": 8.0 * sum(i * j * (a + b) + a * b for i, j, a, b in sh),
                "flops": 2.0 * sum(i * j * a * b for i, j, a, b in sh)}
    if kind == "fock_sym":
        n = case["n"]
        return {"bytes": n ** 4 + 24.0 * n * n, "flops": 1.5 * n ** 4}
    if kind == "fock":
        n = case["n"]
        return {"bytes": 8.0 * n ** 4 + 24.0 * n * n, "flops": 4.0 * n ** 4 + 2.0 * n * n}
    n = (case["o"] * case["v"]) ** 2
    return {"bytes": 8.0 * 5 * n, "flops": 6.0 * n}


# ------------------------------------------------------------------- exact --
def _pieces(X, bits):
    """The rows of X as three summands whose entries are whole multiples, of at most `bits` bits, of one power of two each."""
    mx = X.abs().amax(dim=1, keepdim=True)
    e = torch.where(mx > 0, torch.frexp(mx)[1], 0)
    out, rest = [], X
    for p in range(3):
        unit = torch.ldexp(torch.ones_like(mx), e - bits * (p + 1))
        q = torch.round(rest / unit) * unit
        out.append(q)
        rest = rest - q
    return out


def _mm(A, B):
    """A @ B for FP64 matrices with about one rounding per entry."""
    bits = (52 - max(1, math.ceil(math.log2(max(2, A.shape[1]))))) // 2
    a, b = _pieces(A, bits), _pieces(B.T.contiguous(), bits)
    out = None
    for i, j in ((2, 0), (1, 1), (0, 2), (1, 0), (0, 1), (0, 0)):
        out = a[i] @ b[j].T if out is None else out.addmm_(a[i], b[j].T)
    return out


def _sum2(terms):
    """The sum of a 1-D tensor with the roundings carried along (pairwise)."""
    s, c = terms, torch.zeros_like(terms)
    while s.numel() > 1:
        if s.numel() % 2:
            s, c = torch.cat([s, s.new_zeros(1)]), torch.cat([c, c.new_zeros(1)])
        a, b = s[0::2], s[1::2]
        t = a + b
        z = t - a
        c = c[0::2] + c[1::2] + ((a - (t - z)) + (b - z))
        s = t
    return (s + c).reshape(())


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "gemm":
        A, B = x["A"], x["B"]
        if case["dtype"] == "float64":
            return _mm(A, B)
        A = torch.conj(A).resolve_conj()
        re = _mm(torch.cat([A.real, -A.imag], 1), torch.cat([B.real, B.imag], 0))
        im = _mm(torch.cat([A.real, A.imag], 1), torch.cat([B.imag, B.real], 0))
        return torch.complex(re, im)
    if kind == "ladder":
        o, v = case["o"], case["v"]
        return x["r"] + 0.5 * _mm(x["t"].view(o * o, v * v), x["g"].view(v * v, v * v)).view(o, o, v, v)
    if kind in ("ring", "grad"):
        o, v = case["o"], case["v"]
        ov = o * v
        T = x["t"].permute(0, 3, 1, 2).reshape(ov, ov)   # (j b) x (n f)
        G = x["g"].permute(0, 2, 1, 3).reshape(ov, ov)   # (m e) x (n f)
        back = lambda P: P.view(o, v, o, v)
        P = back(_mm(G, T.T)).permute(0, 3, 1, 2)        # m e j b -> m b e j
        if kind == "ring":
            return x["w"] + (-0.5) * P
        R = x["R"].permute(0, 2, 3, 1).reshape(ov, ov)   # (m e) x (j b)
        dt = back(_mm(R.T, G)).permute(0, 2, 3, 1)       # j b n f -> j n f b
        dg = back(_mm(R, T)).permute(0, 2, 1, 3)         # m e n f -> m n e f
        return {"C": P.contiguous(), "dt": dt.contiguous(), "dg": dg.contiguous()}
    if kind == "ao2mo":
        n, Q, t = case["n"], x["Q"], x["g"]
        for d in range(4):
            t = torch.movedim(_mm(torch.movedim(t, d, 3).reshape(n ** 3, n), Q).view(n, n, n, n), 3, d)
        return t.contiguous()
    if kind == "ccd":
        o, v, t, g = case["o"], case["v"], x["t"], x["g"]
        ov = o * v
        E = 0.25 * _sum2((t * g).reshape(-1))
        mnij = x["mnij"] + 0.25 * _mm(g.view(o * o, v * v), t.view(o * o, v * v).T).view(o, o, o, o)
        T = t.permute(0, 3, 1, 2).reshape(ov, ov)
        G = g.permute(0, 2, 1, 3).reshape(ov, ov)
        mbej = x["mbej"] + (-0.5) * _mm(G, T.T).view(o, v, o, v).permute(0, 3, 1, 2)
        abef = x["abef"]
        tt, gg = t.view(o * o, v * v).T.contiguous(), g.view(o * o, v * v)
        out = abef.view(v * v, v * v)
        for r in range(0, v * v, 4096):
            out[r:r + 4096] += 0.25 * _mm(tt[r:r + 4096], gg)
        return {"mnij": mnij, "abef": abef, "mbej": mbej, "E": E}
    if kind == "pairs":
        sh = x["shapes"]
        As = _views(x["A"], [(i * j, a) for i, j, a, b in sh])
        Bs = _views(x["B"], [(i * j, b) for i, j, a, b in sh])
        return torch.cat([_mm(A.T.contiguous(), B).reshape(-1) for A, B in zip(As, Bs)])
    if kind in ("fock", "fock_sym"):
        n, g, D, H = case["n"], x["g"], x["D"], x["H"]
        d = D.reshape(n * n, 1)
        J = _mm(g.view(n * n, n * n), d).view(n, n)
        K = _mm(g.permute(0, 2, 1, 3).reshape(n * n, n * n), d).view(n, n)
        F = H + 2.0 * J - K
        return F if kind == "fock_sym" else {"F": F, "E": _sum2((D * F).reshape(-1))}
    g, amps = x["g"], x["g"] * x["scale"]
    L = 2.0 * g - g.permute(0, 3, 2, 1)
    return {"L": L, "K": amps.permute(0, 2, 1, 3).contiguous(), "T": amps.permute(1, 3, 0, 2).contiguous(),
            "E": _sum2((amps * L).reshape(-1))}
