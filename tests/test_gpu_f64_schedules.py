"""The bits of an FP64 contraction on the tensor cores do not depend on how its tiles are scheduled:
CTA pairs or single CTAs, cut along K or whole, in panels or at once.  Rows graded so that many
regions lie near the line of the accuracy check."""
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [(256, 256, 4100), (600, 500, 700), (129, 1500, 2304), (2304, 2304, 300), (300, 77, 20000)]


def operands(m, n, k):
    rng = np.random.default_rng(m + n + k)
    # row r of A falls off over K at a rate of its own, against it the columns of B
    fall = np.exp(-rng.uniform(0, 3.2, (m, 1)) * np.arange(k) / k)
    rise = np.exp(-rng.uniform(0, 3.2, (n, 1)) * np.arange(k)[::-1] / k)
    return rng.standard_normal((m, k)) * fall, (rng.standard_normal((n, k)) * rise).T.copy()


def digests():
    import einsums_gb300 as eg
    for m, n, k in CASES:
        A, B = operands(m, n, k)
        C = torch.full((m, n), 0.5, dtype=torch.float64, device="cuda")
        eg.einsum(-1.0, "ij", C, 3.0, "ik", torch.from_numpy(A).cuda(), "kj", torch.from_numpy(B).cuda())
        print(m, n, k, hashlib.sha256(C.cpu().numpy().tobytes()).hexdigest())


def test_same_bits():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from einsums_gb300 import build
    build.build()
    here = os.path.dirname(os.path.abspath(__file__))
    path = os.pathsep.join([os.path.dirname(here), here, os.environ.get("PYTHONPATH", "")])
    outs = []
    for pairs in ("0", "1", ""):
        env = dict(os.environ, EINSUMS_GB300_TC_PAIRS=pairs, PYTHONPATH=path)
        r = subprocess.run([sys.executable, "-c", "import test_gpu_f64_schedules as t; t.digests()"], cwd=here, env=env,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        outs.append(r.stdout.split("\n"))
    assert len(outs[0]) == len(CASES) + 1
    assert outs[0] == outs[1] == outs[2]
