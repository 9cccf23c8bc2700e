"""No exception leaves the C entry points that allocate on the host or lock: each body that can throw
stands in a try block."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def body(path, start):
    text = open(os.path.join(ROOT, "einsums_gb300", "csrc", path)).read()
    at = re.search(start, text).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end], text[end:end + 10]


def test_try_blocks():
    inside, _ = body("complex.cu", r'extern "C" eg_status eg_einsum_complex\([^{]*\{')
    assert re.search(r"try \{\s*return einsum_complex\(", inside) and "catch" in inside
    _, after = body("batched.cu", r"eg_status run_plan\([^{]*try \{")
    assert after.strip().startswith("catch")
