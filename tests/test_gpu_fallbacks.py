"""GPU parity of the kernels that only an environment variable selects.

Each variable is read once per process by the library, so every alternative runs in a child process
(tests/fallback_worker.py) that checks its cases against the oracle.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
WORKER = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fallback_worker.py")


@pytest.mark.parametrize("what,var,value", [
    ("streamed", "FB200_GEMM16_STREAMED", "1"),
    ("exact_small", "FB200_EXACT_SMALL_BATCH", "1"),
    ("decode_scalar", "FB200_ATTN_DECODE_TC", "0"),
    ("prefill_mma", "FB200_ATTN_TCGEN05", "0"),
    ("prefill_sequential", "FB200_TC_GROUP", "0"),
    ("prefill_chunks", "FB200_TCGEN05", "0"),
    ("q5k_row_copies", "FB200_Q5K_TENSOR_TMA", "0"),
])
def test_alternative_kernel(what, var, value):
    out = subprocess.run([sys.executable, WORKER, what], env=dict(os.environ, **{var: value}),
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout[-2000:] + out.stderr[-4000:]
    assert f"done {what}" in out.stdout


@pytest.mark.parametrize("tcgen05,expected", [("1", {"q_mat_mul (> 32 rows)": 4, "rms_norm + q_mat_mul": 3}),
                                              ("0", {"q_mat_mul (> 32 rows)": 12, "rms_norm + q_mat_mul": 1})])
def test_trace_lines_of_a_prompt(tcgen05, expected):
    # a line per product that ran. Two layers: q, k and v go out side by side without a line and gate / up runs under its norm, or
    # (without the tcgen05 kernels) all six products of a layer one after the other; the head takes one row under its norm
    out = subprocess.run([sys.executable, WORKER, "trace"], env=dict(os.environ, FB200_TCGEN05=tcgen05, FB200_TRACE="1"),
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout[-2000:] + out.stderr[-4000:]
    names = [line.split("fb200 trace: ")[1][:26].rstrip() for line in out.stderr.splitlines() if line.startswith("fb200 trace: ")]
    assert {n: names.count(n) for n in expected} == expected, names
