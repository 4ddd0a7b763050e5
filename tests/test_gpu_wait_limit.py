"""Kernels with bounded waits that wait for what was never started: the waits run
out, the kernels return, and the call that launched them reports it."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
PKG = Path(__file__).resolve().parents[1] / "flock-challenge-multi_b200"


# a process of its own for each kernel; prints what the call raised
def _child(code: str) -> str:
    code = f"import sys; sys.path.insert(0, {str(PKG)!r})\nimport numpy as np\nimport flockgpu\n" + code
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return r.stdout


# one tile of fewest layers, several tiles a CTA in two passes, several 64-lane groups
@pytest.mark.parametrize("log_pos,lanes", [(2, 64), (12, 64), (6, 256)])
def test_ntt_pass_gives_up(log_pos, lanes):
    out = _child(f"""
ctx = flockgpu.Context(0)
msg = np.ones(2 * ({lanes} << {log_pos}), np.uint64)
plan = [i for i, d in enumerate(flockgpu.ntt_plan_descs({log_pos}, {lanes}, 1)) if "/mma" in d][0]
ctx.set_wait_polls(0)
try:
    ctx.ntt_rs_encode_plan(msg, {log_pos}, {lanes}, 1, plan)
    print("no error")
except flockgpu.FlockError as e:
    print(e)
""")
    assert "wait ran out" in out


def test_block_fold_gives_up():
    """A proof's kernels that wait outside its captured commitment: the lincheck's block fold."""
    out = _child("""
p = flockgpu.Prover(flockgpu.Context(0), 8)
p.set_wait_polls(0)
try:
    p.prove_seed(5)
    print("no error")
except flockgpu.FlockError as e:
    print(e)
""")
    assert "wait ran out" in out
