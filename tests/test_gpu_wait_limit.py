"""Kernels with bounded waits that wait for what was never started: the waits run
out, the kernels return, and the call that launched them reports it."""
import subprocess
import sys
from pathlib import Path

import numpy as np
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


def test_error_belongs_to_its_context(gpu_ctx, oracle):
    """The call that failed reports it once: other contexts are right meanwhile, the same one afterwards."""
    import flockgpu
    msg = np.random.default_rng(1).integers(0, 2**64, 2 * (64 << 5), dtype=np.uint64)
    plan = [i for i, d in enumerate(flockgpu.ntt_plan_descs(5, 64, 1)) if "/mma" in d][0]
    want = oracle.rs_encode(msg, 32, 64, 1)
    ctx = flockgpu.Context(0)
    try:
        ctx.set_wait_polls(0)
        with pytest.raises(flockgpu.FlockError, match="wait ran out"):
            ctx.ntt_rs_encode_plan(msg, 5, 64, 1, plan)
        with pytest.raises(flockgpu.FlockError, match="wait ran out"):
            ctx.bench_ntt_plan(5, 64, 1, plan, 1)
        assert np.array_equal(gpu_ctx.ntt_rs_encode_plan(msg, 5, 64, 1, plan), want)
        ctx.set_wait_polls(1 << 18)
        assert np.array_equal(ctx.ntt_rs_encode_plan(msg, 5, 64, 1, plan), want)
    finally:
        ctx.close()


def test_error_belongs_to_its_setup(gpu_ctx):
    import flockgpu
    p, q = flockgpu.Prover(gpu_ctx, 8), flockgpu.Prover(gpu_ctx, 8)
    want = p.prove_seed(5)
    p.set_wait_polls(0)
    with pytest.raises(flockgpu.FlockError, match="wait ran out"):
        p.prove_seed(5)
    assert q.prove_seed(5) == want
    p.set_wait_polls(1 << 18)
    assert p.prove_seed(5) == want
    p.close()
    q.close()


def test_tuner_keeps_no_plan_that_gave_up(gpu_ctx):
    import flockgpu
    ctx = flockgpu.Context(0)
    try:
        ctx.set_wait_polls(0)
        with pytest.raises(flockgpu.FlockError, match="wait ran out"):
            ctx.ntt_autotune(11, 128, 1)
        ctx.set_wait_polls(1 << 18)
        ms, desc = ctx.ntt_autotune(11, 128, 1)
        assert ms > 0 and "/mma" in desc  # timed now: -1 for a plan that was kept
    finally:
        ctx.close()


def test_batched_commit_gives_up(gpu_ctx):
    """Tensor passes of several jobs in one launch (2^10 and 2^11), and a job of other passes (2^8)."""
    import flockgpu
    jobs = [(10, 3), (8, 4), (11, 5)]
    ctx = flockgpu.Context(0)
    try:
        ctx.set_wait_polls(0)
        with pytest.raises(flockgpu.FlockError):
            ctx.prove_batch(jobs, threads=2)
        ctx.set_wait_polls(1 << 18)
        got = [r["bytes"] for r in ctx.prove_batch(jobs, threads=2)]
        for (log2, seed), proof in zip(jobs, got):
            p = flockgpu.Prover(gpu_ctx, log2)
            assert p.prove_seed(seed) == proof
            p.close()
    finally:
        ctx.close()
