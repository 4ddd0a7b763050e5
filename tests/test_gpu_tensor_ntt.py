"""The tensor-core NTT passes at the edges of their tiles and operands, and the
witness kernels on both sides of their split, against the oracle or each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mma_plans(log_pos, lanes, rate):
    import flockgpu
    descs = flockgpu.ntt_plan_descs(log_pos, lanes, rate)
    return [i for i, d in enumerate(descs) if "/mma" in d]


# fewest layers a pass takes, one and two passes, several 64-lane groups, a
# rate whose first pass starts below layer 1, more tiles than one wave of CTAs
@pytest.mark.parametrize("lanes,log_pos,rate", [(64, 2, 1), (64, 3, 1), (64, 5, 1), (64, 6, 1), (128, 4, 1),
                                                (256, 3, 2), (64, 7, 3), (64, 14, 1)])
def test_tensor_passes(gpu_ctx, oracle, lanes, log_pos, rate):
    plans = _mma_plans(log_pos, lanes, rate)
    assert plans
    msg = np.random.default_rng(log_pos * 100 + lanes).integers(0, 2**64, 2 * (lanes << log_pos), dtype=np.uint64)
    want = oracle.rs_encode(msg, 1 << log_pos, lanes, rate)
    for k in plans:
        assert np.array_equal(gpu_ctx.ntt_rs_encode_plan(msg, log_pos, lanes, rate, k), want), f"plan {k}"


@pytest.mark.parametrize("fill", ["zeros", "ones", "one_bit"])
def test_tensor_passes_extreme_values(gpu_ctx, oracle, fill):
    """All-ones values give the largest counts of the packed parities."""
    lanes, log_pos, rate = 64, 8, 1
    msg = np.zeros(2 * (lanes << log_pos), np.uint64)
    if fill == "ones":
        msg[:] = np.uint64(2**64 - 1)
    elif fill == "one_bit":
        i = np.arange(msg.size // 2)
        msg[2 * i + (i % 128) // 64] = np.uint64(1) << (i % 64).astype(np.uint64)
    want = oracle.rs_encode(msg, 1 << log_pos, lanes, rate)
    for k in _mma_plans(log_pos, lanes, rate):
        assert np.array_equal(gpu_ctx.ntt_rs_encode_plan(msg, log_pos, lanes, rate, k), want)


@pytest.mark.parametrize("log2", [9, 15, 16])
def test_witness_split(gpu_ctx, log2):
    """Four writers per compression up to 2^15 slots, one beyond: the seeded and
    the two host-input kernels prove the same bytes on both sides."""
    import flockgpu
    blocks = flockgpu.generate_compressions(log2, 77)
    p = flockgpu.Prover(gpu_ctx, log2)
    want = p.prove_seed(77)
    assert p.prove_blocks(blocks) == want
    assert p.prove_compressions(flockgpu.to_records(blocks)) == want
    assert p.verify(want) == ""
    p.close()
