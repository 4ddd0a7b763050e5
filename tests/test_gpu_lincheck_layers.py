"""The lincheck's kernels by themselves, against numpy over the oracle's matrices
and field product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ALPHA, BETA = (0x0123456789ABCDEF, 0xFEDCBA9876543210), (0x1111, 0x2222)


@pytest.mark.parametrize("sms", [1, 5, 132, 148])
def test_column_combination_on_some_sms(gpu_ctx, oracle, sms):
    """SHA-256 (four parts of the table): the values, and no more CTAs than the SMs asked for
    (the parts are at least one CTA each)."""
    rng = np.random.default_rng(2)
    e = rng.integers(0, 2**64, (1 << 15, 2), dtype=np.uint64)
    sums = []
    for which in (0, 1):
        ptr, col = oracle.sha256_matrix(which)
        rows = np.repeat(np.arange(1 << 15), np.diff(ptr.astype(np.int64)))
        t = np.zeros((1 << 15, 2), np.uint64)
        np.bitwise_xor.at(t, col, e[rows])
        sums.append(t)
    al = np.tile(np.array(ALPHA, np.uint64), 1 << 15)
    want = oracle.f128_mul(al, sums[0].reshape(-1)).reshape(-1, 2) ^ sums[1]
    got, ctas = gpu_ctx.lincheck_comb("sha256", e, ALPHA, BETA, sms)
    diff = np.flatnonzero((got ^ want).any(axis=1))
    assert diff.size == 1 and tuple(got[diff[0]] ^ want[diff[0]]) == BETA  # the constant column
    assert ctas <= max(sms, 4)


def test_column_combination_is_the_same_on_any_sms(gpu_ctx):
    """BLAKE3 (two parts): 15 million row indices a column set, by the SMs that take them."""
    e = np.random.default_rng(3).integers(0, 2**64, (1 << 14, 2), dtype=np.uint64)
    want, _ = gpu_ctx.lincheck_comb("blake3", e, ALPHA, BETA, 148)
    for sms in (1, 7, 132):
        got, ctas = gpu_ctx.lincheck_comb("blake3", e, ALPHA, BETA, sms)
        assert np.array_equal(got, want) and ctas <= max(sms, 2)
