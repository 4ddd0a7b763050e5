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


# one step and less, a step's remainders on both sides, CTAs that start mid-column
# and span columns (few SMs), a single column, the narrowest and widest blocks
@pytest.mark.parametrize("n,k_log", [(1, 14), (8, 15), (63, 14), (64, 14), (65, 16), (1000, 14), (1000, 8), (65, 17),
                                     (4097, 9)])
@pytest.mark.parametrize("sms", [1, 3, 148])
def test_block_fold(gpu_ctx, n, k_log, sms):
    rng = np.random.default_rng(n + k_log)
    z = rng.integers(0, 2**64, (n, 1 << (k_log - 6)), dtype=np.uint64)
    eq = rng.integers(0, 2**64, (n, 2), dtype=np.uint64)
    want = np.zeros((1 << k_log, 2), np.uint64)
    for o in range(n):
        bits = np.unpackbits(z[o].view(np.uint8), bitorder="little").astype(bool)
        want[bits] ^= eq[o]
    assert np.array_equal(gpu_ctx.lincheck_fold(z, eq, k_log, sms), want)


def test_block_fold_refuses_more_steps_than_it_counts(gpu_ctx):
    """2^29 blocks of 2^17 bits: 2^32 steps (refused before a byte is read)."""
    word = np.zeros(2, np.uint64)
    p = word.ctypes.data
    for n, k_log in ((1 << 29, 17), (1 << 30, 8), (1, 7), (1, 18)):
        assert gpu_ctx.lib.flock_lincheck_fold(gpu_ctx.h, p, p, n, k_log, 1, p) == 1
