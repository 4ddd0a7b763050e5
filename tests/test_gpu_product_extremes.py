"""The integer carry-less products at the fullest operands: every 32-bit word
zero, all ones or one or two whole bit classes, where the class sums are the
largest a 4-bit field can hold, against the oracle."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WORDS = np.array([0, 0xFFFFFFFF, 0x11111111, 0x22222222, 0x44444444, 0x88888888, 0x33333333, 0xCCCCCCCC], np.uint32)


def _values(rng, n):
    return WORDS[rng.integers(0, WORDS.size, (n, 4))].view(np.uint64).reshape(-1)


def test_products(gpu_ctx, oracle):
    low = np.zeros((WORDS.size**2, 2, 4), np.uint32)
    for k, (x, y) in enumerate(itertools.product(WORDS, WORDS)):
        low[k, 0, 0], low[k, 1, 0] = x, y
    rng = np.random.default_rng(3)
    a = np.concatenate([low[:, 0].copy().view(np.uint64).reshape(-1), _values(rng, 4096)])
    b = np.concatenate([low[:, 1].copy().view(np.uint64).reshape(-1), _values(rng, 4096)])
    assert np.array_equal(gpu_ctx.f128_mul(a, b), oracle.f128_mul(a, b))


@pytest.mark.parametrize("rho", [(0xFFFFFFFF, 0), (2**64 - 1, 0), (0, 2**64 - 1), (0x1111111133333333, 0x88888888CCCCCCCC)])
def test_fold_by_prepared_factor(gpu_ctx, oracle, rho):
    rng = np.random.default_rng(4)
    a, b, e = _values(rng, 256), _values(rng, 256), _values(rng, 64)
    _, fa, fb = gpu_ctx.sumcheck_round3(e, a, b, rho)
    for x, got in ((a, fa), (b, fb)):
        x0, x1 = x.reshape(-1, 2)[0::2].reshape(-1), x.reshape(-1, 2)[1::2].reshape(-1)
        r = np.tile(np.array(rho, np.uint64), x0.size // 2)
        assert np.array_equal(got, x0 ^ oracle.f128_mul(r, x0 ^ x1))
