"""The condition under which the tensor-core NTT passes may pack two counts in one
word: no twiddle's bit matrix has a row of ones alone.  Row n of the matrix of t is
the 128 top bits of t x^(127 - n) x^k, so the elements with such a row are those
whose multiple by some x^o, o < 128, has only ones for its first 128 top bits.
Restated over Python integers for every layer of every size."""
import numpy as np
import pytest

MASK = (1 << 128) - 1


def mul_x(a):
    return ((a << 1) & MASK) ^ (0x87 if a >> 127 else 0)


def div_x(a):
    return (((a ^ 0x87) >> 1) | 1 << 127) if a & 1 else a >> 1


def mul(a, b):
    r = 0
    while b:
        if b & 1:
            r ^= a
        a, b = mul_x(a), b >> 1
    return r


def inv(a):
    r0, r1, t0, t1 = (1 << 128) | 0x87, a, 0, 1
    while r1 != 1:
        d = r0.bit_length() - r1.bit_length()
        if d < 0:
            r0, r1, t0, t1 = r1, r0, t1, t0
            continue
        r0, t0 = r0 ^ (r1 << d), t0 ^ (t1 << d)
    while t1 >> 128:  # below x^128
        d = t1.bit_length() - 129
        t1 ^= ((1 << 128) | 0x87) << d
    return t1


def layer_bases(dim):
    """Values whose sums are the twiddles of layer l, l = 0..dim-1 (the subspace
    polynomials' normalised values on the standard basis)."""
    rows = [[1 << i for i in range(dim)]]
    for _ in range(1, dim):
        p = rows[-1]
        rows.append([mul(v, v ^ p[0]) for v in p[1:]])
    rows = [[mul(v, i) for v in r] for r, i in ((r, inv(r[0])) for r in rows)]
    return [rows[dim - l - 1][1:1 + l] for l in range(dim)]


def ones_element():
    """The element whose first 128 top bits are ones: bits 127..7 are the first 121."""
    found = []
    for low in range(128):
        c = (MASK >> 7 << 7) | low
        t, ok = c, True
        for _ in range(128):
            ok = ok and t >> 127 == 1
            t = mul_x(t)
        if ok:
            found.append(c)
    assert len(found) == 1
    return found[0]


def in_span(basis, v):
    pivots = {}
    for b in basis:
        while b and b.bit_length() in pivots:
            b ^= pivots[b.bit_length()]
        if b:
            pivots[b.bit_length()] = b
    while v and v.bit_length() in pivots:
        v ^= pivots[v.bit_length()]
    return v == 0


def test_no_twiddle_of_any_size_has_a_row_of_ones():
    bad, t = [], ones_element()
    for _ in range(128):
        bad.append(t)
        t = div_x(t)
    for dim in range(2, 31):
        for basis in layer_bases(dim):
            assert not any(in_span(basis, v) for v in bad), dim


def test_the_bases_give_the_oracles_twiddles(oracle):
    dim = 7
    tw = np.zeros((1 << dim, 2), np.uint64)
    oracle.L.flockref_ntt_twiddles(dim, tw.ctypes.data)
    for layer, basis in enumerate(layer_bases(dim)):
        for blk in range(1 << len(basis)):
            v = 0
            for j, b in enumerate(basis):
                v ^= b if blk >> j & 1 else 0
            lo, hi = tw[(1 << layer) - 1 + blk]
            assert v == int(lo) | int(hi) << 64


@pytest.mark.parametrize("log_d", range(3, 31))
def test_every_size_has_tensor_passes(log_d):
    import flockgpu
    assert any("/mma" in d for d in flockgpu.ntt_plan_descs(log_d - 1, 64, 1))
