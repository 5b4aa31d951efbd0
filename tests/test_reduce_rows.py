"""The row-wise reduction (csrc/reduce.cuh) restated with integers, against exact arithmetic: the
quotient taken from the top word sums before any carry, the single signed-carry pass, its int64
bounds, and rows cut into segments that start without a carry."""
import random

import pytest

M32, M64 = (1 << 32) - 1, (1 << 64) - 1


def signed_shift(z):
    assert -(1 << 63) <= z < 1 << 63  # int64 in the kernel
    return z & M32, z >> 32


def row_quotient(d, k, r_words, q, limbs):
    """Barrett quotient from words ws-2 .. ws+4, without the carry of the words below."""
    top_shift = q.bit_length() - 64
    ws, offset = top_shift // 32, top_shift % 32
    acc, z = 0, []
    for j in range(-2, 5):
        w = ws + j
        if 0 <= w < limbs + 2:
            acc += d[w] + k * r_words[w]
        if j >= 0:
            z.append(acc & M32)
        acc >>= 32
    window = sum(x << (32 * i) for i, x in enumerate(z)) >> offset
    tl, th = window & M64, (window >> 64) & M64
    q_top = q >> top_shift if top_shift >= 0 else q << -top_shift
    mu_low = ((1 << 128) - 1) // (q_top + 1) - (1 << 64) if q_top != M64 else 0
    return th + ((th * mu_low + ((tl * mu_low) >> 64) + tl) >> 64)


def row_pass(d, k, r_words, q_words, quotient, first, last, carry=0):
    low, high = quotient & M32, quotient >> 32
    q_below = q_words[first - 1] if first else 0
    below = (low * q_below >> 32) + high * q_below
    out = []
    for w in range(first, last):
        a = low * q_words[w]
        y = d[w] + k * r_words[w] - (a & M32) - below
        below = (a >> 32) + high * q_words[w]
        o, carry = signed_shift(y + carry)
        out.append(o)
    return out, carry


@pytest.mark.parametrize("limbs,q_bits", [(1, 2), (1, 20), (1, 32), (2, 33), (2, 63), (2, 64), (3, 65), (3, 40), (5, 160),
                                          (16, 481), (40, 1280), (40, 700)])
def test_quotient_before_carries_leaves_at_most_three_corrections(limbs, q_bits):
    rng = random.Random(limbs * 1000 + q_bits)
    for trial in range(300):
        q = rng.getrandbits(q_bits) | 1 << (q_bits - 1) if trial % 3 else (1 << q_bits) - 1 - trial % 2
        q = max(q, 2)
        k = rng.choice([0, 1, 7272, rng.randrange(7273)])
        r = rng.randrange(q)
        r_words = [(r >> (32 * w)) & M32 for w in range(limbs + 16)]
        q_words = [(q >> (32 * w)) & M32 for w in range(limbs + 16)]
        t = rng.randrange(q << 46)  # T < 2^47 q, in a carry-save form with word sums below 2^56
        if trial % 4 == 0:
            t = min(t, (1 << (32 * (limbs + 2))) - 1)
        d, rest = [], t
        for w in range(limbs + 2):
            x = rest >> (32 * w)
            extra = min(x >> 32, rng.choice([0, (1 << 24) - 1, rng.randrange(1 << 24)])) if w + 1 < limbs + 2 else 0
            digit = (x & M32) + (extra << 32)
            d.append(digit)
            rest -= digit << (32 * w)
        assert rest == 0 and all(0 <= x < 1 << 56 for x in d)
        tp = t + k * r
        quotient = row_quotient(d, k, r_words, q, limbs)
        assert quotient >> 48 == 0 and quotient <= tp // q <= quotient + 3
        out, carry = row_pass(d, k, r_words, q_words, quotient, 0, limbs + 2)
        assert carry == 0 and sum(o << (32 * w) for w, o in enumerate(out)) == tp - quotient * q
        # the same row in segments: partial words, then each segment's carry into the next
        for span in (1, 2, 3, 16):
            total = sum(
                (sum(o << (32 * (at + i)) for i, o in enumerate(words)) + (c << (32 * min(at + span, limbs + 2))))
                for at in range(0, limbs + 2, span)
                for words, c in [row_pass(d, k, r_words, q_words, quotient, at, min(at + span, limbs + 2))])
            assert total == tp - quotient * q
