"""A float32 number as three bfloat16 numbers (csrc/f32_pieces.cuh: split), restated in numpy: what is exact, what the products leave out."""

import numpy as np


def bfloat16_down(x):
    return (x.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)


def bfloat16_nearest(x):
    bits = x.view(np.uint32)
    return ((bits + np.uint32(0x7FFF) + ((bits >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)).view(np.float32)


def pieces(x):
    first = bfloat16_down(x)
    rest = x - first
    second = bfloat16_nearest(rest)
    return first, second, bfloat16_down(rest - second)


def numbers(low, high):
    rng = np.random.default_rng(1)
    mantissas = np.concatenate([rng.integers(0, 1 << 23, 20000), np.arange(1 << 9), (1 << 23) - 1 - np.arange(1 << 9),
                                np.array([0x00FE80, 0x00FF80, 0x008080, 0x017F80])]).astype(np.uint32)
    exponents = rng.integers(low + 127, high + 128, mantissas.size).astype(np.uint32)
    return ((exponents << np.uint32(23)) | mantissas).view(np.float32) * rng.choice(np.array([-1, 1], dtype=np.float32), mantissas.size)


def test_the_pieces_add_up_exactly_down_to_two_to_the_minus_110():
    x = numbers(-110, 127)
    assert np.array_equal(sum(piece.astype(np.float64) for piece in pieces(x)), x.astype(np.float64))
    # below, the third piece ends at the smallest bfloat16 number, 2^-133
    x = numbers(-126, -111)
    lost = np.abs(sum(piece.astype(np.float64) for piece in pieces(x)) - x.astype(np.float64))
    assert 0 < lost.max() < 2.0 ** -133


def test_what_the_six_products_leave_out():
    """a1 b2 + a2 b1 + a2 b2: second pieces are below 2^-7 of their number's power of two, third pieces at most 2^-16 of it."""
    x = numbers(0, 0)
    _, second, third = (piece.astype(np.float64) for piece in pieces(x))
    assert np.abs(second).max() <= 2.0 ** -7 and np.abs(third).max() <= 2.0 ** -16
    y = np.float32(np.concatenate([x[1:], x[:1]]))
    terms = []
    for other in (x, y):
        _, second2, third2 = (piece.astype(np.float64) for piece in pieces(other))
        terms.append((second * third2 + third * second2 + third * third2) / (x.astype(np.float64) * other))
    worst = max(np.abs(term).max() for term in terms)
    assert 3.5 * 2.0 ** -24 < worst < 2.0 ** -22
    assert abs(float(np.mean(terms[1]))) < 2.0 ** -27            # (of either sign)
