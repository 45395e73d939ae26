"""The bounds that the arithmetic of long primes next to 2^60 rests on (LongPm and convert_target_pm), restated with whole numbers of any size: no sum
leaves 64 bits, no difference falls below zero, every value stays congruent.  Transforms of canonical residues come nowhere near these bounds, so
the comparisons on the GPU cannot show one that is too tight."""
import random

import pytest

UNIT, WORD = 1 << 60, 1 << 64
# 2^60 - d with d odd and below 2^26, smallest to largest; only the form of q matters here, not that it is prime
DISTANCES = [1, (1 << 17) - 1, (1 << 25) + 1, (1 << 26) - 1]


def pieces(v):
    assert v < UNIT
    return v & (1 << 29) - 1, v >> 29  # 29 and 31 bits


def fold_sums(a, b, d):
    """A + B * 2^29 with B folded by 2^61 = 2d"""
    assert a < WORD and b < WORD
    r = a + ((b & 0xFFFFFFFF) << 29) + (b >> 32) * 2 * d
    assert r < WORD
    return r


def mul(x, w, d):
    q = UNIT - d
    assert x < WORD and w < q
    (wl, wh), (cl, ch) = pieces(w), pieces(w * (1 << 32) % q)
    x0, x1 = x & 0xFFFFFFFF, x >> 32
    r = fold_sums(x0 * wl + x1 * cl, x0 * wh + x1 * ch, d)
    assert r % q == x * w % q
    return r


def largest_product(limit, d):
    """An upper bound of mul(x, any constant) for x below `limit`: every piece at its largest."""
    x0, x1 = (1 << 32) - 1, min(limit - 1, WORD - 1) >> 32
    low, high = (1 << 29) - 1, (1 << 31) - 1
    return (x0 + x1) * low + (((1 << 32) - 1) << 29) + ((x0 + x1) * high >> 32) * 2 * d + 1


def fold(x, d):
    assert x < 16 * UNIT
    r = (x & UNIT - 1) + (x >> 60) * d
    assert r < UNIT + (1 << 30) and (r - x) % (UNIT - d) == 0
    return r


def canon(x, d):
    r, q = fold(x, d), UNIT - d
    r = r - q if r >= q else r
    assert r < q
    return r


@pytest.mark.parametrize("d", DISTANCES)
def test_products_and_folds(d):
    q, rng = UNIT - d, random.Random(d)
    edges = [0, 1, (1 << 29) - 1, 1 << 29, (1 << 32) - 1, 1 << 32, q - 1, q // 2]
    words = [0, 1, (1 << 32) - 1, WORD - (1 << 32), WORD - 1, 7 * q, 14 * q] + [rng.randrange(WORD) for _ in range(50)]
    for x in words:
        for w in edges + [rng.randrange(q) for _ in range(50)]:
            r = mul(x, w, d)
            assert r < 4.5 * UNIT + x / 8 + 1 and r < largest_product(x + 1, d) <= 6.5 * UNIT
            canon(r, d)
        if x < 16 * UNIT:
            canon(x, d)


@pytest.mark.parametrize("d", DISTANCES)
@pytest.mark.parametrize("start", ["canonical", "a conversion, whose upper half is made"])
def test_forward_rounds(d, start):
    """Sixteen stages; sums and differences are of a value below `bound` (folded at every second stage) and a product."""
    q = UNIT - d
    made = start != "canonical"
    bound = 6.5 * UNIT if made else q
    for stage in range(16):
        product = bound if made and stage == 0 else largest_product(int(bound), d)
        assert product < 7 * q  # y = x + 7q - t
        x = UNIT + (1 << 30) if stage % 2 else bound
        bound = max(x + 7 * q, x + product)
        assert bound < (8.1 if stage % 2 else 15.1) * UNIT < WORD
    assert 14 * q > bound and q + 14 * q < 16 * UNIT  # the last step of ModDown and of the rescale: a residue + 14q - v


@pytest.mark.parametrize("d", DISTANCES)
def test_inverse_rounds(d):
    q = UNIT - d
    bound = q
    for stage in range(15):
        assert bound < 7 * q and 2 * bound < 16 * UNIT and bound + 7 * q < 16 * UNIT
        bound = max(UNIT + (1 << 30), largest_product(int(bound) + 7 * q, d))
        assert bound < 6.3 * UNIT
    assert 2 * bound < 16 * UNIT and bound + 7 * q < 16 * UNIT  # the last stage, multiplied by the scale


@pytest.mark.parametrize("d", DISTANCES)
def test_conversions_of_four_sources(d):
    q, rng = UNIT - d, random.Random(d)
    top = (1 << 30) - 1
    worst = fold_sums(4 * top * 2 * ((1 << 29) - 1), 4 * top * 2 * ((1 << 31) - 1), d)  # both sums stay words, every piece at its largest
    assert worst < 6.5 * UNIT
    assert 4 * top * 2 * ((1 << 29) - 1) < 1 << 63
    assert (5 * top * 2 * ((1 << 31) - 1)) >= WORD  # a fifth source would not fit
    for trial in range(200):
        a = b = true = 0
        for _ in range(4):
            y = UNIT - 1 if trial % 4 == 0 else rng.randrange(UNIT)
            c = q - 1 - rng.randrange(3) if trial % 3 == 0 else rng.randrange(q)
            (cl, ch), (el, eh) = pieces(c), pieces(c * (1 << 30) % q)
            a += (y & top) * cl + (y >> 30) * el
            b += (y & top) * ch + (y >> 30) * eh
            true += y * c
        assert fold_sums(a, b, d) % q == true % q
