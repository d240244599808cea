"""The mixed windows of the scalars' recoding (c and c - 1 bits, the wider ones
first), restated on Python integers: every scalar is the sum of its digits at
the windows' offsets, digits fit the 2^(c - 1) buckets, and no carry leaves the
top window."""
import random

import pytest

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001


@pytest.mark.parametrize("c", range(8, 17))
def test_mixed_windows(c):
    rng = random.Random(c)
    count = 255 // c + 1
    wide = 255 - count * (c - 1)
    assert 0 <= wide < count
    bits = [c if j < wide else c - 1 for j in range(count)]
    offs = [sum(bits[:j]) for j in range(count)]
    assert sum(bits) == 255
    edge = [0, 1, 2, R - 1, R - 2, (1 << 254), (1 << 254) - 1, (1 << c) - 1, 1 << (c - 1), (1 << (c - 1)) + 1]
    for s in edge + [rng.randrange(R) for _ in range(300)]:
        carry, total = 0, 0
        for j in range(count):
            raw = ((s >> offs[j]) & ((1 << bits[j]) - 1)) + carry
            carry = int(raw > 1 << (c - 1))
            digit = raw - (carry << c)
            assert abs(digit) <= 1 << (c - 1)
            total += digit << offs[j]
        assert carry == 0 and total == s
