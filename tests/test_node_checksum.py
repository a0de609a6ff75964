"""The rule by which a tile tells whether a node image carries its own checksum
(mt_node.cuh, node::verified), restated on the host: the checksum is a 64-bit
sum of word times odd factor, the lanes add up the low and the high halves of
their parts (less the stored words) apart, and the high sum may fall short by
the carries of the low one, 0 .. T - 1.  Checked against the plain 64-bit comparison."""
import numpy as np
import pytest

M64, M32 = (1 << 64) - 1, (1 << 32) - 1
CSUM, META, LOCK = 26, 30, 1 << 4


def factor(g):
    x = ((2 * g + 1) * 0x9E3779B1) & M32
    return (x ^ (x >> 15)) | 1


def term(g, v):
    if g in (CSUM, CSUM + 1):
        return 0
    return (v & ~LOCK if g == META else v) * factor(g)


def checksum(w):
    return (0x5BD1E9955BD1E995 + sum(term(g, v) for g, v in enumerate(w))) & M64


def verified(w, T):
    per = 32 // T
    low = high = 0
    for lane in range(T):
        h = 0
        for g in range(lane * per, lane * per + per):
            h += term(g, w[g])
            h -= w[g] if g == CSUM else w[g] << 32 if g == CSUM + 1 else 0
        h &= M64
        low, high = (low + (h & M32)) & M32, (high + (h >> 32)) & M32
    whole = -0x5BD1E9955BD1E995 & M64
    return low == whole & M32 and ((whole >> 32) - high & M32) < T


@pytest.mark.parametrize("T", [4, 8, 16, 32])
@pytest.mark.parametrize("kind", ["random", "small", "full", "zero"])
def test_an_image_passes_and_a_changed_one_does_not(T, kind):
    rng = np.random.default_rng(T)
    for _ in range(200):
        w = [int(x) for x in rng.integers(0, {"random": 1 << 32, "small": 16, "full": 1 << 32, "zero": 1}[kind], 32)]
        if kind == "full":
            w = [x | 0xFFFFFF00 for x in w]
        h = checksum(w)
        w[CSUM], w[CSUM + 1] = h & M32, h >> 32
        assert verified(w, T)
        locked = list(w)
        locked[META] ^= LOCK
        assert verified(locked, T)  # the lock bit moves without a republish
        g = int(rng.integers(0, 32))
        one = list(w)
        one[g] ^= 1 << int(rng.integers(0, 32))
        # (The high half of the stored sum alone may be off by the carries: the
        # other 31 words are then those of one image.)
        if g != CSUM + 1 and (g != META or one[g] ^ w[g] != LOCK):
            assert not verified(one, T)
        # Two words of another image (a torn read), and the entries from one
        # place on moved up by one, as an insert does.
        torn = list(w)
        for g in rng.choice(26, 2, replace=False):
            torn[g] = (torn[g] + 1 + int(rng.integers(0, 1 << 20))) & M32
        at = 2 * int(rng.integers(0, 12))
        moved = w[:at] + [1, 2] + w[at:24] + w[26:]
        for image in (torn, moved):
            same = checksum(image) == (image[CSUM + 1] << 32 | image[CSUM])
            assert verified(image, T) == same
