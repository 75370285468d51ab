"""CPU replay of the small-batch kernel's index arithmetic (nrldpc_split.cu): which 16-bit half of which shared word a
belief lives in, and where an edge of the row pair (zx, zx + H) reads and writes."""

import numpy as np
import pytest

ZCS = sorted({a << j for a in (2, 3, 5, 7, 9, 11, 13, 15) for j in range(8) if (a << j) <= 384})


def slot_of(i, Zc):
    """The kernel's slot_of: high multiply by ceil(2^32 / Zc), then the half."""
    H = Zc if Zc & 1 else Zc // 2
    magic = 0xFFFFFFFF // Zc + 1
    c = (i * magic) >> 32
    off = i - c * Zc
    hi = (off >= H).astype(np.int64)
    return 2 * (c * H + off - hi * H) + hi


@pytest.mark.parametrize("Zc", ZCS)
def test_every_belief_has_its_own_half(Zc):
    H = Zc if Zc & 1 else Zc // 2
    s = slot_of(np.arange(68 * Zc, dtype=np.int64), Zc)
    assert s.min() >= 0 and s.max() < 2 * 68 * H and len(np.unique(s)) == 68 * Zc


@pytest.mark.parametrize("Zc", ZCS)
def test_edges_of_a_row_pair(Zc):
    """For every circulant shift and row pair: the word's byte address and the selector give rows zx and zx + H their
    beliefs (column base + (row + shift) mod Zc) in halves 0 and 1."""
    odd = Zc & 1
    H = Zc if odd else Zc // 2
    h4, swap = 4 * H, 0 if odd else 0x2222
    zx = np.arange(H, dtype=np.int64)
    col = 67 if Zc <= 256 else 40                            # the last column of the sizes the kernel takes
    for s in range(Zc):
        upper = (not odd) and s >= H
        ex, ey, ez = (col * Zc) * (4 if odd else 2), 4 * (s - (H if upper else 0)), 0x3210 ^ (0x2222 if upper else 0)
        a = 4 * zx + ey
        b = (a - h4) & 0xFFFFFFFF
        addr = np.minimum(a, b) + ex
        neg = (b >> 31) & 1                                  # arithmetic shift by 31: all ones when negative
        sel = ez ^ np.where(neg == 1, 0, swap)
        packed = ((addr << 16) & 0xFFFFFFFF) | sel            # address and selector share a word
        assert addr.max() < 1 << 16 and np.array_equal(packed >> 16, addr) and np.array_equal(packed & 0xFFFF, sel)
        assert set(np.unique(sel)) <= {0x3210, 0x1032}
        swapped = sel == 0x1032
        for half in (0, 1) if not odd else (0,):
            want = slot_of(col * Zc + (zx + half * H + s) % Zc, Zc)
            got = 2 * (addr // 4) + np.where(swapped, 1 - half, half)
            assert np.array_equal(got, want), (s, half)
