"""Joint tables on minimizer lines: builds in which half of the keys have two
places, and the longest k of the 32-bit layout at the edges of the scan's blocks."""
import numpy as np
import pytest

import ibs_b200 as ib
from test_gpu_mz_edges import _world

pytestmark = pytest.mark.gpu


def test_keys_of_two_places():
    """k = 17: every k-mer that holds a reverse-palindromic 16-mer; it is the
    minimizer of half of them, which are filed under two places each (130,684 of
    262,142), more than the build's lists have room for at once."""
    k = 17
    half = np.arange(1 << 16, dtype=np.uint64)
    rc = np.zeros_like(half)
    for i in range(8):
        rc |= (np.uint64(3) - ((half >> np.uint64(2 * i)) & np.uint64(3))) << np.uint64(2 * (7 - i))
    pal = (half << np.uint64(16)) | rc
    mers = np.concatenate([(pal << np.uint64(2)) | np.uint64(x) for x in range(4)] +
                          [pal | np.uint64(x << 32) for x in range(4)])
    other = np.zeros_like(mers)
    for i in range(k):
        other |= (np.uint64(3) - ((mers >> np.uint64(2 * i)) & np.uint64(3))) << np.uint64(2 * (k - 1 - i))
    codes = np.unique(np.minimum(mers, other))
    assert len(codes) == 262_142
    samples = [codes, codes[::2].copy(), codes[1::3].copy()]
    t = ib.PanelTable(k, len(codes), force_format=7)
    h = ib.PanelTable(k, len(codes), force_format=3)
    for c in samples:
        t.add_codes(c, len(c), on_device=False)
        h.add_codes(c, len(c), on_device=False)
    want = sum(np.isin(codes, c).astype(np.uint32) << np.uint32(i) for i, c in enumerate(samples))
    assert np.array_equal(t.probe(codes), want)
    rng = np.random.default_rng(2)
    text = np.frombuffer(b"ACGT", np.uint8)
    bases = (codes[rng.integers(0, len(codes), 20_000), None] >> np.uint64(2) * np.arange(k - 1, -1, -1).astype(np.uint64)) & np.uint64(3)
    fwd = bases.astype(np.uint8).ravel()
    ref = ib.Reference(*ib.pack_ascii([text[fwd].tobytes(), text[3 - fwd[::-1]].tobytes()]))
    for W in (k + 1, 300, 5000):
        rows = t.scan(ref, W)
        assert rows["observed_kmers"].sum() > 0 and np.array_equal(rows, h.scan(ref, W))


@pytest.mark.parametrize("k", [26, 27])
def test_block_edges_of_the_longest_k(k):
    """2^(2k - 28) lines at least: 2.1 and 8.6 GB."""
    seqs, codes = _world(k)
    ref = ib.Reference(*ib.pack_ascii(seqs))
    joint = ib.PanelTable(k, 2 * len(codes), force_format=7)
    share = [codes[::2].copy(), codes, codes[1::5].copy()]
    for c in share:
        joint.add_codes(c, len(c), on_device=False)
    single = [ib.Table.from_codes(c, len(c), k, on_device=False, force_format=5) for c in share]
    for W in (k + 1, k + 127, k + 128, k + 129, 1000, 20_000):
        rows = joint.scan(ref, W)
        for r, t in zip(rows, single):
            assert np.array_equal(r, ib.scan(t, ref, W)), (k, W)
    joint.close()
