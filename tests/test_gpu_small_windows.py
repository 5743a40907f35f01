"""Rows of windows of very different span counts: groups of 1 to 32 lanes finish
a window, and a window of many spans among hundreds of thousands of one-span
windows is finished by fewer lanes than it has spans; and tables of both kinds
on one reference, whose spans differ in length."""
import numpy as np
import pytest

import ibs_b200 as ib
import oracle as orc

pytestmark = pytest.mark.gpu
K = 21


def _text(rng, n):
    return np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes()


def _sample(seqs, rng, share=0.6):
    codes = np.unique(np.concatenate([orc.canonical_codes(s, K) for s in seqs if len(s) >= K]))
    return codes[rng.random(len(codes)) < share]


def _tables(codes):
    joint = ib.PanelTable(K, 2 * len(codes), force_format=7)
    joint.add_codes(codes[::3].copy(), len(codes[::3]), on_device=False)
    joint.add_codes(codes, len(codes), on_device=False)
    hashed = ib.PanelTable(K, 2 * len(codes), force_format=3)
    hashed.add_codes(codes, len(codes), on_device=False)
    return [ib.Table.from_codes(codes, len(codes), K, on_device=False, force_format=f) for f in (5, 4, 6)], joint, hashed


@pytest.mark.parametrize("positions", [1, 2, 33, 64, 97, 127, 128, 129, 255, 257, 513, 1025, 2049, 4097, 4300])
def test_spans_a_window(positions):
    """Windows of 1 to 34 spans of 128 positions."""
    rng = np.random.default_rng(positions)
    W = positions + K - 1
    if W <= K:
        W = K + 1
    seqs = [_text(rng, n) for n in (3 * W + 7, K, 40, W, W + 1, max(W // 2, K))]
    codes = _sample(seqs, rng)
    ref = ib.Reference(*ib.pack_ascii(seqs))
    singles, joint, hashed = _tables(codes)
    want = ib.scan(singles[0], ref, W)
    r = 0
    for s in seqs:  # the counts of every window, position by position
        c = orc.canonical_codes(s, K) if len(s) >= K else np.zeros(0, np.uint64)
        hit = np.isin(c, codes)
        for a in range(0, len(s), W - K):
            n = max(0, min(a + W, len(s)) - a - K + 1)
            assert want[r]["total_kmers"] == n and want[r]["observed_kmers"] == hit[a:a + n].sum()
            r += 1
    assert r == len(want)
    for t in singles[1:]:
        assert np.array_equal(ib.scan(t, ref, W), want)
    assert np.array_equal(joint.scan(ref, W)[1], want)
    assert np.array_equal(hashed.scan(ref, W)[0], want)


def test_long_windows_among_very_many_short_ones():
    rng = np.random.default_rng(5)
    W, n_short = 20_000, 310_000
    long_ = [_text(rng, 130_000), _text(rng, 50_001)]
    short = [_text(rng, K + 3)] * 7 + [_text(rng, K)] * 3
    seqs = long_[:1] + short * (n_short // 10) + long_[1:]
    codes = _sample(long_ + short, rng)
    ref, few = ib.Reference(*ib.pack_ascii(seqs)), ib.Reference(*ib.pack_ascii(long_ + short))
    singles, joint, hashed = _tables(codes)
    first, second = ib.window_count([130_000], W, K), ib.window_count([50_001], W, K)
    for rows, alone in [(ib.scan(t, ref, W), ib.scan(t, few, W)) for t in singles] + \
                       [(joint.scan(ref, W)[1], joint.scan(few, W)[1]), (hashed.scan(ref, W)[0], hashed.scan(few, W)[0])]:
        assert np.array_equal(rows[:first], alone[:first])
        assert np.array_equal(rows[-second:], alone[first:first + second])
        assert np.array_equal(rows[first:-second], np.tile(alone[first + second:], n_short // 10))
        assert rows["observed_kmers"].sum() > 0


def test_tables_of_both_kinds_in_turn():
    """24 Mbp: spans of 512 positions for hash buckets, 1024 for minimizer lines."""
    import torch
    spec = ib.RefSpec(seed=77, lens=[20_000_000, 4_000_001], n_frac=0.003, n_run=(1, 300))
    sw, mw = spec.packed_words()
    seq, mask = (torch.empty(n, dtype=torch.int64, device="cuda") for n in (sw, mw))
    spec.reference_device(seq, mask)
    smp = ib.SampleSpec(seed=78, k=K, class_rate=(0.001, 0.03), class_prob=(0.5, 0.5), block_len=100_000,
                        random_frac=0.05)
    cap = smp.codes_device_bound(spec, seq, mask)
    codes = torch.empty(cap, dtype=torch.int64, device="cuda")
    n = smp.codes_device(spec, seq, mask, codes, cap)
    ref = ib.Reference(seq, mask, spec.lens, on_device=True)
    hashed, lined = (ib.Table.from_codes(codes, n, K, on_device=True, force_format=f) for f in (5, 4))
    other = ib.Table.from_codes(codes, n // 2, K, on_device=True, force_format=5)
    for W in (5000, 50_000):
        want, half = ib.scan(hashed, ref, W), ib.scan(other, ref, W)
        assert 0 < half["observed_kmers"].sum() < want["observed_kmers"].sum()
        for _ in range(2):
            assert np.array_equal(ib.scan(lined, ref, W), want)
            assert np.array_equal(ib.scan(hashed, ref, W), want)
        for tables, rows in (([hashed, other], [want, half]), ([other, lined], [half, want])):
            assert np.array_equal(np.asarray(ib.scan_panel(tables, ref, W)).reshape(2, -1), np.stack(rows))
