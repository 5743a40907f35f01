"""The minimizer-line scan at the edges of its 128-position blocks: every k of
either sector layout, contigs and windows around a block's length, runs of N
at the edges, tandem repeats (several smallest keys in a k-mer) and reverse
palindromes; the joint minimizer-line table and its single-sample tables on
the same input. Rows against the hash-bucket table's, which share none of it."""
import numpy as np
import pytest

import ibs_b200 as ib
import oracle as orc

pytestmark = pytest.mark.gpu


def _world(k):
    rng = np.random.default_rng(1000 + k)
    lens = [1, k - 1, k, k + 1, 127, 128, 129, 127 + k, 128 + k, 129 + k, 128 + 2 * k, 255 + k, 256 + k, 257 + k,
            2047 + k, 2048 + k, 2049 + k, 4321, 9000]
    seqs = []
    for n in lens:
        s = rng.integers(0, 4, n)
        if n > 200:
            a = int(rng.integers(0, n - 150))
            s[a:a + 120] = np.tile(rng.integers(0, 4, int(rng.integers(1, 9))), 120)[:120]
            half = rng.integers(0, 4, 30)
            s[n - 60:] = np.concatenate([half, 3 - half[::-1]])
        t = np.frombuffer(b"ACGT", np.uint8)[s].copy()
        if n > 300:
            for p in (0, 127, 128, n - 1, int(rng.integers(0, n))):
                t[p] = ord("N")
        seqs.append(t.tobytes())
    # the sample: the k-mers of every other 37-base piece, from either strand
    pieces = [s[i:i + 37 + k - 1] for s in seqs for i in range(0, len(s), 74)]
    comp = bytes.maketrans(b"ACGTN", b"TGCAN")
    pieces = [p if i % 2 else p.translate(comp)[::-1] for i, p in enumerate(pieces)]
    codes = np.unique(np.concatenate([orc.canonical_codes(p, k) for p in pieces if len(p) >= k]
                                     + [rng.integers(0, 1 << (2 * k - 2), 500).astype(np.uint64)]))
    return seqs, codes


@pytest.mark.parametrize("k", range(16, 32))
def test_block_edges(k):
    seqs, codes = _world(k)
    ref = ib.Reference(*ib.pack_ascii(seqs))
    hashed = ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=5)
    tables = [ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=6)]
    if k <= 27:
        tables.append(ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=4))
    joint = None
    if k <= 25:  # 16-sample masks on minimizer lines (at least 2^(2k - 28) of them)
        joint = ib.PanelTable(k, 2 * len(codes), force_format=7)
        joint.add_codes(codes[::2].copy(), len(codes[::2]), on_device=False)
        joint.add_codes(codes, len(codes), on_device=False)
        half = ib.Table.from_codes(codes[::2].copy(), len(codes[::2]), k, on_device=False, force_format=5)
    for W in (k + 1, k + 127, k + 128, k + 129, 1000, 20_000):
        want = ib.scan(hashed, ref, W)
        assert want["observed_kmers"].sum() > 0
        for t in tables:
            assert np.array_equal(ib.scan(t, ref, W), want), (k, W, t.info().format)
        if joint is not None:
            rows = joint.scan(ref, W)
            assert np.array_equal(rows[1], want) and np.array_equal(rows[0], ib.scan(half, ref, W)), (k, W)


@pytest.mark.parametrize("fmt,kpb", [(4, 7.9), (6, 5.9), (4, 30.0), (6, 30.0)])
def test_full_lines(fmt, kpb):
    """Loads at which sectors, lines and the list of leftover keys overflow."""
    k = 16
    seqs, _ = _world(k)
    rng = np.random.default_rng(9)
    codes = np.unique(np.concatenate([orc.canonical_codes(s, k) for s in seqs if len(s) >= k]))
    keep = rng.random(len(codes)) < 0.7
    codes = np.concatenate([codes[keep], codes[keep][:50]])  # some twice
    t = ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=fmt, keys_per_bucket=kpb)
    h = ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=5)
    assert t.probe(codes).all()
    q = rng.integers(0, 1 << 32, 20_000).astype(np.uint64)  # half of them not canonical
    assert np.array_equal(t.probe(q), h.probe(q))
    odd = ib.Table.from_codes(q, len(q), k, on_device=False, force_format=fmt)
    assert odd.probe(q).all()
    ref = ib.Reference(*ib.pack_ascii(seqs))
    assert np.array_equal(ib.scan(t, ref, 500), ib.scan(h, ref, 500))


@pytest.mark.parametrize("k", range(16, 32))
def test_coverage_edges(k):
    seqs, codes = _world(k)
    rng = np.random.default_rng(k)
    for n in (4063, 4064, 4065, 4064 + k, 8128 + k - 1):  # around the mapper's spans
        seqs.append(np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes())
        codes = np.concatenate([codes, orc.canonical_codes(seqs[-1], k)[::3]])
    codes = np.unique(codes)
    ref = ib.Reference(*ib.pack_ascii(seqs))
    want = ib.map_coverage(ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=5), ref)
    assert want.max() > 1
    for fmt in (4, 6) if k <= 27 else (6,):
        t = ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=fmt)
        assert np.array_equal(ib.map_coverage(t, ref), want), (k, fmt)


@pytest.mark.parametrize("k", [16, 21, 25, 27, 28, 31])
def test_noalloc_edges(k):
    import torch
    seqs, codes = _world(k)
    seq, mask, lens = ib.pack_ascii(seqs)
    ref = ib.Reference(seq, mask, lens)
    dseq, dmask = torch.from_numpy(seq.view(np.int64)).cuda(), torch.from_numpy(mask.view(np.int64)).cuda()
    h = ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=5)
    for fmt in (4, 6) if k <= 27 else (6,):
        t = ib.Table.from_codes(codes, len(codes), k, on_device=False, force_format=fmt)
        for W in (k + 1, k + 128, 1000, 20_000):
            want = ib.scan(h, ref, W)
            rows = torch.zeros((len(want), 6), dtype=torch.int32, device="cuda")
            ib.scan_noalloc(t, dseq, dmask, lens, W, rows, len(want), torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert np.array_equal(rows.cpu().numpy(), want.view(np.int32).reshape(-1, 6)), (k, fmt, W)


@pytest.mark.parametrize("k", [28, 29, 30, 31])
@pytest.mark.parametrize("passes", [1, 3])
def test_joint_lines_of_long_k(k, passes):
    """Joint tables of k = 28 .. 31 that expect enough keys take minimizer lines
    of 40-bit slots: masks and rows as the hash sectors', in one pass and in
    bucket ranges."""
    seqs, codes = _world(k)
    rng = np.random.default_rng(k)
    share = [codes[rng.random(len(codes)) < 0.2 + 0.05 * i] for i in range(16)]
    ref = ib.Reference(*ib.pack_ascii(seqs))
    many = int((1 << (2 * k - 37)) * 4 * 1.2) + 100_000
    t = ib.PanelTable(k, many)
    h = ib.PanelTable(k, 16, force_format=3) if k < 30 else None  # 2^(2k - 32) sectors at least
    for c in share:
        t.add_codes(c, len(c), on_device=False)
        if h is not None:
            h.add_codes(c, len(c), on_device=False)
    assert t.info()[0].format not in (3, 7)
    want = sum(np.isin(codes, c).astype(np.uint32) << np.uint32(i) for i, c in enumerate(share))
    assert np.array_equal(t.probe(codes), want)
    tune = ib.get_tuning()
    kept = tune.panel_pass_mb
    if passes > 1:
        tune.panel_pass_mb = max(1, int(t.info()[0].n_buckets * 32 / passes / (1 << 20)) + 1)
        ib.set_tuning(tune)
    try:
        for W in (k + 1, k + 128, 1000, 20_000):
            rows = t.scan(ref, W)
            if h is not None:
                assert np.array_equal(rows, h.scan(ref, W)), (k, W)
            one = ib.Table.from_codes(share[7], len(share[7]), k, on_device=False, force_format=5)
            assert np.array_equal(rows[7], ib.scan(one, ref, W)), (k, W)
    finally:
        tune.panel_pass_mb = kept if kept else 0xFFFFFFFF
        ib.set_tuning(tune)
