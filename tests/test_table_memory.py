"""The device memory that tables of the default layouts take: what callers who
keep many tables, or serve them under a budget, have planned."""
import numpy as np
import pytest

import ibs_b200 as ib


@pytest.mark.parametrize("k,log2_lines", [(20, 13), (23, 19), (25, 23), (27, 27), (28, 20), (31, 26)])
def test_default_layout_by_size(k, log2_lines):
    """Minimizer lines (1.5 keys a 32-byte sector of four a line) from 2^log2_lines
    lines on, hash sectors of 4 keys below: the smallest line count that slot
    values allow is half of that, and such tables are not oversized for it."""
    first = 6 << log2_lines
    lines = ib.table_bytes_for(first, k)
    assert lines >= (128 << log2_lines)
    for n in (first - 6, first * 3 // 4, first // 2 + 6):
        hashed = ib.table_bytes_for(n, k, force_format=5)
        assert ib.table_bytes_for(n, k) == hashed < 0.55 * lines


@pytest.mark.gpu
def test_tables_of_hash_sectors_fit_a_small_budget():
    """Four samples whose hash sectors a budget holds all at once; on minimizer
    lines (which k = 20 allows from 2^12 lines) one of them would not fit."""
    k, W, n = 20, 1000, 30_000
    rng = np.random.default_rng(3)
    text = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 50_000)].tobytes()
    ref = ib.Reference(*ib.pack_ascii([text]))
    one = ib.table_bytes_for(n, k, force_format=5)
    srv = ib.Server(ref, W, k, memory_budget=int(4.4 * one))
    codes = [np.unique(rng.integers(0, 1 << 38, n).astype(np.uint64)) for _ in range(4)]
    for i, c in enumerate(codes):
        assert srv.add_codes(c, len(c), on_device=False) == i
    st = srv.stats()
    assert st["resident_tables"] == 4 and st["resident_bytes"] <= 4.4 * one
    srv.close()
    t = ib.Table.from_codes(codes[0], len(codes[0]), k, on_device=False)
    assert t.info().format == 1
    lined = ib.Table.from_codes(codes[0], len(codes[0]), k, on_device=False, force_format=4)
    assert lined.info().device_bytes > 2 * one


@pytest.mark.gpu
@pytest.mark.parametrize("k,few,many", [(28, 3_000_000, 30_000_000), (29, 11_000_000, 90_000_000)])
def test_joint_lines_take_no_more_than_hash_sectors(k, few, many):
    """Joint tables of k = 28 .. 31: minimizer lines (format 9) while they fit in
    the 2^(2k - 32) hash sectors that the keys would take at least, with room
    for the stash to double; hash sectors beyond that, and for a given load."""
    sectors = 32 << (2 * k - 32)
    for n, fmt in ((few, 9), (many, 3)):
        pt = ib.PanelTable(k, n)
        info = pt.info()[0]
        assert info.format == fmt
        assert info.device_bytes + 2 * info.stash_buckets * 32 <= 1.05 * sectors
        pt.close()
    pt = ib.PanelTable(k, few, keys_per_bucket=3.0)
    assert pt.info()[0].format == 3
    pt.close()


def _leave(nbytes):
    """Takes all the device's free memory but nbytes."""
    import torch
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - nbytes, dtype=torch.uint8, device="cuda")


@pytest.mark.gpu
def test_dense_tables_build_with_little_scratch():
    """Loads at which four keys in ten find no slot: the build's scratch is 8
    bytes for each of those (16 for a wide key), not for every key."""
    import torch
    n, kpb = 40_000_000, 12.0
    codes = torch.randint(0, 1 << 62, (n,), device="cuda")
    table = ib.table_bytes_for(n, 31, force_format=5, keys_per_bucket=kpb)

    def build():
        t = ib.Table.from_codes(codes, n, 31, on_device=True, force_format=5, keys_per_bucket=kpb)
        info = t.info()
        assert info.format in (1, 2) and 0.3 * n < info.stash_keys < 0.6 * n
        assert info.device_bytes < table + (600 << 20)
        t.close()

    build()
    held = _leave(table + (480 << 20))  # the table, its 256 MiB of stash and 5.9 bytes a key
    build()
    del held
    rng = np.random.default_rng(1)
    m = 10_000_000
    lo, hi = rng.integers(0, 1 << 62, m).astype(np.uint64), rng.integers(0, 1 << 17, m).astype(np.uint64)

    def build_wide():
        ib.Table.from_codes128(lo, hi, 41, keys_per_bucket=7.9).close()

    build_wide()
    wide = int(m / 7.9 * 128)
    held = _leave(16 * m + wide + wide // 2 + (60 << 20))  # codes, level 0, the later levels, 6 bytes a key
    build_wide()
    del held
    torch.cuda.empty_cache()
