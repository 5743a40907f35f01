"""Every table layout through the server, in each of its launch modes: lone
requests of part of a contig and overlapping bursts, rows equal to full scans of
each sample's hash-bucket table."""
import time

import numpy as np
import pytest

import ibs_b200 as ib

pytestmark = pytest.mark.gpu
W = 3000


def _world(k):
    spec = ib.RefSpec(seed=900 + k, lens=[700_000, 311_111, 2_000, k, 90_001], n_frac=0.004, n_run=(1, 200))
    seq, mask = spec.reference_host()
    samples = [ib.SampleSpec(seed=950 + s, k=k, class_rate=(0.0005, 0.03), class_prob=(0.6, 0.4), block_len=20_000,
                             present_frac=0.5 + 0.2 * s, random_frac=0.05).codes_host(spec, seq, mask)
               for s in range(3)]
    ref = ib.Reference(seq, mask, spec.lens)
    full = [ib.scan(ib.Table.from_codes(c, len(c), k, on_device=False, force_format=5), ref, W) for c in samples]
    starts = np.concatenate([[0], np.cumsum([ib.window_count([n], W, k) for n in spec.lens])])
    return spec, ref, samples, full, starts


@pytest.mark.parametrize("mode", ["persistent", "iteration", "serial"])
@pytest.mark.parametrize("k,layout", [(15, 1), (17, 1), (25, 2), (31, 2), (32, 2), (16, 4), (21, 4), (24, 4), (20, 6), (29, 6),
                                      (15, "joint 3"), (25, "joint 3"), (28, "joint 3"), (16, "joint 7"),
                                      (21, "joint 7"), (25, "joint 7"), (28, "joint 9"), (29, "joint 9")])
def test_layouts_served(k, layout, mode):
    spec, ref, samples, full, starts = _world(k)
    joint = isinstance(layout, str)
    fmt = int(layout.split()[-1]) if joint else layout
    srv = ib.Server(ref, W, k, iteration_launches=mode == "iteration", one_request_per_launch=mode == "serial",
                    table_format={1: 5, 2: 5}.get(fmt, fmt))
    if joint:
        keys = sum(len(c) for c in samples)
        if fmt == 9:  # the fewest that take minimizer lines of 40-bit slots
            keys = int((1 << (2 * k - 37)) * 4 * 1.2) + 100_000
        pt = ib.PanelTable(k, keys, force_format=0 if fmt == 9 else fmt)
        for c in samples:
            pt.add_codes(c, len(c), on_device=False)
        assert pt.info()[0].format == fmt
        assert srv.add_panel(pt, release=True) == [0, 1, 2]
        pt.close()
    else:
        one = ib.Table.from_codes(samples[0], len(samples[0]), k, on_device=False, force_format=5 if fmt < 3 else fmt)
        assert one.info().format == fmt
        for i, c in enumerate(samples):
            assert srv.add_codes(c, len(c), on_device=False) == i
    rng = np.random.default_rng(k)

    def some():
        c = int(rng.integers(0, 5))
        nw = int(starts[c + 1] - starts[c])
        first = int(rng.integers(0, nw))
        return int(rng.integers(0, 3)), c, first, int(rng.integers(1, nw - first + 1))

    def check(r):
        assert r["status"] == 0
        a = int(starts[r["contig"]] + r["first_window"])
        assert np.array_equal(r["rows"], full[r["sample"]][a:a + r["n_windows"]]), (r["sample"], r["contig"])

    for _ in range(4):
        req = some()
        srv.submit(*req)
        got = srv.poll(1, timeout_ms=60_000)
        assert len(got) == 1, ("no result within 60 s", req, srv.stats())
        check(got[0])
    reqs = [(s, c, 0, 0) for c in range(5) for s in range(3)] + [some() for _ in range(30)]
    for req in reqs:
        srv.submit(*req)
    done, deadline = [], time.time() + 120
    while len(done) < len(reqs) and time.time() < deadline:
        done += srv.poll(64, timeout_ms=2000)
    assert len(done) == len(reqs), ("requests left unfinished", srv.stats())
    for r in done:
        check(r)
    srv.close()
    ref.free()
