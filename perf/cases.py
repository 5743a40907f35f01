"""The work a user of ibs_b200 has it do, as measured cases.

Every kind of pass goes through the package's public calls, on synthetic inputs of the shapes the
repository's workloads have (configs.py): a reference of one or many contigs with N runs, and
samples that are SNP-divergent copies of it, in blocks of different divergence, plus k-mers the
reference does not hold. All of it is made from the seed, on the GPU.

Every output is a whole number (window rows, coverage text, counts): there is nothing to round.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-ibs_b200", "python"))
import ibs_b200 as ib  # noqa: E402

# SNP rates of a sample's blocks and how often each occurs (the block model of configs.py)
RATES = (0.0001, 0.005, 0.02, 0.05)
PROBS = (0.2, 0.4, 0.3, 0.1)


def listed():
    return [
        # the 1 Mbp workload of configs.py, scanned by itself: launches and latency count
        {"name": "scan_1mbp_k25", "kind": "scan", "k": 25, "bases": 1_000_000, "contigs": 2, "W": 50_000},
        # a draft assembly: thousands of scaffolds of very different lengths, small windows, a k
        # that the kernels do not fix at compile time
        {"name": "scan_scaffolds_k21", "kind": "scan", "k": 21, "bases": 60_000_001, "contigs": 3000, "W": 5_000},
        # the headline workload (plain 2 Gbp, k = 25, 50 kbp windows) at half its size, so that several fit
        {"name": "scan_1gbp_k25", "kind": "scan_async", "k": 25, "bases": 1_000_000_000, "contigs": 10, "W": 50_000},
        # the k of the 4 Gbp panel's samples, one of them scanned alone (40-bit slots)
        {"name": "scan_500mbp_k31", "kind": "scan_async", "k": 31, "bases": 500_000_000, "contigs": 7, "W": 50_000},
        # end to end: the packed reference comes from pinned host memory at every call
        {"name": "packed_400mbp_k25", "kind": "packed", "k": 25, "bases": 400_000_000, "contigs": 10, "W": 50_000},
        # the command line's path: FASTA text in host memory, parsed and scanned
        {"name": "fasta_150mbp_k25", "kind": "fasta", "k": 25, "bases": 150_000_003, "contigs": 40, "W": 50_000},
        # k-mers of more than 32 bases
        {"name": "wide_16mbp_k41", "kind": "wide", "k": 41, "bases": 16_000_000, "contigs": 5, "W": 50_000},
        # the batched panel: 16 samples of k = 31 in one joint table
        {"name": "panel_200mbp_k31", "kind": "panel", "k": 31, "bases": 200_000_000, "contigs": 7, "W": 50_000,
         "samples": 16},
        # the served stream: regions of 16 resident samples requested at once, batched by the server
        {"name": "serve_100mbp_k25", "kind": "serve", "k": 25, "bases": 100_000_000, "contigs": 10, "W": 50_000,
         "samples": 16, "requests": 64},
        # the mapper: how many of the sample's k-mers cover each base
        {"name": "map_64mbp_k25", "kind": "map", "k": 25, "bases": 64_000_000, "contigs": 6},
        # a service that cannot allocate while it scans
        {"name": "noalloc_250mbp_k25", "kind": "noalloc", "k": 25, "bases": 250_000_000, "contigs": 10, "W": 50_000},
        # KDBIntersect: one sample's k-mers built into a table, another's counted in it
        {"name": "intersect_200mbp_k25", "kind": "intersect", "k": 25, "bases": 200_000_000, "contigs": 8},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd, every kind, k and window in use."""
    kind = rng.choice(["scan", "scan", "scan_async", "scan_async", "packed", "fasta", "wide", "panel", "panel",
                       "serve", "map", "noalloc", "intersect"])
    case = {"kind": kind}
    if kind == "wide":
        case["k"] = rng.choice([33, 41, 63, 64])
    elif kind == "serve":
        case["k"] = rng.choice([21, 25])
    elif kind == "panel":
        case["k"] = rng.choice([21, 25, 31])
    else:
        case["k"] = rng.choice([15, 21, 25, 25, 27, 31, 31, 32])
    top = {"scan": 5e8, "scan_async": 6e8, "packed": 3e8, "fasta": 1.5e8, "wide": 1.6e7, "panel": 1.5e8,
           "serve": 8e7, "map": 6e7, "noalloc": 2.5e8, "intersect": 1.5e8}[kind]
    case["bases"] = _log(rng, 300_000, top)
    case["contigs"] = min(_log(rng, 1, 3000), case["bases"] // 5000)
    if kind not in ("map", "intersect"):
        case["W"] = rng.choice([1_000, 5_000, 20_000, 50_000, 50_000, 100_003])
    if kind == "panel":
        case["samples"] = rng.choice([2, 5, 8, 16])
    if kind == "serve":
        case["samples"] = rng.choice([4, 16])
        case["requests"] = rng.choice([1, 16, 64])
    return case


def _lens(case):
    """Contig lengths over two orders of magnitude, adding up to the case's bases; the same for every seed."""
    n, total = case["contigs"], case["bases"]
    if n <= 1:
        return [total]
    r = random.Random(total * 31 + n)
    weight = [math.exp(r.uniform(0, math.log(100 if n > 50 else 4))) for _ in range(n)]
    lens = [max(1, int(total * w / sum(weight))) for w in weight]
    lens[0] += total - sum(lens)
    return lens


def _block(case):
    return max(20_000, min(1_000_000, case["bases"] // 50))


def _reference(case, seed):
    """The reference's spec and its packed words on the GPU."""
    spec = ib.RefSpec(seed=2 * seed + 1, lens=_lens(case), n_frac=0.005, n_run=(50, 500))
    sw, mw = spec.packed_words()
    seq = torch.empty(sw, dtype=torch.int64, device="cuda")
    mask = torch.empty(mw, dtype=torch.int64, device="cuda")
    spec.reference_device(seq, mask)
    return spec, seq, mask


def _codes(case, spec, seq, mask, seed, present=1.0):
    """One sample's canonical k-mers on the GPU: (codes, how many)."""
    s = ib.SampleSpec(seed=seed, k=case["k"], class_rate=RATES, class_prob=PROBS, block_len=_block(case),
                      present_frac=present, random_frac=0.10 * present)
    cap = s.codes_device_bound(spec, seq, mask)
    codes = torch.empty(max(cap, 1), dtype=torch.int64, device="cuda")
    return codes, s.codes_device(spec, seq, mask, codes, cap)


def _present(case):
    """How much of the reference each sample of a panel holds (their sizes are log-uniform)."""
    r = random.Random(case["bases"] * 7 + case["samples"])
    return [math.exp(r.uniform(math.log(0.15), 0.0)) for _ in range(case["samples"])]


def _joint(case, spec, seq, mask, seed):
    """A joint table of the case's samples."""
    share = _present(case)
    # the samples share their undiverged k-mers (about half); the rest is their own
    union = int(case["bases"] * (0.6 + 0.55 * sum(share)))
    panel = ib.PanelTable(case["k"], union)
    for i, p in enumerate(share):
        codes, n = _codes(case, spec, seq, mask, 1000 * seed + i, p)
        panel.add_codes(codes, n, on_device=True)
    return panel


def _bases(seq, n):
    """The 2-bit bases [0, n) of packed words, one byte each."""
    out = torch.empty(seq.numel() * 32, dtype=torch.uint8, device="cuda")
    shift = 2 * torch.arange(32, device="cuda")
    for a in range(0, seq.numel(), 1 << 20):
        part = (seq[a:a + (1 << 20), None] >> shift) & 3
        out[32 * a:32 * a + part.numel()] = part.reshape(-1).to(torch.uint8)
    return out[:n]


def _bits(mask, n):
    shift = torch.arange(64, device="cuda")
    return ((mask[:, None] >> shift) & 1).reshape(-1)[:n].bool()


def _fasta(spec, seq, mask, seed):
    """The reference as FASTA text: 80 bases a line, N runs, lowercase (masked) repeats."""
    total = 64 * (mask.numel() - 1)
    text = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")[_bases(seq, total).int()]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lower = torch.rand(total // 256 + 1, generator=gen, device="cuda") < 0.3
    text |= (lower.repeat_interleave(256)[:total] * 32).to(torch.uint8)
    text[_bits(mask, total)] = ord("N")
    out, at = [], 0
    for name, n in zip(spec.names, (int(x) for x in spec.lens)):
        line = torch.full((-(-n // 80), 81), ord("\n"), dtype=torch.uint8, device="cuda")
        body = torch.zeros(line.shape[0] * 80, dtype=torch.uint8, device="cuda")
        body[:n] = text[at:at + n]
        line[:, :80] = body.view(-1, 80)
        flat = line.reshape(-1)
        last = n - 80 * (line.shape[0] - 1)
        out += [b">" + name.encode() + b"\n", flat[:81 * (line.shape[0] - 1) + last].cpu().numpy().tobytes(), b"\n"]
        at += (n + 63) // 64 * 64
    return b"".join(out)


def _wide_codes(case, spec, seq, seed):
    """Low and high words of the canonical k-mers (k > 32) of a diverged copy of every other block."""
    k, lo, hi, at = case["k"], [], [], 0
    gen = torch.Generator(device="cuda").manual_seed(seed)
    all_bases = _bases(seq, 32 * (seq.numel() - 1)).long()
    for n in (int(x) for x in spec.lens):
        b = all_bases[at:at + n]
        at += (n + 63) // 64 * 64
        if n < k:
            continue
        block = _block(case)
        rate = torch.tensor(RATES, device="cuda")[torch.multinomial(torch.tensor(PROBS, device="cuda"), n // block + 1,
                                                                    replacement=True, generator=gen)]
        snp = torch.rand(n, generator=gen, device="cuda") < rate.repeat_interleave(block)[:n]
        b = (b + snp * torch.randint(1, 4, (n,), generator=gen, device="cuda")) & 3
        m = n - k + 1
        fwd, rev = [torch.zeros(m, dtype=torch.int64, device="cuda") for _ in "lh"], \
                   [torch.zeros(m, dtype=torch.int64, device="cuda") for _ in "lh"]
        for j in range(k):
            for code, sym, place in ((fwd, b[j:j + m], 2 * (k - 1 - j)), (rev, 3 - b[j:j + m], 2 * j)):
                code[place >= 64] |= sym << (place % 64)
        flip = torch.iinfo(torch.int64).min  # unsigned order of the signed words
        first = (fwd[1] ^ flip < rev[1] ^ flip) | ((fwd[1] == rev[1]) & (fwd[0] ^ flip <= rev[0] ^ flip))
        keep = (torch.arange(m, device="cuda") // block) % 2 == seed % 2
        lo.append(torch.where(first, fwd[0], rev[0])[keep])
        hi.append(torch.where(first, fwd[1], rev[1])[keep])
    if not lo:
        lo, hi = [torch.zeros(1, dtype=torch.int64)], [torch.zeros(1, dtype=torch.int64)]
    return torch.cat(lo).cpu().numpy().view(np.uint64), torch.cat(hi).cpu().numpy().view(np.uint64)


def _requests(case, seed):
    """Regions of one contig for one sample each: log-uniform lengths up to the whole contig (the same for every
    seed), of a sample and a place that the seed says."""
    size, r, got = random.Random(case["bases"] + case["requests"]), random.Random(seed), []
    lens = _lens(case)
    for _ in range(case["requests"]):
        c = size.randrange(len(lens))
        nw = ib.window_count([lens[c]], case["W"], case["k"])
        n = max(1, min(nw, int(math.exp(size.uniform(0, math.log(nw + 1))))))
        got.append((r.randrange(case["samples"]), c, r.randrange(nw - n + 1), n))
    return got


def prepare(case, seed):
    kind, k = case["kind"], case["k"]
    spec, seq, mask = _reference(case, seed)
    s = {"kind": kind, "W": case.get("W"), "lens": spec.lens}
    if kind in ("scan", "scan_async", "map", "wide", "panel", "serve"):
        s["ref"] = ib.Reference(seq, mask, spec.lens, on_device=True)
    if kind in ("scan_async", "noalloc", "panel"):
        s["windows"] = ib.window_count(spec.lens, case["W"], k)
        s["rows"] = torch.empty((case.get("samples", 1), s["windows"], 6), dtype=torch.int32, device="cuda")
    if kind == "wide":
        s["table"] = ib.Table.from_codes128(*_wide_codes(case, spec, seq, seed), k)
    elif kind in ("panel", "serve"):
        joint = _joint(case, spec, seq, mask, seed)
        if kind == "panel":
            s["table"] = joint
        else:
            s["server"] = ib.Server(s["ref"], case["W"], k, iteration_launches=True)
            s["server"].add_panel(joint, release=True)
            s["asked"] = _requests(case, seed)
            joint.close()
    elif kind == "intersect":
        s["k"] = k
        s["a"] = _codes(case, spec, seq, mask, 2 * seed + 2)
        s["b"] = _codes(case, spec, seq, mask, 2 * seed + 3, 0.5)
    else:
        codes, n = _codes(case, spec, seq, mask, 2 * seed + 2)
        s["table"] = ib.Table.from_codes(codes, n, k, on_device=True)
    if kind == "packed":
        s["seq"], s["mask"] = seq.cpu().pin_memory(), mask.cpu().pin_memory()
    elif kind == "fasta":
        s["text"] = _fasta(spec, seq, mask, seed)
    elif kind == "noalloc":
        s["seq"], s["mask"] = seq, mask
    return s


def _plain(rows):
    """Window rows as numbers: start, end, total, observed, variations, distance."""
    return np.ascontiguousarray(rows).view(np.int32).reshape(rows.shape + (6,))


def run(s):
    kind, W = s["kind"], s["W"]
    if kind in ("scan", "wide"):
        return _plain(ib.scan(s["table"], s["ref"], W))
    if kind == "scan_async":
        ib.scan_async(s["table"], s["ref"], W, s["rows"], s["windows"], torch.cuda.current_stream().cuda_stream)
        return s["rows"]
    if kind == "packed":
        return _plain(ib.scan_packed(s["table"], s["seq"], s["mask"], s["lens"], W))
    if kind == "fasta":
        ref = ib.Reference.from_fasta(s["text"])
        rows = _plain(ib.scan(s["table"], ref, W))
        ref.free()
        return rows
    if kind == "panel":
        s["table"].scan_async(s["ref"], W, s["rows"], s["rows"].shape[0] * s["windows"],
                              torch.cuda.current_stream().cuda_stream)
        return s["rows"]
    if kind == "serve":
        server, done = s["server"], {}
        ids = [server.submit(*asked) for asked in s["asked"]]
        while len(done) < len(ids):
            for r in server.poll(len(ids), timeout_ms=-1):
                if r["status"]:
                    raise RuntimeError("request ended with status %d" % r["status"])
                done[r["request_id"]] = r["rows"]
        return _plain(np.concatenate([done[i] for i in ids]))
    if kind == "map":
        return ib.map_coverage(s["table"], s["ref"])
    if kind == "noalloc":
        ib.scan_noalloc(s["table"], s["seq"], s["mask"], s["lens"], W, s["rows"], s["windows"],
                        torch.cuda.current_stream().cuda_stream)
        return s["rows"]
    table = ib.Table.from_codes(*s["a"], s["k"], on_device=True)
    count = table.count_present(*s["b"], on_device=True)
    table.close()
    return count


def work(case):
    """Bytes: the reference at 2 bits and an N bit a base, each key of the table once at 2 bits a base (and the
    sample mask of a joint table's key), the rows or the coverage. Nothing here is a floating-point operation."""
    kind, k, n = case["kind"], case["k"], case["bases"]
    windows = ib.window_count(_lens(case), case["W"], k) if "W" in case else 0
    key = k / 4
    if kind == "intersect":
        return {"bytes": 8.0 * (1.1 * n + 0.55 * n) + key * 1.1 * n, "flops": 0}
    if kind == "serve":
        asked = sum(min(case["W"] * r[3], n) for r in _requests(case, 1))
        share = min(1.0, asked / n)
        return {"bytes": share * (0.375 * n + (key + 2) * n) + 24.0 * sum(r[3] for r in _requests(case, 1)), "flops": 0}
    if kind == "panel":
        union = n * (0.6 + 0.55 * sum(_present(case)))
        return {"bytes": 0.375 * n + (key + 2) * union + 24.0 * windows * case["samples"], "flops": 0}
    keys = 0.5 * n if kind == "wide" else 1.1 * n
    ref = n * 82 / 81 if kind == "fasta" else 0.375 * n
    return {"bytes": ref + key * keys + (1.0 * n if kind == "map" else 24.0 * windows), "flops": 0}


def exact(case, seed):
    """No output is a rounded number: all are whole and the same wherever they are computed."""
    return None
