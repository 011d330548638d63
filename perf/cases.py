"""Work that a variant-calling program hands to this library, for measuring it.

Every path takes host data and returns host data, as the callers in a HaplotypeCaller-like program have
it: likelihoods of one active region (``call_pairhmm``, ``schedule_pairhmm``), of a batch of regions
(``Engine.compute``), region requests kept in flight on the serving loop (``Engine.submit_region``) and
Smith-Waterman alignments (``Engine.sw_align``).  Sizes are those of ``rovaca_b200.synth``'s
configurations and of the library's limits (reads up to 768 bases, haplotypes up to 1536).

A case is a dict of plain values:
  path      call | schedule | compute | serve | align
  regions   active regions in one pass (align: regions whose reads are aligned)
  reads, haps          [lo, hi] of the reads and haplotypes of a region, as two keys each
  depth     uniform: reads drawn in [reads_lo, reads_hi]; lognormal: around 60 as in whole-genome data
  read_lo/hi, hap_lo/hi  lengths;  qual_lo/hi  base qualities;  err  substitution rate
  indels_lo/hi         short indels of a haplotype against the reference window
  gaps      flat: 45/45/10 for every base; per_base: recalibrated indel qualities, one per base
  n_rate    share of reads that hold an N;  flags  pair flags wanted as well
  pcr       PCR indel model of the region API (call, serve)
  params    genotyping | assembly (align)
"""
from __future__ import annotations

import math
import zlib

import numpy as np

from rovaca_b200 import pairhmm
from rovaca_b200 import sw as smith_waterman

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)

BASE = {
    "path": "compute", "regions": 1, "reads_lo": 10, "reads_hi": 500, "depth": "uniform", "haps_lo": 2, "haps_hi": 32,
    "read_lo": 100, "read_hi": 250, "hap_lo": 150, "hap_hi": 600, "qual_lo": 2, "qual_hi": 41, "err": 0.01,
    "indels_lo": 0, "indels_hi": 2, "gaps": "flat", "n_rate": 0.0, "flags": False, "pcr": "CONSERVATIVE",
    "params": "genotyping",
}


def _case(**kw) -> dict:
    return {**BASE, **kw}


def listed() -> list[dict]:
    return [
        # one region of a whole-genome run through the HaplotypeCaller entry point: a thread of the
        # region pool that calls and waits, the smallest call there is
        _case(name="call_region", path="call", reads_lo=40, reads_hi=40, read_lo=150, read_hi=150, haps_lo=6, haps_hi=6,
              hap_lo=300, hap_hi=400, qual_lo=15, qual_hi=40, err=0.004),
        # one region through the vector interface, a deep one: the reference's own test driver
        _case(name="schedule_region", path="schedule", reads_lo=250, reads_hi=250, haps_lo=16, haps_hi=16),
        # a handful of regions gathered by one caller
        _case(name="batch_8", regions=8),
        # a full batch of targeted-sequencing regions (the benchmark's shape)
        _case(name="batch_1000", regions=1000),
        # recalibrated indel qualities (one per base), some reads with an N, pair flags asked for
        _case(name="batch_per_base_gaps", regions=150, gaps="per_base", n_rate=0.1, flags=True),
        # long reads (merged pairs, up to the limits) against long haplotypes
        _case(name="batch_long_reads", regions=24, reads_lo=20, reads_hi=200, read_lo=257, read_hi=768, haps_lo=2,
              haps_hi=16, hap_lo=800, hap_hi=1536),
        # low base qualities and divergent haplotypes: most pairs underflow single precision
        _case(name="batch_low_quality", regions=60, reads_lo=200, reads_hi=200, read_lo=250, read_hi=250, haps_lo=16,
              haps_hi=16, hap_lo=800, hap_hi=1000, qual_lo=2, qual_hi=15, err=0.05, indels_lo=5, indels_hi=10),
        # whole-genome depth: many small regions of reads of 150 bases
        _case(name="batch_genome", regions=1500, depth="lognormal", reads_lo=5, reads_hi=2000, read_lo=150, read_hi=150,
              haps_lo=1, haps_hi=12, hap_lo=200, hap_hi=1200),
        # regions of a whole-genome run as requests in flight: likelihoods, genotyping of two events
        # and realignment of the kept reads in one request each
        _case(name="serve_100", path="serve", regions=100, reads_lo=20, reads_hi=100, read_lo=150, read_hi=150, haps_lo=2,
              haps_hi=8, hap_lo=300, hap_hi=400, qual_lo=15, qual_hi=40, err=0.004),
        # realignment of one region's reads
        _case(name="align_region", path="align", reads_lo=64, reads_hi=64, haps_lo=8, haps_hi=8),
        # realignment of the reads of many regions
        _case(name="align_300", path="align", regions=300),
        # alignment of assembled haplotypes to their reference windows with the assembly parameters:
        # both sequences of one length, 32-bit scores
        _case(name="align_assembly", path="align", regions=150, reads_lo=4, reads_hi=32, read_lo=300, read_hi=760,
              haps_lo=1, haps_hi=1, hap_lo=500, hap_hi=1000, err=0.002, params="assembly"),
    ]


def draw(rng) -> dict:
    """One more case of these ranges; the costliest stays below batch_1000."""

    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    def lengths(lo, hi, step=1.4):
        a = rng.randint(lo, hi)
        return a, min(hi, int(a * rng.uniform(1.0, step)))

    path = rng.choice(["call", "schedule", "compute", "compute", "compute", "serve", "align", "align"])
    read = lengths(60, 300, 2.0)
    hap = lengths(max(150, read[0]), 700, 2.0)
    reads = log(10, 500)
    haps = log(1, 32)
    c = _case(path=path, reads_lo=max(1, reads // 2), reads_hi=reads, haps_lo=max(1, haps // 2), haps_hi=haps,
              read_lo=read[0], read_hi=read[1], hap_lo=hap[0], hap_hi=hap[1], qual_lo=rng.choice([2, 6, 10]),
              qual_hi=rng.choice([38, 40, 41]), err=round(rng.uniform(0.002, 0.02), 4), flags=rng.random() < 0.3)
    if path == "compute":
        kind = rng.choice(["flat", "per_base", "long", "low_quality", "genome"])
        c["regions"] = log(2, 400)
        if kind == "per_base":
            c.update(gaps="per_base", n_rate=rng.choice([0.0, 0.05, 0.3]), regions=log(2, 300))
        elif kind == "long":
            read = lengths(257, 768)
            hap = lengths(800, 1536)
            c.update(read_lo=read[0], read_hi=read[1], hap_lo=hap[0], hap_hi=hap[1], regions=log(2, 20),
                     reads_lo=10, reads_hi=log(20, 200), haps_lo=2, haps_hi=log(2, 16))
        elif kind == "low_quality":
            c.update(read_lo=150, read_hi=250, hap_lo=600, hap_hi=1000, qual_hi=15, qual_lo=2, err=0.05, indels_lo=5,
                     indels_hi=10, regions=log(2, 50), reads_lo=50, reads_hi=200, haps_lo=4, haps_hi=16)
        elif kind == "genome":
            c.update(depth="lognormal", reads_lo=5, reads_hi=2000, haps_lo=1, haps_hi=12, hap_lo=200, hap_hi=1200,
                     regions=log(20, 1500), read_lo=read[0], read_hi=read[0])
    elif path == "serve":
        c.update(regions=log(8, 150), reads_lo=10, reads_hi=log(20, 150), haps_lo=2, haps_hi=rng.randint(2, 12),
                 pcr=rng.choice(["CONSERVATIVE", "NONE"]), qual_lo=rng.randint(12, 20), err=0.004, flags=False)
    elif path == "call":
        c.update(pcr=rng.choice(["CONSERVATIVE", "AGGRESSIVE", "NONE"]), qual_lo=rng.randint(12, 20), err=0.004, flags=False)
    elif path == "schedule":
        c.update(gaps=rng.choice(["flat", "per_base"]), flags=False)
    else:
        c["flags"] = False
        c["regions"] = log(1, 400)
        if rng.random() < 0.35:
            hap = lengths(300, 1400)
            c.update(regions=log(1, 120), params="assembly", read_lo=max(100, hap[0] // 2), read_hi=max(200, hap[0] * 3 // 4),
                     reads_lo=1, reads_hi=log(2, 32), haps_lo=1, haps_hi=1, hap_lo=hap[0], hap_hi=hap[1], err=0.002)
    return c


# ---- inputs -----------------------------------------------------------------------------------


def _edited(rng, seq, n_snp, n_indel):
    s = seq.copy()
    pos = rng.integers(0, len(s), n_snp)
    s[pos] = (s[pos] + rng.integers(1, 4, n_snp)) % 4
    for _ in range(n_indel):
        p, ln = int(rng.integers(1, len(s) - 12)), int(rng.integers(1, 11))
        s = np.concatenate([s[:p], rng.integers(0, 4, ln).astype(np.uint8), s[p:]] if rng.random() < 0.5 else [s[:p], s[p + ln:]])
    return s


def _sizes(c: dict) -> list[tuple[int, int, np.ndarray]]:
    """Haplotypes, window length and read lengths of every region: they belong to the case, the sequences
    and qualities to the seed."""
    size = np.random.default_rng(zlib.crc32(repr([c[k] for k in sorted(BASE)]).encode()))
    out = []
    for _ in range(c["regions"]):
        n_reads = int(size.integers(c["reads_lo"], c["reads_hi"] + 1))
        if c["depth"] == "lognormal":
            n_reads = int(np.clip(round(60 * math.exp(0.5 * size.standard_normal())), c["reads_lo"], c["reads_hi"]))
        n_haps = int(size.integers(c["haps_lo"], c["haps_hi"] + 1))
        length = int(size.integers(c["hap_lo"], c["hap_hi"] + 1))
        out.append((n_haps, length, size.integers(c["read_lo"], c["read_hi"] + 1, n_reads)))
    return out


def _regions(c: dict, seed: int) -> list[dict]:
    """The case's regions: a random reference window, haplotypes that are edits of it, reads sampled from
    the haplotypes (running on into the reference flank) with substitution errors."""
    rng = np.random.default_rng([seed, 77])
    out = []
    for n_haps, length, rl in _sizes(c):
        n_reads = len(rl)
        ref = rng.integers(0, 4, length + 768 + 200).astype(np.uint8)
        haps = [_edited(rng, ref[:length], int(rng.integers(0, 4)), int(rng.integers(c["indels_lo"], c["indels_hi"] + 1)))[:1536]
                for _ in range(n_haps)]
        ext = np.stack([np.concatenate([h, ref[length:]])[:length + 768] for h in haps])
        src = rng.integers(0, n_haps, n_reads)
        start = (rng.random(n_reads) * np.maximum(np.array([len(h) for h in haps])[src] - rl + 1, 1)).astype(np.int64)
        off = np.concatenate([[0], np.cumsum(rl)])
        tot = int(off[-1])
        within = np.arange(tot) - np.repeat(off[:-1], rl)
        bases = ext[np.repeat(src, rl), np.repeat(start, rl) + within]
        bases = ACGT[np.where(rng.random(tot) < c["err"], (bases + rng.integers(1, 4, tot)) % 4, bases)].copy()
        if c["n_rate"]:
            for r in np.nonzero(rng.random(n_reads) < c["n_rate"])[0]:
                bases[off[r] + int(rng.integers(0, rl[r]))] = ord("N")
        qual = rng.integers(c["qual_lo"], c["qual_hi"] + 1, tot).astype(np.uint8)
        if c["gaps"] == "per_base":
            gaps = [rng.integers(30, 46, tot).astype(np.uint8), rng.integers(30, 46, tot).astype(np.uint8),
                    rng.integers(8, 13, tot).astype(np.uint8)]
        else:
            gaps = [np.full(tot, q, np.uint8) for q in (45, 45, 10)]
        out.append({"haps": [ACGT[h] for h in haps], "bases": bases, "off": off, "qual": qual, "gaps": gaps})
    return out


def _packed(regs: list[dict]) -> pairhmm.PackedBatch:
    cat = lambda key: np.concatenate([r[key] for r in regs])
    gap = lambda k: np.concatenate([r["gaps"][k] for r in regs])
    hl = [len(h) for r in regs for h in r["haps"]]
    rl = np.concatenate([np.diff(r["off"]) for r in regs])
    return pairhmm.PackedBatch(
        np.array([len(r["haps"]) for r in regs], np.uint32), np.array([len(r["off"]) - 1 for r in regs], np.uint32),
        np.concatenate([h for r in regs for h in r["haps"]]), np.concatenate([[0], np.cumsum(hl)]).astype(np.uint64),
        cat("bases"), cat("qual"), gap(0), gap(1), gap(2), np.concatenate([[0], np.cumsum(rl)]).astype(np.uint64))


def _split(reg: dict, a: np.ndarray) -> list[bytes]:
    return [a[s:e].tobytes() for s, e in zip(reg["off"][:-1], reg["off"][1:])]


def _events(reg: dict) -> list:
    """Two events of a region: the haplotypes split by parity, and by halves into up to three alleles."""
    m = len(reg["haps"])
    h = np.arange(m)
    return [(2, (h % 2).astype(np.int8)), (min(m, 3), (h * min(m, 3) // m).astype(np.int8))]


def prepare(case: dict, seed: int) -> dict:
    c = {**BASE, **case}
    regs = _regions(c, seed)
    s = {"case": c, "engine": pairhmm.default_engine()}
    if c["path"] == "compute":
        s["batch"] = _packed(regs).pinned()
        n = s["batch"].out_size
        import torch

        s["keep"] = torch.empty(n, dtype=torch.float64, pin_memory=True)
        s["out"] = s["keep"].numpy()
        s["flags"] = np.zeros(n, np.uint8) if c["flags"] else None
    elif c["path"] == "align":
        batch = _packed(regs)
        nh, nr = batch.n_haps.astype(np.int64), batch.n_reads.astype(np.int64)
        items = np.zeros(int(nr.sum()), smith_waterman.SW_ITEM_DTYPE)
        g = np.repeat(np.arange(len(nr)), nr)
        hap = np.concatenate([[0], np.cumsum(nh)])[g] + np.random.default_rng([seed, 78]).integers(0, 1 << 30, len(g)) % nh[g]
        items["hap_offset"], items["hap_len"] = batch.hap_off[hap], (batch.hap_off[hap + 1] - batch.hap_off[hap])
        items["read_offset"], items["read_len"] = batch.read_off[:-1], np.diff(batch.read_off)
        s["pairs"] = smith_waterman.SwBatch(batch.hap_bases, batch.read_bases, items)
        s["params"] = smith_waterman.ASSEMBLY if c["params"] == "assembly" else smith_waterman.GENOTYPING
    else:
        s["regions"] = [{"haps": [h.tobytes() for h in r["haps"]], "reads": _split(r, r["bases"]), "qual": _split(r, r["qual"]),
                         "gaps": [_split(r, g) for g in r["gaps"]], "mapq": np.full(len(r["off"]) - 1, 60, np.uint8),
                         "events": _events(r), "priority": -np.arange(len(r["haps"]), dtype=np.float64)} for r in regs]
    if c["path"] in ("align", "serve"):
        s["cigars"] = np.zeros(12 * sum(len(r["off"]) - 1 for r in regs), np.uint32)
    return s


def _kept_cigars(s: dict, parts: list[np.ndarray]) -> np.ndarray:
    """The compact CIGAR operations in the program's own buffer, zeros after the last."""
    buf, at = s["cigars"], 0
    for p in parts:
        p = p[:len(buf) - at]
        buf[at:at + len(p)] = p
        at += len(p)
    buf[at:] = 0
    return buf


def run(s: dict):
    c, eng = s["case"], s["engine"]
    if c["path"] == "compute":
        out, flags, _ = eng.compute(s["batch"], want_flags=c["flags"], out=s["out"], flags=s["flags"])
        return {"likelihoods": out, "flags": flags}
    if c["path"] == "align":
        r = eng.sw_align(s["pairs"], s["params"])
        return {"fields": [r.fields[f] for f in r.fields.dtype.names], "cigars": _kept_cigars(s, [r.cigars])}
    if c["path"] == "schedule":
        r = s["regions"][0]
        return {"likelihoods": pairhmm.schedule_pairhmm(r["haps"], r["reads"], r["qual"], *r["gaps"], engine=eng)[1]}
    if c["path"] == "call":
        r = s["regions"][0]
        matrix, kept = pairhmm.call_pairhmm(r["haps"], r["reads"], r["qual"], r["mapq"], pcr_option=c["pcr"], engine=eng)
        mask = np.zeros(matrix.shape[1], bool)
        mask[kept] = True
        return {"likelihoods": matrix, "kept": mask}
    tickets = [eng.submit_region(r["haps"], r["reads"], r["qual"], r["mapq"], pcr_option=c["pcr"], events=r["events"],
                                 realign={"priority": r["priority"]}) for r in s["regions"]]
    got = []
    for t in tickets:
        matrix, keep = t.wait()
        got.append((matrix, keep, t.genotypes(), t.realignment()))
    cat = np.concatenate
    return {
        "likelihoods": cat([m.reshape(-1) for m, _, _, _ in got]), "keep": cat([k for _, k, _, _ in got]),
        "genotypes": cat([gl for _, _, ev, _ in got for gl, _, _ in ev]),
        "best": np.array([b for _, _, ev, _ in got for _, b, _ in ev]), "best_haplotype": cat([al[0] for *_, al in got]),
        "fields": [cat([al[1].fields[f] for *_, al in got]) for f in smith_waterman.SW_RESULT_DTYPE.names],
        "cigars": _kept_cigars(s, [al[1].cigars for *_, al in got]),
    }


# ---- what a pass cannot do without ---------------------------------------------------------------


def _cells(c: dict) -> float:
    return float(sum(m * length * int(rl.sum()) for m, length, rl in _sizes(c)))


def work(case: dict) -> dict:
    """Bytes and operations of one pass: a likelihood cell is 4 multiply-adds and 4 multiplies (12
    operations), an alignment cell 4 adds, 4 maxima and 2 compares.  A region's haplotypes count with the
    length of its window."""
    c = {**BASE, **case}
    sizes = _sizes(c)
    align_cells = float(sum(length * int(rl.sum()) for _, length, rl in sizes))
    align_bytes = float(sum(m * length + int(rl.sum()) + len(rl) * (24 + 24 + 16) for m, length, rl in sizes))
    if c["path"] == "align":
        return {"bytes": align_bytes, "flops": 10.0 * align_cells}
    per_base = 5 if c["path"] in ("compute", "schedule") else 2
    per_pair = 9 if c["flags"] else 8
    w = {"bytes": float(sum(per_base * int(rl.sum()) + m * length + len(rl) * m * per_pair for m, length, rl in sizes)),
         "flops": 12.0 * _cells(c)}
    if c["path"] == "serve":
        w["bytes"] += align_bytes
        w["flops"] += 10.0 * align_cells
    return w


# ---- the same in 64 bits ------------------------------------------------------------------------


def _log10_likelihoods(regs: list[dict]) -> list[np.ndarray]:
    """[haps][reads] of every region: the pair-HMM forward algorithm in double precision, one
    anti-diagonal at a time over blocks of pairs of similar size."""
    import torch

    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pairs = [(g, h, r) for g, reg in enumerate(regs) for h in range(len(reg["haps"])) for r in range(len(reg["off"]) - 1)]
    rlen = [np.diff(reg["off"]) for reg in regs]
    R = np.array([rlen[g][r] for g, _, r in pairs])
    H = np.array([len(regs[g]["haps"][h]) for g, h, _ in pairs])
    order = np.argsort(R * 4096 + H, kind="stable")
    total = np.zeros(len(pairs))
    at = 0
    while at < len(order):
        rmax_guess = int(R[order[min(len(order), at + 1) - 1]])
        take = order[at:at + max(64, 40_000_000 // max(rmax_guess, 1))]
        at += len(take)
        P, rmax, hmax = len(take), int(R[take].max()), int(H[take].max())
        rows = np.zeros((5, P, rmax + 1), np.uint8)  # base, quality, insertion, deletion, continuation of row i at i
        hrev = np.zeros((P, hmax + 2 * rmax + 2), np.uint8)  # haplotype reversed: base j at hmax + rmax - j
        wild = np.zeros(P, bool)
        cols = {}
        for k, q in enumerate(take):
            g, h, r = pairs[q]
            reg = regs[g]
            a, b = reg["off"][r], reg["off"][r + 1]
            if (g, r) not in cols:
                cols[(g, r)] = (np.stack([x[a:b] for x in (reg["bases"], reg["qual"], *reg["gaps"])]), bool((reg["bases"][a:b] == 78).any()))
            rows[:, k, 1:b - a + 1] = cols[(g, r)][0]
            hb = reg["haps"][h]
            hrev[k, hmax + rmax - len(hb):hmax + rmax] = hb[::-1]
            wild[k] = cols[(g, r)][1] or bool((hb == 78).any())
        t = torch.from_numpy(rows).to(dev)
        hr = torch.from_numpy(hrev).to(dev)
        w = torch.from_numpy(wild).to(dev)[:, None]
        ph = torch.pow(10.0, -torch.arange(256, dtype=torch.float64, device=dev) / 10.0)
        err, pi, pd, pc = (ph[t[k].long()] for k in range(1, 5))
        mm, gm = 1.0 - pi - pd, 1.0 - pc
        hit, miss = 1.0 - err, err / 3.0
        rd = t[0]
        Rt, Ht = torch.from_numpy(R[take]).to(dev), torch.from_numpy(H[take]).to(dev)
        c0 = 2.0 ** 1020
        z = lambda: torch.zeros(P, rmax + 1, dtype=torch.float64, device=dev)
        M1, I1, D1, M2, I2, D2 = (z() for _ in range(6))
        top = c0 / Ht.double()
        D1[:, 0] = top
        D2[:, 0] = top
        acc = torch.zeros(P, dtype=torch.float64, device=dev)
        pick = Rt.long()[:, None]
        for d in range(2, rmax + hmax + 1):
            n = min(d - 1, rmax)
            i = slice(1, n + 1)
            u = slice(0, n)
            hb = hr[:, hmax + rmax - d + 1:hmax + rmax - d + 1 + n]  # base j - 1 = d - i - 1
            same = (rd[:, i] == hb) | (w & ((rd[:, i] == 78) | (hb == 78)))
            M, I, D = z(), z(), z()
            M[:, i] = torch.where(same, hit[:, i], miss[:, i]) * (M2[:, u] * mm[:, i] + (I2[:, u] + D2[:, u]) * gm[:, i])
            I[:, i] = M1[:, u] * pi[:, i] + I1[:, u] * pc[:, i]
            D[:, i] = M1[:, i] * pd[:, i] + D1[:, i] * pc[:, i]
            D[:, 0] = top
            j = d - Rt
            acc += torch.where((j >= 1) & (j <= Ht), (M.gather(1, pick) + I.gather(1, pick))[:, 0], 0.0)
            M2, I2, D2, M1, I1, D1 = M1, I1, D1, M, I, D
        total[take] = (torch.log10(acc) - math.log10(c0)).cpu().numpy()
    out, at = [], 0
    for g, reg in enumerate(regs):
        m, n = len(reg["haps"]), len(reg["off"]) - 1
        out.append(total[at:at + m * n].reshape(m, n))
        at += m * n
    return out


_PCR_CAPS = {
    "AGGRESSIVE": [40, 40, 40, 39, 39, 39, 38, 38, 37, 37, 36, 35, 34, 33, 32, 30, 28, 26, 23, 20, 17],
    "CONSERVATIVE": [40, 40, 40, 40, 39, 39, 39, 39, 39, 38, 38, 38, 37, 37, 37, 36, 36, 35, 34, 33, 33],
}


def _repeat_length(s: bytes, o: int) -> int:
    """Copies of the shortest unit (of up to 8 bases) that repeats from o + 1 on, with those that end at o."""
    unit, copies = s[o + 1:o + 2], 1
    for k in range(1, 9):
        if o + k + 1 > len(s):
            break
        u, n = s[o + 1:o + 1 + k], 0
        while s[o + 1 + n * k:o + 1 + (n + 1) * k] == u:
            n += 1
        copies = n
        if n > 1:
            unit = u
            break
    back, e = 0, o + 1
    while e >= len(unit) and s[e - len(unit):e] == unit:
        back, e = back + 1, e - len(unit)
    return min(20, copies + back)


def _region_call(c: dict, reg: dict) -> dict:
    """The region with its reads as the region interface prepares them (threshold 18, mapping quality 60)."""
    q = np.minimum(reg["qual"], 60)
    gap = np.full(len(q), 45, np.uint8)
    if c["pcr"] != "NONE":
        caps = _PCR_CAPS[c["pcr"]]
        for a, b in zip(reg["off"][:-1], reg["off"][1:]):
            s = reg["bases"][a:b].tobytes()
            for i in range(len(s) - 1):
                gap[a + i] = min(gap[a + i], caps[_repeat_length(s, i)])
    return {**reg, "qual": np.where(q < 18, 6, q).astype(np.uint8), "gaps": [gap, gap, np.full(len(q), 10, np.uint8)]}


def _kept_first(reg: dict, lk: np.ndarray) -> np.ndarray:
    best = lk.max(axis=0)
    lk = np.maximum(lk, best - 4.5)
    keep = best >= -4.0 * np.minimum(2.0, np.ceil(np.diff(reg["off"]) * 0.02))
    out = np.full(lk.shape, np.nan)
    out[:, :int(keep.sum())] = lk[:, keep]
    return out


def exact(case: dict, seed: int):
    c = {**BASE, **case}
    if c["path"] == "align" or _cells(c) > 1.5e10:
        return None  # whole numbers only, or too many cells for a plain implementation
    regs = _regions(c, seed)
    if c["path"] == "compute":
        return {"likelihoods": np.concatenate([x.reshape(-1) for x in _log10_likelihoods(regs)]), "flags": None}
    if c["path"] == "schedule":
        return {"likelihoods": np.ascontiguousarray(_log10_likelihoods(regs)[0].T)}
    regs = [_region_call(c, r) for r in regs]
    lk = [_kept_first(r, x) for r, x in zip(regs, _log10_likelihoods(regs))]
    if c["path"] == "call":
        return {"likelihoods": lk[0], "kept": None}
    return {"likelihoods": np.concatenate([x.reshape(-1) for x in lk]), "keep": None, "genotypes": None, "best": None,
            "best_haplotype": None, "fields": [None] * 6, "cigars": None}
