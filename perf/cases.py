"""Timing cases of the mapper: what its users have it do, through its public entry points.

A case names a genome (size and kind), an index seed length, reads (count,
lengths, error rate), a threshold and the call that is timed:

  map     Mapper.map: a block of host reads, results in the reference's layout
  host    Mapper.submit + swm_map_wait_packed on page-locked host buffers (the
          block loop of an integration; every byte in and out is copied)
  device  Mapper.submit_device / wait_device on reads in device memory, then
          swm_map_fetch_packed into page-locked buffers
  serve   one request through Server.submit / Server.poll
  build   Index.build_device, then swm_index_download of all six arrays into
          page-locked buffers (what saving an index does before the files)

Genomes and reads are made on the GPU from the seed with the shapes of the
package's synthetic workloads (swmapper_gb300/synth.py): "uniform", "repeats"
(41% GC, 10% repeat copies of 300 bp-6 kb at 1% divergence) and "human" (41%
GC, 5% N runs, half of it repeat families at 2-15% divergence). All outputs
are whole numbers and bytes.
"""
import ctypes as C
import math

import numpy as np
import torch

import swmapper_gb300 as swm

KINDS = {
    "uniform": dict(gc=0.5),
    "repeats": dict(gc=0.41, repeat=0.10, copies=16, div=(0.01, 0.01)),
    "human": dict(gc=0.41, repeat=0.50, copies=400, div=(0.02, 0.15), n_frac=0.05),
}
LETTERS = (65, 67, 71, 84, 78)  # A C G T N
CHUNK = 1 << 26                 # bases made at a time


def _case(name, op, genome, kind, k=12, reads=0, lmin=0, lmax=0, err=0.0, e=0, block=0):
    """e = 0: each read's threshold is ceil(0.05 length); block: reads the mapper is made for."""
    c = dict(op=op, genome=genome, kind=kind, k=k, reads=reads, lmin=lmin, lmax=lmax, err=err, e=e,
             block=block or max(1, reads))
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a handful of reads looked up against a small genome: launches and round trips
        _case("map_16_reads_1mbp", "map", 1_000_000, "uniform", reads=16, lmin=100, lmax=100, err=0.02, e=5, block=4096),
        # the plain block of the reference's loop: 4,096 reads of 100 bp, 1 Mbp genome
        _case("map_4096_1mbp", "map", 1_000_000, "uniform", reads=4096, lmin=100, lmax=100, err=0.02, e=5),
        # a host loop over blocks against a bacterial-to-chromosome sized genome
        _case("host_65536_100mbp", "host", 100_000_000, "repeats", reads=65536, lmin=150, lmax=150, err=0.03, e=7),
        # throughput mapping of resident reads, the batched workload's block
        _case("device_524288_100mbp", "device", 100_000_000, "repeats", reads=524288, lmin=150, lmax=150, err=0.03, e=7),
        # trimmed reads of any length with a threshold each, an odd count
        _case("host_uneven_200003_100mbp", "host", 100_000_000, "repeats", reads=200_003, lmin=50, lmax=250, err=0.04),
        # another seed length (-s 13): the seed kernel of any k, no candidate table
        _case("host_k13_50000_100mbp", "host", 100_000_000, "repeats", k=13, reads=50_000, lmin=155, lmax=155,
              err=0.03, e=7),
        # one request of a server on a human-like genome (mean request of the serving workload)
        _case("serve_483_human1g", "serve", 1_000_000_000, "human", reads=483, lmin=50, lmax=250, err=0.03, block=65536),
        # the block size of a latency-minded loop on a human-like genome
        _case("host_4096_human1g", "host", 1_000_000_000, "human", reads=4096, lmin=150, lmax=150, err=0.03, e=7),
        # a full server block of uneven reads on the human-scale genome
        _case("host_uneven_65536_human3g", "host", 3_100_000_000, "human", reads=65536, lmin=50, lmax=250, err=0.03),
        # the headline: resident reads against the human-scale genome
        _case("device_524288_human3g", "device", 3_100_000_000, "human", reads=524288, lmin=150, lmax=150, err=0.03, e=7),
        # index build of a small genome, where the 4^k bucket arrays are most of it
        _case("build_5mbp", "build", 5_000_001, "repeats"),
        # index build of a genome with large repeat families
        _case("build_human1g", "build", 1_000_000_000, "human"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _kind(rng, n):
    """Genome kinds by size: uniform ones are small, human-like ones are not."""
    if n < 20_000_000:
        return rng.choice(["uniform", "repeats"])
    if n < 300_000_000:
        return rng.choice(["repeats", "repeats", "human"])
    return "human"


def _unit(c):
    """Rough cost of one read, in reads of 150 bp at e = 7 on the 100 Mbp genome."""
    L = 0.5 * (c["lmin"] + c["lmax"])
    e = c["e"] or math.ceil(0.05 * L)
    rep = 1 + 14 * c["genome"] / 3.1e9 if c["kind"] == "human" else 1
    return rep * max(0.2, L / 150) * (1 + e) / 8


def draw(rng):
    op = rng.choice(["map", "host", "host", "host", "device", "device", "serve", "build"])
    if op == "build":
        n = _log(rng, 1_000_000, 1_000_000_000)
        k = rng.choice([12, 12, 12, 11, 13]) if n < 200_000_000 else 12
        return _case("", "build", n, _kind(rng, n), k=k)
    k = rng.choice([12, 12, 12, 12, 10, 13, 14])
    n = _log(rng, 1_000_000, {10: 10_000_000, 12: 3_100_000_000, 13: 200_000_000, 14: 200_000_000}[k])
    if rng.random() < 0.5:
        # a library of one length, one that the read encoding (the reference's)
        # holds whole: it garbles the last bases of many others, and few of
        # those reads map
        lmin = lmax = rng.choice([L for L in range(4 * k + 7, min(251, 17 * (k + 3)), k + 3) if L % 16])
    else:
        lmin = rng.randint(40, 150)
        lmax = rng.randint(lmin + 60, 254)
    lmax = min(lmax, 17 * (k + 3) - 1)  # at most 16 seeds of k + 3 bases a read
    lmin = min(lmin, lmax)
    err = round(rng.uniform(0.005, 0.04), 4)
    few = math.ceil(err * lmax) + 1  # a threshold that most reads pass
    c = _case("", op, n, _kind(rng, n), k=k, reads=1, lmin=lmin, lmax=lmax, err=err,
              e=0 if rng.random() < 0.5 else rng.randint(few, max(few, min(14, lmin // 12))))
    top = {"map": 16384, "serve": 4096}.get(op, 524288)
    top = max(32, min(top, int(524288 * 8 / _unit(c))))
    c["reads"] = _log(rng, 16, top)
    c["block"] = 65536 if op == "serve" else c["reads"]
    return c


# ------------------------------------------------------------------ inputs

def _letters(codes, out):
    lut = torch.tensor(LETTERS, dtype=torch.uint8, device="cuda")
    for a in range(0, codes.numel(), CHUNK):
        torch.index_select(lut, 0, codes[a:a + CHUNK].int(), out=out[a:a + CHUNK])


def _background(codes, gc, gen):
    half = round(gc * 128)  # C below half, G below 2 half, then A / T evenly (of 256)
    mid = 2 * half + (256 - 2 * half) // 2
    for a in range(0, codes.numel(), CHUNK):
        u = torch.randint(0, 256, (min(CHUNK, codes.numel() - a),), dtype=torch.uint8, device="cuda", generator=gen)
        c = (u >= mid).to(torch.uint8).mul_(3)  # A 0, T 3
        c.masked_fill_(u < 2 * half, 2)
        c.masked_fill_(u < half, 1)
        codes[a:a + u.numel()] = c


def make_genome(n, kind, seed):
    """n bases as ASCII letters in device memory."""
    g = KINDS[kind]
    gen = torch.Generator("cuda").manual_seed(seed)
    codes = torch.empty(n, dtype=torch.uint8, device="cuda")
    _background(codes, g["gc"], gen)
    if g.get("repeat"):
        # families of `copies` diverged copies of a consensus, placed side by
        # side in random order with random gaps; they cover what copies thrown
        # at random places would
        lo, hi = 300, min(6000, max(301, n // 20))
        cover = 1 - math.exp(-g["repeat"])
        nfam = max(1, int(cover * n / ((lo + hi) / 2 * g["copies"])))
        flen = torch.randint(lo, hi + 1, (nfam,), device="cuda", generator=gen)
        foff = torch.cumsum(flen, 0) - flen
        cons = torch.empty(int(flen.sum()), dtype=torch.uint8, device="cuda")
        _background(cons, g["gc"], gen)
        fam = torch.arange(nfam, device="cuda").repeat_interleave(g["copies"])
        fam = fam[torch.randperm(fam.numel(), device="cuda", generator=gen)]
        clen = flen[fam]
        keep = torch.cumsum(clen, 0) <= cover * n
        fam, clen = fam[keep], clen[keep]
        gap = torch.rand(fam.numel() + 1, device="cuda", generator=gen, dtype=torch.float64)
        gap = (gap / gap.sum() * (n - int(clen.sum()))).long()[:-1]
        at = torch.cumsum(gap + clen, 0) - clen
        d0, d1 = g["div"]
        div = d0 + (d1 - d0) * torch.rand(fam.numel(), device="cuda", generator=gen)
        for a in range(0, fam.numel(), 8192):
            f, L, p, d = fam[a:a + 8192], clen[a:a + 8192], at[a:a + 8192], div[a:a + 8192]
            first = torch.cumsum(L, 0) - L
            within = torch.arange(int(L.sum()), device="cuda") - first.repeat_interleave(L)
            b = cons[foff[f].repeat_interleave(L) + within]
            mut = torch.rand(b.numel(), device="cuda", generator=gen) < d.repeat_interleave(L)
            other = torch.randint(1, 4, (b.numel(),), dtype=torch.uint8, device="cuda", generator=gen)
            codes[p.repeat_interleave(L) + within] = torch.where(mut, (b + other) & 3, b)
    if g.get("n_frac"):
        left = int(g["n_frac"] * n)
        while left > 0:
            r = torch.rand(256, 2, generator=gen, device="cuda").tolist()
            for u, v in r:
                run = min(left, int(10_000 + u * min(990_000, n / 50)))
                p = int(v * (n - run))
                codes[p:p + run] = 4
                left -= run
                if left <= 0:
                    break
    seq = torch.empty_like(codes)
    _letters(codes, seq)
    return seq


def make_reads(seq, nreads, lmin, lmax, err, seed):
    """(reads[nreads, lmax] letters, lens) on the GPU: both strands, err of the
    bases wrong (70% substituted, 15% inserted, 15% deleted)."""
    gen = torch.Generator("cuda").manual_seed(seed)
    n = seq.numel()
    lens = torch.randint(lmin, lmax + 1, (nreads,), device="cuda", generator=gen)
    start = torch.randint(0, n - 2 * lmax - 16, (nreads,), device="cuda", generator=gen)
    for _ in range(6):  # few reads lie in N runs
        bad = (seq[start] == 78) | (seq[start + lmax] == 78)
        start = torch.where(bad, torch.randint(0, n - 2 * lmax - 16, (nreads,), device="cuda", generator=gen), start)
    out = torch.zeros(nreads, lmax, dtype=torch.uint8, device="cuda")
    lut = torch.tensor(LETTERS, dtype=torch.uint8, device="cuda")
    step = 65536
    for a in range(0, nreads, step):
        s, L = start[a:a + step], lens[a:a + step]
        u = torch.rand(s.numel(), lmax, device="cuda", generator=gen)
        rnd = torch.randint(0, 4, u.shape, dtype=torch.uint8, device="cuda", generator=gen)
        sub, ins, dele = u < 0.7 * err, (u >= 0.7 * err) & (u < 0.85 * err), (u >= 0.85 * err) & (u < err)
        adv = 1 + dele.int() - ins.int()
        src = s[:, None] + torch.cumsum(adv, 1) - adv + dele
        b = seq[src]
        b = torch.where(sub | ins, lut[rnd.int()], b)
        rev = torch.rand(s.numel(), device="cuda", generator=gen) < 0.5
        j = torch.arange(lmax, device="cuda")[None, :].expand_as(b)
        inside = j < L[:, None]
        back = torch.gather(b, 1, (L[:, None] - 1 - j).clamp_(min=0))
        comp = back.clone()
        for x, y in ((65, 84), (84, 65), (67, 71), (71, 67)):
            comp.masked_fill_(back == x, y)
        b = torch.where(rev[:, None], comp, b)
        out[a:a + step] = b * inside
    return out, lens.int()


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _pinned_zeros(n, dtype):
    return torch.zeros(n, dtype=dtype, pin_memory=True).numpy()


class PinnedResults:
    """Page-locked packed result buffers of one block (swm_packed_result)."""

    def __init__(self, nreads):
        self.words = _pinned_zeros(20 * nreads + 16384, torch.int32)
        self.cigar = _pinned_zeros(160 * nreads + 65536, torch.uint8)
        self.rlen = _pinned_zeros(3 * nreads + 1024, torch.int32)
        self.unmapped = _pinned_zeros(nreads, torch.int32)
        self.c = swm.PackedResult(self.words.ctypes.data, self.cigar.ctypes.data, self.rlen.ctypes.data,
                                  self.unmapped.ctypes.data, self.words.size, self.cigar.size, self.rlen.size,
                                  self.unmapped.size, 0, 0, 0, 0)


def _packed(b):
    """The results in buffers b, whole (they are zero past the counts)."""
    c = b.c
    return dict(words=b.words.view(np.int32), cigar=b.cigar, record_cigar_len=b.rlen.view(np.int32),
                unmapped=b.unmapped.view(np.int32), n_words=c.n_words, n_cigar=c.n_cigar, n_records=c.n_records,
                n_unmapped=c.n_unmapped)


def prepare(case, seed):
    c = dict(case)
    seq = make_genome(c["genome"], c["kind"], seed)
    s = dict(op=c["op"], k=c["k"], e=c["e"] or 0)
    if c["op"] == "build":
        s["seq"] = seq
        nb, S, W = 1 << (2 * c["k"]), c["genome"] // 4 + 1, (c["genome"] + 31) // 32
        i32 = torch.int32
        s["bufs"] = dict(hash_count=_pinned_zeros(nb, i32), hash_offset=_pinned_zeros(nb + 1, i32),
                         positions=_pinned_zeros(S, i32), pos_lseeds=_pinned_zeros(S, torch.int16),
                         base_2bits=_pinned_zeros(2 * W, i32), base_3bits=_pinned_zeros(W, i32))
        torch.cuda.empty_cache()
        return s
    reads, lens = make_reads(seq, c["reads"], c["lmin"], c["lmax"], c["err"], seed + 1)
    per_read = None if c["e"] else (lens + 19) // 20  # ceil(0.05 L)
    torch.cuda.synchronize()
    s["index"] = swm.Index.build_device(seq.data_ptr(), seq.numel(), k=c["k"])
    del seq
    if c["op"] == "device":
        s["reads"], s["lens"] = reads, lens
        s["per_read"] = None if per_read is None else per_read.to(torch.uint8)
    else:
        move = _pinned if c["op"] == "host" else torch.Tensor.cpu
        s["reads"], s["lens"] = move(reads).numpy(), move(lens).numpy().view(np.uint32)
        s["per_read"] = None if per_read is None else move(per_read.to(torch.uint8)).numpy()
    torch.cuda.empty_cache()
    if c["op"] == "serve":
        s["server"] = swm.Server(s["index"], block_reads=c["block"], max_slots=1)
    else:
        s["mapper"] = swm.Mapper(s["index"], max_reads=c["block"])
    if c["op"] in ("host", "device"):
        s["out"] = PinnedResults(c["reads"])
    return s


def _ok(rc):
    if rc != 0:
        raise swm.SwmError(swm.lib().swm_last_error().decode(), rc)


def run(s):
    op = s["op"]
    if op == "map":
        r = s["mapper"].map(s["reads"], s["lens"], s["e"], errors_per_read=s["per_read"])
        # the buffers the records are views of: zero past them
        return dict(records=r.ref_pos.base.view(np.int32), cigar=r.cigar.base, unmapped=r.unmapped.base.view(np.int32),
                    n_records=r.ref_pos.shape[0], n_unmapped=r.unmapped.shape[0])
    if op == "host":
        s["mapper"].submit(s["reads"], s["lens"], s["e"], errors_per_read=s["per_read"])
        return _packed(s["mapper"].wait_packed(s["out"]))
    if op == "device":
        m, pr = s["mapper"], s["per_read"]
        m.submit_device(s["reads"].data_ptr(), s["lens"].data_ptr(), s["reads"].shape[1], s["reads"].shape[0], s["e"],
                        None if pr is None else pr.data_ptr())
        m.wait_device()
        _ok(swm.lib().swm_map_fetch_packed(m._h, C.byref(s["out"].c)))
        return _packed(s["out"])
    if op == "serve":
        v = s["server"]
        v.submit(s["reads"], s["lens"], s["e"], errors_per_read=s["per_read"])
        v.poll(records=False)
        return _packed(v.last)
    ix = swm.Index.build_device(s["seq"].data_ptr(), s["seq"].numel(), k=s["k"])
    b = s["bufs"]
    _ok(swm.lib().swm_index_download(ix._h, *(a.ctypes.data for a in b.values())))
    n_seeds = ix.info().n_seeds
    ix.close()
    return dict(b, n_seeds=n_seeds)


def exact(case, seed):
    """Every output is a whole number or a byte: there is no rounding to measure."""
    return None


def work(case):
    """Bytes: each read in, the bucket range of each of its seeds, the surviving
    positions and the genome windows of its candidates, the records out; for a
    build, the bases in and the six arrays out. flops: integer operations, 21
    per read base of the bit-parallel alignment (16 bases rule a candidate out
    at the earliest, a passing one takes all of them)."""
    c = case
    if c["op"] == "build":
        n, nb = c["genome"], 1 << (2 * c["k"])
        return {"bytes": n + 8 * nb + 6 * (n // 4) + 12 * (n // 32), "flops": 4 * n}
    L = 0.5 * (c["lmin"] + c["lmax"])
    e = c["e"] or math.ceil(0.05 * L)
    nl = int(L // (c["k"] + 3))
    sel = min(nl, e + 1) * 4
    # candidates per read: chance hits of 15-mers on both strands, the true
    # place, and (human) the other copies of its family
    chance = 2 * sel * (c["genome"] / 4) / 4 ** (c["k"] + 3)
    cand = 1.5 + chance + (90 * c["genome"] / 3.1e9 * sel / 32 if c["kind"] == "human" else 0)
    per = (L + 4) + 2 * 4 * nl * 8 + cand * (4 + (L + 2 * e) / 4) + 24
    return {"bytes": c["reads"] * per, "flops": c["reads"] * 21 * (cand * 16 + L)}
