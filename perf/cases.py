"""Performance cases: what programs that use this library have it do, through its entry points.

listed() names the cases, draw() makes more of the same ranges, prepare() makes the inputs and the
handles that a program keeps (an open index, a server), run() is one pass, work() counts the bytes
that a pass cannot do without, and exact() gives the computed numbers in 64 bits.

An index (and the server attached to it) is opened once per process and kept, as a program that
classifies many batches does; the reads of a case come from its seed alone. The reference sets and
the reads have the shapes of mirage_b200.synth's workloads, generated on the GPU:

* ``small``   200 references of 5 kb (synth's ``plain``); no hash-slot table
* ``uneven``  5,000 references, 344 Mbp, log-normal lengths, GC 0.3-0.7 (``uneven``, ``long``)
* ``repeats`` 2,000 references, 5% of each overwritten by shared segments of 500-5,000 bp, each
              segment about 36 times: synth's ``repeats`` at a tenth of its size with a tenth of
              its segments, so that a repeat has the copies it has in the 20,000-reference set
* ``ultra``   16 references of 270 kb and more (``ultralong``)

Classification results are bit-exact by contract, so they are returned as the byte records of the
C ABI (mg_read_result, mg_candidate), the candidates in buffers of a fixed capacity that are zero
past the last one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mirage_b200 as M

K, STEP = 31, 15  # the library's default k; seeds start every k / 2 bases
DEV = "cuda:0"

# Reads per kind: lengths ("fixed" lo = hi, "uniform", "lognormal" around a median, "loguniform"),
# substitution and single-base indel rates, the fraction joining two references (chimera) and the
# fraction of unrelated random reads.
READS = {
    "short150": dict(lengths="fixed", lo=150, hi=150, sub=0.01, indel=0.0, chimera=0.0, unrelated=1 / 11),
    "uneven": dict(lengths="uniform", lo=75, hi=300, sub=0.005, indel=0.001, chimera=0.0, unrelated=0.2),
    "long": dict(lengths="lognormal", lo=1000, hi=20000, median=5000, sub=0.03, indel=0.02, chimera=0.1, unrelated=0.0),
    "mixed": dict(lengths="loguniform", lo=75, hi=20000, sub=0.02, indel=0.01, chimera=0.05, unrelated=0.1),
    "rep250": dict(lengths="fixed", lo=250, hi=250, sub=0.01, indel=0.0, chimera=0.0, unrelated=0.0),
    "ultra": dict(lengths="uniform", lo=66000, hi=250000, sub=0.03, indel=0.02, chimera=0.25, unrelated=0.0),
}


def listed() -> list[dict]:
    return [
        # a caller with a handful of reads at a time (an interactive query): launches and copies count
        dict(name="host_small_16", call="classify", index="small", reads="short150", n=16),
        # the drop-in per-batch call of the plain form, on the reference's own kind of test batch
        dict(name="plain_form_11k", call="plain", index="small", reads="short150", n=11000),
        # a pipeline stage whose reads are on the GPU already: a mid-sized, odd batch
        dict(name="device_uneven_20k", call="device", index="uneven", reads="uneven", n=20011),
        # the same at the size of the library's benchmark
        dict(name="device_uneven_1m", call="device", index="uneven", reads="uneven", n=1000000),
        # end to end from pinned host buffers, the benchmark's batch
        dict(name="host_uneven_1m", call="pinned", index="uneven", reads="uneven", n=1000000),
        # long reads with 5% errors and chimeras, on the GPU
        dict(name="device_long_20k", call="device", index="uneven", reads="long", n=20000),
        # a sample that mixes platforms: 75 bases to 20 kb in one host batch
        dict(name="host_mixed_4k", call="pinned", index="uneven", reads="mixed", n=4001),
        # short reads against references that share repeats: seeds with dozens of hits
        dict(name="device_repeats_200k", call="device", index="repeats", reads="rep250", n=200000),
        # ultra-long reads, past 65,535 bases
        dict(name="device_ultra_12", call="device", index="ultra", reads="ultra", n=12),
        # a service: requests of log-uniform size coalesced into steps
        dict(name="served_24", call="served", index="uneven", reads="uneven", n=24, most=50000),
        # scoring alone, for a caller that keeps its own seed lookup
        dict(name="score_20k", call="score", index="uneven", reads="uneven", n=20000),
        # an index built from references (before it is saved or opened)
        dict(name="build_5m", call="build", index="", reads="", n=100, length=50000),
    ]


def draw(rng) -> dict:
    """One more case of the listed ones' ranges."""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["classify", "plain", "device", "device", "pinned", "long", "mixed", "repeats", "ultra", "served",
                       "score", "build"])
    if kind == "classify":
        return dict(call="classify", index="small", reads="short150", n=size(1, 2000))
    if kind == "plain":
        return dict(call="plain", index="small", reads="short150", n=size(200, 11000))
    if kind == "device":
        return dict(call="device", index="uneven", reads="uneven", n=size(1000, 1000000))
    if kind == "pinned":
        return dict(call="pinned", index="uneven", reads="uneven", n=size(1000, 1000000))
    if kind == "long":
        return dict(call="device", index="uneven", reads="long", n=size(100, 20000))
    if kind == "mixed":
        return dict(call="pinned", index="uneven", reads="mixed", n=size(64, 8000))
    if kind == "repeats":
        return dict(call="device", index="repeats", reads="rep250", n=size(1000, 200000))
    if kind == "ultra":
        return dict(call="device", index="ultra", reads="ultra", n=rng.randint(1, 12))
    if kind == "served":
        return dict(call="served", index="uneven", reads="uneven", n=rng.randint(4, 28), most=size(1000, 50000))
    if kind == "score":
        return dict(call="score", index="uneven", reads="uneven", n=size(200, 20000))
    return dict(call="build", index="", reads="", n=rng.randint(20, 120), length=size(2000, 40000))


# ------------------------------------------------------------------------------ references

ACGT = (65, 67, 71, 84)


def _gen(*seed) -> tuple[torch.Generator, np.random.Generator]:
    g = torch.Generator(device=DEV)
    g.manual_seed(int(np.random.SeedSequence(seed).generate_state(1, np.uint64)[0] >> 1))
    return g, np.random.default_rng(seed)


def _random_bases(n: int, g: torch.Generator, gc: torch.Tensor | float = 0.5) -> torch.Tensor:
    """n random bases; gc: one fraction, or one per base."""
    u = torch.rand(n, generator=g, device=DEV)
    code = (u > (1 - gc) / 2).to(torch.uint8) + (u > 0.5) + (u > (1 + gc) / 2)
    return torch.tensor(ACGT, dtype=torch.uint8, device=DEV)[code.long()]


class Refs:
    """References on the GPU and the host."""

    def __init__(self, lens: np.ndarray, gc: np.ndarray, seed: int, segments: int = 0):
        g, rng = _gen(seed)
        self.lens = lens.astype(np.int64)
        self.offs = np.zeros(len(lens) + 1, np.int64)
        self.offs[1:] = np.cumsum(self.lens)
        data = torch.empty(int(self.offs[-1]), dtype=torch.uint8, device=DEV)
        for i in range(0, len(lens), 256):  # a few references at a time
            j = min(i + 256, len(lens))
            per = torch.repeat_interleave(torch.tensor(gc[i:j], dtype=torch.float32, device=DEV),
                                          torch.tensor(self.lens[i:j], device=DEV))
            data[self.offs[i] : self.offs[j]] = _random_bases(per.numel(), g, per)
        if segments:  # shared repeat segments over 5% of every reference
            pool = [_random_bases(int(x), g) for x in rng.integers(500, 5001, size=segments)]
            for i in range(len(lens)):
                done = 0
                while done < 0.05 * lens[i]:
                    s = pool[int(rng.integers(0, segments))]
                    if len(s) >= lens[i]:
                        break
                    a = int(self.offs[i]) + int(rng.integers(0, lens[i] - len(s) + 1))
                    data[a : a + len(s)] = s
                    done += len(s)
        self.data = data
        self.host = data.cpu().numpy()
        order = np.argsort(-self.lens, kind="stable")  # longest first: a read picks among those that hold it
        self.d_order = torch.tensor(order, device=DEV)
        self.d_neg = torch.tensor(-self.lens[order], device=DEV)
        self.d_offs = torch.tensor(self.offs, device=DEV)
        self.d_lens = torch.tensor(self.lens, device=DEV)

    def names(self) -> list[bytes]:
        return [b"ref%d" % i for i in range(len(self.lens))]


def _lognormal(rng, n, median, sigma, lo):
    return np.maximum(np.round(np.exp(rng.normal(np.log(median), sigma, size=n))), lo).astype(np.int64)


def _reference_set(name: str) -> Refs:
    rng = np.random.default_rng(2024)
    if name == "small":
        return Refs(np.full(200, 5000), np.full(200, 0.5), 1)
    if name == "uneven":
        lens = _lognormal(rng, 5000, 50000, 0.8, 1000)
        return Refs(lens, rng.uniform(0.3, 0.7, size=5000), 2)
    if name == "repeats":
        lens = _lognormal(rng, 2000, 80000, 0.67, 6000)
        return Refs(lens, np.full(2000, 0.5), 3, segments=100)
    return Refs(_lognormal(rng, 16, 400000, 0.3, 270000), rng.uniform(0.35, 0.65, size=16), 4)


_open: dict = {}


def _index(name: str):
    """The references and the open index of a set, opened once per process."""
    if name not in _open:
        refs = _reference_set(name)
        image = M.build_image(refs.host, refs.offs, refs.names(), k=K, device=0)
        _open[name] = (refs, M.Index(image, k=K, device=0))
    return _open[name]


def _server(name: str):
    if ("server", name) not in _open:
        _open["server", name] = M.Server(_index(name)[1])
    return _open["server", name]


# ------------------------------------------------------------------------------ reads


def _lengths(spec: dict, n: int, rng) -> np.ndarray:
    lo, hi = spec["lo"], spec["hi"]
    if spec["lengths"] == "lognormal":
        x = np.exp(rng.normal(np.log(spec["median"]), 0.8, size=n))
    elif spec["lengths"] == "loguniform":
        x = np.exp(rng.uniform(np.log(lo), np.log(hi), size=n))
    else:
        x = rng.integers(lo, hi + 1, size=n)
    return np.clip(np.round(x), lo, hi).astype(np.int64)


def _make_reads(refs: Refs, kind: str, n: int, seed: int):
    """Reads on the GPU: (bases, offsets, first reference, its position, reversed), drawn from random
    references, positions and strands with indels, then substitutions."""
    spec = READS[kind]
    g, rng = _gen(seed, 77)
    lens = _lengths(spec, n, rng)
    offs = np.zeros(n + 1, np.int64)
    offs[1:] = np.cumsum(lens)
    out = torch.empty(int(offs[-1]), dtype=torch.uint8, device=DEV)
    ref, pos = torch.empty(n, dtype=torch.int64, device=DEV), torch.empty(n, dtype=torch.int64, device=DEV)
    flip = torch.rand(n, generator=g, device=DEV) < 0.5
    code_of = torch.zeros(256, dtype=torch.uint8, device=DEV)
    comp = torch.zeros(256, dtype=torch.uint8, device=DEV)
    for i, c in enumerate(ACGT):
        code_of[c], comp[c] = i, ACGT[3 - i]
    acgt = torch.tensor(ACGT, dtype=torch.uint8, device=DEV)
    i = 0
    while i < n:  # at most 2^25 bases at a time (a read at least)
        j = max(i + 1, int(np.searchsorted(offs, offs[i] + (1 << 25), side="right")) - 1)
        L = torch.tensor(lens[i:j], device=DEV)
        m = j - i
        need = L + L // 16 + 16  # the read and its deletions
        span = torch.clamp(need, max=int(refs.lens.max()) - 1)

        def pick():
            count = torch.searchsorted(refs.d_neg, -span, right=True)
            r = refs.d_order[(torch.rand(m, generator=g, device=DEV) * count).long().clamp_(max=count - 1)]
            p = (torch.rand(m, generator=g, device=DEV, dtype=torch.float64) * (refs.d_lens[r] - span + 1)).long()
            return r, p

        (ra, pa), (rb, pb) = pick(), pick()
        ref[i:j], pos[i:j] = ra, pa
        u = torch.rand(2, m, generator=g, device=DEV)
        cut = torch.where(u[0] < spec["chimera"], (u[1] * (L - 1)).long() + 1, L)
        rid = torch.repeat_interleave(torch.arange(m, device=DEV), L)
        start = torch.cumsum(L, 0) - L
        at = torch.arange(rid.numel(), device=DEV) - start[rid]
        src = at
        if spec["indel"]:
            ev = torch.rand(rid.numel(), generator=g, device=DEV)
            ins, dele = (ev < spec["indel"] / 2), (ev >= spec["indel"] / 2) & (ev < spec["indel"])
            shift = torch.cumsum(dele.int() - ins.int(), 0)
            before = torch.cat([torch.zeros(1, dtype=shift.dtype, device=DEV), shift])[start]
            src = torch.minimum((at + shift - before[rid]).clamp_(min=0), (span - 1)[rid])
        a = (refs.d_offs[ra] + pa)[rid] + src
        b = (refs.d_offs[rb] + pb)[rid] + src
        base = refs.data[torch.where(at < cut[rid], a, b)]
        change = torch.rand(rid.numel(), generator=g, device=DEV) < spec["sub"]
        add = torch.randint(1, 4, (rid.numel(),), generator=g, device=DEV, dtype=torch.uint8)
        base = torch.where(change, acgt[((code_of[base.long()] + add) % 4).long()], base)
        if spec["unrelated"]:
            other = torch.rand(m, generator=g, device=DEV) < spec["unrelated"]
            base = torch.where(other[rid], _random_bases(rid.numel(), g), base)
        f = flip[i:j]
        back = torch.where(f[rid], start[rid] + L[rid] - 1 - at, start[rid] + at)
        base = base[back]
        out[offs[i] : offs[j]] = torch.where(f[rid], comp[base.long()], base)
        i = j
    return out, torch.tensor(offs, device=DEV), ref, pos, flip


# ------------------------------------------------------------------------------ the cases


def prepare(case: dict, seed: int) -> dict:
    call, n = case["call"], case["n"]
    if call == "build":
        g, rng = _gen(seed, 5)
        lens = np.linspace(case["length"] // 2, 3 * case["length"] // 2, n).astype(np.int64)
        refs = Refs(rng.permutation(lens), rng.uniform(0.3, 0.7, size=n), seed)
        # an image takes 20 to 28 bytes a base: what is past 19 goes to a buffer of fixed size
        return dict(call=call, bases=refs.host, offs=refs.offs.astype(np.uint64), names=refs.names(),
                    head=19 * int(lens.sum()), tail=np.zeros(11 * int(lens.sum()) + 4096, np.uint8))
    refs, ix = _index(case["index"])
    if call == "served":  # requests of log-uniform size, slices of a pool of reads
        sizes = np.exp(np.linspace(0, math.log(case["most"]), n)).astype(np.int64)
        sizes = np.random.default_rng(9).permutation(sizes)
        bases, offs, *_ = _make_reads(refs, case["reads"], int(sizes.sum()), seed)
        bases, offs = bases.cpu().numpy(), offs.cpu().numpy()
        requests, r = [], 0
        for s in sizes:
            o = offs[r : r + s + 1]
            requests.append((bases[o[0] : o[-1]].copy(), (o - o[0]).astype(np.uint64), _room(8 * int(s) + 64)))
            r += int(s)
        return dict(call=call, server=_server(case["index"]), requests=requests)
    if call == "score":
        return dict(call=call, ix=ix, args=_score_inputs(refs, case, seed))
    bases, offs, *_ = _make_reads(refs, case["reads"], n, seed)
    if call == "classify":
        return dict(call=call, ix=ix, bases=bases.cpu().numpy(), offs=offs.cpu().numpy().astype(np.uint64),
                    cands=_room(8 * n + 64))
    cap = (64 if case["index"] == "repeats" else 8) * n + 1024
    if call == "device":
        return dict(call=call, ix=ix, n=n, cap=cap, bases=bases, offs=offs, stream=torch.cuda.Stream(DEV),
                    reads=torch.empty(n, 16, dtype=torch.uint8, device=DEV),
                    cands=torch.zeros(cap, 16, dtype=torch.uint8, device=DEV),
                    count=torch.zeros(1, dtype=torch.int64, device=DEV))
    return dict(call=call, ix=ix, n=n, cap=cap, bases=bases.cpu().pin_memory(), offs=offs.cpu().pin_memory(),
                reads=torch.empty(n, 16, dtype=torch.uint8, pin_memory=True),
                cands=torch.zeros(cap, 16, dtype=torch.uint8, pin_memory=True))


def _room(cap: int) -> np.ndarray:
    return np.zeros(cap, M.CAND_DTYPE)


def _kept(r: M.Results, room: np.ndarray) -> dict:
    room[: len(r.cands)] = r.cands
    return {"reads": r.reads.view(np.uint8), "cands": room.view(np.uint8)}


def run(s: dict):
    call = s["call"]
    if call == "classify":
        return _kept(s["ix"].classify(s["bases"], s["offs"]), s["cands"])
    if call == "device":
        st = s["stream"].cuda_stream
        s["ix"].classify_device(s["n"], s["offs"].data_ptr(), s["bases"].data_ptr(), s["reads"].data_ptr(),
                                s["cands"].data_ptr(), s["cap"], s["count"].data_ptr(), st)
        nc = s["ix"].device_sync(st)  # the call that reports a batch's errors and its candidates
        return {"reads": s["reads"], "cands": s["cands"], "n": nc}
    if call in ("pinned", "plain"):
        nc = s["ix"].classify_ptrs(s["n"], s["offs"].data_ptr(), s["bases"].data_ptr(), s["reads"].data_ptr(),
                                   s["cands"].data_ptr(), s["cap"], "plain" if call == "plain" else "batched")
        return {"reads": s["reads"], "cands": s["cands"], "n": nc}
    if call == "served":
        sv, tickets, got = s["server"], [], []
        for bases, offs, _ in s["requests"]:
            while (t := sv.submit_into(bases, offs)) is None:  # not admitted now: take a result first
                got.append(sv.wait(tickets[len(got)]))
            tickets.append(t)
        while len(got) < len(tickets):
            got.append(sv.wait(tickets[len(got)]))
        return [_kept(r, q[2]) for r, q in zip(got, s["requests"])]
    if call == "score":
        score, pct, rel, highest = s["ix"].score_candidates(*s["args"])
        return {"score": score, "pct": pct, "rel": rel, "highest": highest}
    image = M.build_image(s["bases"], s["offs"], s["names"], k=K, device=0)
    s["tail"][: len(image) - s["head"]] = image[s["head"] :]
    return {"image": image[: s["head"]], "tail": s["tail"], "n": len(image)}


def _score_inputs(refs: Refs, case: dict, seed: int):
    """Strands with their candidates and runs, as a caller's own seed lookup gives them: the read's
    reference with one to three runs on its diagonal, and for every third strand another reference
    with one short run."""
    n = case["n"]
    bases, offs, ref, pos, flip = _make_reads(refs, case["reads"], n, seed)
    bases, offs, ref, pos, flip = (x.cpu().numpy() for x in (bases, offs, ref, pos, flip))
    _, rng = _gen(seed, 11)
    comp = np.zeros(256, np.uint8)
    comp[list(ACGT)] = ACGT[::-1]
    c_off, cand, r_off, runs = [0], [], [0], []
    for i in range(n):
        a, b = int(offs[i]), int(offs[i + 1])
        if flip[i]:  # the strand that lies on the reference
            bases[a:b] = comp[bases[a:b][::-1]]
        seeds = (b - a - K - 1) // STEP + 1
        parts = np.unique(np.append(rng.integers(0, seeds, size=int(rng.integers(0, 3))), [0, seeds]))
        for s0, s1 in zip(parts[:-1], parts[1:]):
            sq, lq = int(s0) * STEP, min(int(s1) * STEP, b - a)
            runs.append((int(pos[i]) + sq, sq, int(pos[i]) + lq, lq))
        cand.append(int(ref[i]))
        r_off.append(len(runs))
        if i % 3 == 0:
            r = int(rng.integers(0, len(refs.lens)))
            p = int(rng.integers(0, refs.lens[r] - 2 * STEP))
            runs.append((p, STEP, p + 2 * STEP, 3 * STEP))
            cand.append(r)
            r_off.append(len(runs))
        c_off.append(len(cand))
    return (offs.astype(np.uint64), bases, np.array(c_off, np.uint64), np.array(cand, np.uint32),
            np.array(r_off, np.uint64), np.array(runs, np.uint32))


def work(case: dict) -> dict:
    n = case["n"]
    if case["call"] == "build":  # references in, an image of about 25 bytes a window out
        return {"bytes": 26.0 * n * case["length"], "flops": 0}
    spec = READS[case["reads"]]
    lo, hi = spec["lo"], spec["hi"]
    if spec["lengths"] == "lognormal":
        mean = spec["median"] * 1.3
    elif spec["lengths"] == "loguniform":
        mean = (hi - lo) / math.log(hi / lo)
    else:
        mean = (lo + hi) / 2
    if case["call"] == "served":
        n = n * (case["most"] - 1) / math.log(case["most"])
    if case["call"] == "score":  # bases, a candidate and a few runs with their windows, the scores
        return {"bytes": n * (mean + 1.4 * (4 + 12) + 2 * (16 + 64) + 4), "flops": 0}
    # the bases, one 32-byte sector per seed of both strands, the results, and for each candidate its
    # record and the two reference windows
    cands = n * (1 - spec["unrelated"]) * (1 + spec["chimera"])
    return {"bytes": n * (mean + 2 * 32 * max(0.0, mean - K) / STEP + 16) + 80 * cands, "flops": 0}


def exact(case: dict, seed: int):
    """The scores of score_candidates in 64 bits; the other cases return byte records."""
    if case["call"] != "score":
        return None
    refs = _index(case["index"])[0]
    q_off, bases, c_off, cand, r_off, runs = (x.astype(np.int64) for x in _score_inputs(refs, case, seed))
    nc, ns = len(cand), len(q_off) - 1
    strand = np.repeat(np.arange(ns), np.diff(c_off))
    of = np.repeat(np.arange(nc), np.diff(r_off))  # the candidate of each run
    L, q0 = np.diff(q_off)[strand][of], q_off[:-1][strand][of]
    rlen, r0 = refs.lens[cand][of], refs.offs[cand][of]
    sr, sq, lr, lq = runs.T
    tail, on = np.zeros(len(of), np.int64), np.ones(len(of), bool)
    lim = np.minimum(np.minimum(rlen - lr, K), L - lq)
    head, hon = np.zeros(len(of), np.int64), (sq > 0) & (np.minimum(sr, K) > 0)
    jb = np.minimum(sq - 1, np.minimum(sr, K) - 1)  # the head stops at jb, matched or not
    for t in range(K):
        on &= t < lim
        x = np.flatnonzero(on)
        on[x] = bases[(q0 + lq + t)[x]] == refs.host[(r0 + lr + t)[x]]
        tail[on] += 1
        hon &= t < jb
        x = np.flatnonzero(hon)
        hon[x] = bases[(q0 + sq - 1 - t)[x]] == refs.host[(r0 + sr - t)[x]]
        head[hon] += 1
    total = tail + head + (lq - sq)
    kept = total >= K
    sumc = np.bincount(of, np.where(kept, total, 0), nc)
    sumr = np.bincount(of, np.where(kept, total * (total + 1) / 2, 0.0), nc)
    cover = np.zeros(nc * 512 + 1, np.int64)  # the query bases that a candidate's runs cover
    np.add.at(cover, of[kept] * 512 + (sq - head)[kept], 1)
    np.add.at(cover, of[kept] * 512 + (sq - head + total)[kept], -1)
    hits = (np.cumsum(cover)[:-1].reshape(nc, 512) > 0).sum(1)
    Lc, rc = np.diff(q_off)[strand].astype(np.float64), refs.lens[cand].astype(np.float64)
    ok = sumc > 0
    pct = np.where(ok, 100.0 / Lc * hits, 0.0)
    score = np.where(ok, sumr / np.maximum(sumc, 1) / 100.0 * pct, -2.0)
    lm = np.minimum(Lc, rc)
    rel = np.where(ok, np.log(np.maximum(score, 0) + 1) / np.log(lm * (lm + 1) / 2 / lm + 1), -1.0)
    highest = np.full(ns, -1.0)
    np.maximum.at(highest, strand, rel)
    return {"score": score, "pct": pct, "rel": rel, "highest": highest}
