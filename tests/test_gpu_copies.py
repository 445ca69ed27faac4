"""Reads that meet segments shared by many references, through the long-read tier and what it hands
on: results against the CPU restatement (oracle/), routes by the tier counts."""
import os

import numpy as np
import pytest

import mirage_b200 as M
from parity_util import canon_from_dump, canon_from_gpu, diff

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)
K, STEP, HLEN = 31, 15, 17


def _open(refs, path):
    from oracle import oracle as O

    offs = np.zeros(len(refs) + 1, np.uint64)
    offs[1:] = np.cumsum([len(r) for r in refs])
    image = M.build_image(np.concatenate(refs), offs, [f"ref{i}" for i in range(len(refs))], k=K)
    image.tofile(path)
    return M.Index(image, k=K), O.Index(str(path), k=K)


def _check(gix, oix, seqs, form="batched"):
    offs = np.zeros(len(seqs) + 1, np.uint64)
    offs[1:] = np.cumsum([len(s) for s in seqs])
    data = np.concatenate([np.frombuffer(bytes(s), np.uint8) for s in seqs])
    r = gix.classify(data, offs, form=form)
    d = diff(canon_from_gpu(r), canon_from_dump(oix.classify(data, offs, threads=os.cpu_count() or 1)))
    assert not d, "\n".join(d)
    c = gix.last_tier_counts()
    if form == "batched":  # the same reads in a batch that both classes of the long-read tier share
        reps = 300 // len(seqs) + 1
        big = gix.classify(np.tile(data, reps), np.append(0, np.cumsum(np.tile(np.diff(offs), reps))).astype(np.uint64))
        for f in r.reads.dtype.names:
            if f != "cand_off":
                assert np.array_equal(big.reads[f], np.tile(r.reads[f], reps)), f
        assert np.array_equal(big.cands.view(np.uint8), np.tile(r.cands, reps).view(np.uint8))
        assert gix.last_tier_counts()["block"] == reps * c["block"]
    return r, c


def _copies(rng, copies, n_refs, ref_len, seg_len, n_segs):
    """References in which every segment lies in `copies` of them, and the segments' places."""
    refs = [ACGT[rng.integers(0, 4, ref_len)] for _ in range(n_refs)]
    places = []
    for t in range(n_segs):
        seg = ACGT[rng.integers(0, 4, seg_len)]
        for r in rng.choice(n_refs, copies, replace=False):
            a = int(rng.integers(400, ref_len - seg_len - 400))
            refs[r][a:a + seg_len] = seg
            places.append((int(r), a, t))
    return refs, places


@pytest.mark.parametrize("slots", [False, True])
@pytest.mark.parametrize("copies", [88, 89, 130, 200])
def test_reads_on_the_flank_of_a_segment_with_many_copies(tmp_path, copies, slots):
    """Reads of 250 bases, half in a segment that 88 to 200 references share, half in the flank of one:
    the keep rule drops the copies, so the reads stay in the long-read tier however many there are (at
    most 8 seeds of 200 postings: within the tier's 4,096)."""
    rng = np.random.default_rng(101)
    refs, places = _copies(rng, copies, 220, 3000, 600, 1)
    gix, oix = _open(refs, tmp_path / "flank.mhm")
    gix.set_probe_slots(slots)
    seqs = [refs[r][a - 140:a + 110] for r, a, _ in places[:: max(1, len(places) // 40)]]
    r, c = _check(gix, oix, seqs)
    assert c["block"] == 0, c
    _check(gix, oix, seqs, "plain")


def test_long_reads_across_several_repeats(tmp_path):
    """Reads of 2 to 16 kb that cross segments of 500 bases with 12 copies each: dozens of linked
    references on a strand of a thousand found seeds, of which the keep rule leaves the read's own."""
    rng = np.random.default_rng(103)
    refs, _ = _copies(rng, 12, 60, 20000, 500, 25)
    gix, oix = _open(refs, tmp_path / "several.mhm")
    seqs = []
    for n in (2000, 5000, 8000, 12000, 16000):
        for _ in range(6):
            a = int(rng.integers(0, 20000 - n))
            r = refs[int(rng.integers(0, 60))][a:a + n].copy()
            hit = rng.random(n) < 0.01
            r[hit] = ACGT[rng.integers(0, 4, int(hit.sum()))]
            seqs.append(r)
    _, c = _check(gix, oix, seqs)
    assert c["block"] == 0, c
    _check(gix, oix, seqs, "plain")


@pytest.mark.parametrize("n_refs", [15, 16, 40])
def test_kept_references_spread_over_a_long_read(tmp_path, n_refs):
    """A read of 20,480 bases whose seeds lie in runs of three, the references in turn: every reference
    is kept, with runs all over the read, more of them than bitmaps of its found seeds fit for. Runs
    moved by a base, a reference twice under a seed, and positions out of seed order among them."""
    rng = np.random.default_rng(107)
    L = 20480
    read = ACGT[rng.integers(0, 4, L)]
    ns = (L - K + STEP - 1) // STEP
    parts = [[] for _ in range(n_refs)]
    for t, j in enumerate(range(0, ns - 2, 3)):
        w = read[j * STEP:(j + 2) * STEP + HLEN]
        parts[t % n_refs].append(w)
        if t % 17 == 0:
            parts[t % n_refs].append(w)
    refs = []
    for p in parts:
        order = rng.permutation(len(p)) if len(refs) % 3 == 0 else np.arange(len(p))
        refs.append(np.concatenate([np.concatenate([ACGT[rng.integers(0, 4, 23)], p[o]]) for o in order]))
    gix, oix = _open(refs, tmp_path / "spread.mhm")
    r, c = _check(gix, oix, [read, read[:14000].copy(), read[4500:].copy()])
    assert c["block"] == 0, c
    assert (r.reads["n_fwd"] >= 10).all()


@pytest.mark.parametrize("copies", [87, 88, 89, 223, 224, 225])
def test_reads_inside_a_segment_with_many_copies(tmp_path, copies):
    """Reads of 220 bases (13 seeds: at most 2,925 postings) from a segment that 87 to 225 references
    share: every copy is kept and a candidate. Either side of what the long-read tier's tables hold,
    88 and, in its second class, 224; beyond that the global-memory tier takes them."""
    rng = np.random.default_rng(109)
    refs, places = _copies(rng, copies, 230, 1500, 400, 1)
    gix, oix = _open(refs, tmp_path / "inside.mhm")
    r0, a0, _ = places[0]
    seqs = [refs[r0][a0 + i:a0 + i + 220] for i in range(0, 180, 20)]
    for part in (seqs[:3], seqs[3:6], seqs[6:]):  # the oracle's wrapper has room for 1,216 of their top candidates
        r, c = _check(gix, oix, part)
        assert (r.reads["n_fwd"] == copies).all()
        assert c["block"] == (len(part) if copies > 224 else 0), c
        _check(gix, oix, part, "plain")


def test_long_reads_on_a_few_strains(tmp_path):
    """Reads of 10 to 18 kb on four strains that differ by a base in 300: more than 2,048 kept postings a
    strand, up to the 4,096 of the long-read tier's second class."""
    rng = np.random.default_rng(113)
    core = ACGT[rng.integers(0, 4, 30000)]
    refs = []
    for _ in range(4):
        r = core.copy()
        hit = rng.random(len(r)) < 1 / 300
        r[hit] = ACGT[rng.integers(0, 4, int(hit.sum()))]
        refs.append(r)
    gix, oix = _open(refs, tmp_path / "strains.mhm")
    seqs = [refs[i % 4][100 * i:100 * i + n] for i, n in enumerate((10000, 12000, 13000, 14000, 15000, 15400, 18000))]
    _, c = _check(gix, oix, seqs)
    assert c["block"] <= 1, c  # the last may hold more


@pytest.mark.parametrize("k", [20, 21, 25])
def test_long_reads_with_a_shorter_key(tmp_path, k):
    """Reads of 14,070 to 20,480 bases with keys below the default: up to 2,046 seeds a strand."""
    from oracle import oracle as O

    rng = np.random.default_rng(127)
    refs = [ACGT[rng.integers(0, 4, 40000)] for _ in range(3)]
    offs = np.arange(0, 120001, 40000, dtype=np.uint64)
    image = M.build_image(np.concatenate(refs), offs, [f"ref{i}" for i in range(3)], k=k)
    path = tmp_path / "k.mhm"
    image.tofile(path)
    gix, oix = M.Index(image, k=k), O.Index(str(path), k=k)
    seqs = []
    for n in (14070, 14081, 17000, 20470, 20480):
        s = int(rng.integers(0, 40000 - n))
        r = refs[n % 3][s:s + n].copy()
        hit = rng.random(n) < 0.02
        r[hit] = ACGT[rng.integers(0, 4, int(hit.sum()))]
        seqs += [r, r[::-1].copy()]
    _, c = _check(gix, oix, seqs)
    assert c["block"] == 0, c
