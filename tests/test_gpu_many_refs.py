"""Indexes either side of 2^21 references, where the long-read tier's packed postings end: beyond, its
place (and the plain form's kernel) is taken by the shared-memory block tier."""
import os

import numpy as np
import pytest

import mirage_b200 as M
from parity_util import canon_from_dump, canon_from_gpu, diff

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)
COMP = np.zeros(256, np.uint8)
COMP[list(b"ACGT")] = list(b"TGCA")


@pytest.mark.parametrize("n_refs", [1 << 21, (1 << 21) + 1])
def test_reads_on_the_last_of_two_million_references(tmp_path, n_refs):
    """References of 20 bases, then five of 40 kb with the highest numbers, of which two are the same and
    one shares a segment: reads of 150 bases to 30 kb, with substitutions, reversed, joined and in lower
    case, in both forms."""
    from oracle import oracle as O

    rng = np.random.default_rng(131)
    core = [ACGT[rng.integers(0, 4, 40000)] for _ in range(4)]
    core[3][2000:9000] = core[1][11000:18000]
    core.append(core[0])
    n_small = n_refs - len(core)
    lens = np.full(n_refs, 20, np.uint64)
    lens[n_small:] = 40000
    offs = np.zeros(n_refs + 1, np.uint64)
    offs[1:] = np.cumsum(lens)
    image = M.build_image(np.concatenate([ACGT[rng.integers(0, 4, 20 * n_small)]] + core), offs,
                          [b"r%d" % i for i in range(n_refs)], device=0)
    path = tmp_path / "many.mhm"
    image.tofile(path)
    gix, oix = M.Index(image), O.Index(str(path))
    seqs = []
    for n in (150, 320, 321, 1000, 6000, 10577, 20480, 30000):
        for c in core[:4]:
            s = int(rng.integers(0, 40000 - n))
            r = c[s:s + n].copy()
            hit = rng.random(n) < 0.02
            r[hit] = ACGT[rng.integers(0, 4, int(hit.sum()))]
            seqs += [r, COMP[r[::-1]]]
    seqs += [np.concatenate([core[1][14000:18000], core[2][:3000]]), core[3][1500:9500], core[0][:2000] | 0x20]
    offs = np.zeros(len(seqs) + 1, np.uint64)
    offs[1:] = np.cumsum([len(s) for s in seqs])
    data = np.concatenate(seqs)
    want = canon_from_dump(oix.classify(data, offs, threads=os.cpu_count() or 1))
    for form in ("batched", "plain"):
        r = gix.classify(data, offs, form=form)
        d = diff(canon_from_gpu(r), want)
        assert not d, form + "\n" + "\n".join(d)
        assert r.reads["reported"].all()
    gix.close()
