"""The oversize tier's workspaces when memory is short: the counts asked for, on the CPU against an
allocator with a limit, and a batch on a device that has room for few of them."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mirage_b200", "csrc")


def test_slab_counts_under_a_memory_limit(tmp_path):
    exe = str(tmp_path / "slabs_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "native", "slabs_check.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
def test_oversize_reads_with_memory_for_few_workspaces():
    """64 reads of 160-180 kb, whose 64 workspaces (2^16 postings a strand: 1.7 MB each and more) do
    not fit the 72 MiB that are left on the device: the batch runs with fewer, its results equal those
    of an index with all of them byte for byte, and so does a second batch, after which more
    workspaces were asked for in vain."""
    import torch

    import mirage_b200 as M

    rng = np.random.default_rng(83)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    core = acgt[rng.integers(0, 4, 400_000)]
    refs = [core] * 4
    offs = np.zeros(len(refs) + 1, np.uint64)
    offs[1:] = np.cumsum([len(r) for r in refs])
    image = M.build_image(np.concatenate(refs), offs, [f"ref{i}" for i in range(len(refs))])
    roomy, tight = M.Index(image), M.Index(image)
    lens = rng.integers(160_000, 180_000, 64)
    roffs = np.zeros(65, np.uint64)
    roffs[1:] = np.cumsum(lens)
    data = np.concatenate([core[s:s + n] for s, n in zip(rng.integers(0, 220_000, 64), lens)])
    want = roomy.classify(data, roffs)
    # the other buffers of such a batch, from reads of 321 bases that go through the other tiers
    small = np.zeros(len(data) // 321 + 1, np.uint64)
    small[1:] = 321 * np.arange(1, len(small), dtype=np.uint64)
    tight.classify(data, small)
    one = np.array([0, lens[0]], np.uint64)
    tight.classify(data[:lens[0]], one)  # and one workspace
    torch.cuda.empty_cache()
    held = []
    try:
        while (spare := torch.cuda.mem_get_info(0)[0] - (72 << 20)) > (4 << 20):
            held.append(torch.empty(min(spare, 16 << 30), dtype=torch.uint8, device="cuda:0"))
        got = [tight.classify(data, roffs) for _ in range(2)]
    finally:
        del held
        torch.cuda.empty_cache()
    for g in got:
        assert np.array_equal(g.reads.view(np.uint8), want.reads.view(np.uint8))
        assert np.array_equal(g.cands.view(np.uint8), want.cands.view(np.uint8))
    roomy.close()
    tight.close()
