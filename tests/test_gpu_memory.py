"""Calls that take device memory for their own use give it back."""
import numpy as np
import pytest

import mirage_b200 as M
from test_gpu_build import _toc_entry

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _references(n, length, seed):
    rng = np.random.default_rng(seed)
    offs = np.arange(0, n * length + 1, length, dtype=np.uint64)
    return ACGT[rng.integers(0, 4, n * length)], offs, [f"ref{i}" for i in range(n)]


def _free() -> int:
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def _build():
    bases, offs, names = _references(20, 100_000, 1)
    return M.build_image(bases, offs, names, device=0)


def _open_and_close(image):
    M.Index(image).close()


def _refused(image):
    """An image whose first hash is wider than 28 bits: the open fails after its device work has begun."""
    at, _, _ = _toc_entry(image, 0)
    bad = image.copy()
    bad[at:at + 4] = 0xFF
    with pytest.raises(M.MirageError):
        M.Index(bad)


def _parse():
    bases, offs, names = _references(50, 20_000, 2)
    text = b"".join(b">%s\n%s\n" % (n.encode(), bases[int(a):int(b)].tobytes())
                    for n, a, b in zip(names, offs[:-1], offs[1:]))
    M.parse_fasta(text, device=0)


@pytest.mark.parametrize("call", ["build", "open", "refused", "parse", "bucket_sizes", "logf", "gather"])
def test_free_memory_is_the_same_after_many_calls(call):
    image = _build()
    ix = M.Index(image)
    run = {"build": _build, "open": lambda: _open_and_close(image), "refused": lambda: _refused(image), "parse": _parse,
           "bucket_sizes": lambda: ix.bucket_sizes(np.arange(1 << 20, dtype=np.uint32)),
           "logf": lambda: ix.eval_logf(np.linspace(1, 1000, 1 << 20).astype(np.float32)),
           "gather": lambda: M.gather_bandwidth(0, 1 << 26)}[call]
    run()
    before = _free()
    for _ in range(12):
        run()
    assert _free() >= before, (call, before - _free())
    ix.close()
