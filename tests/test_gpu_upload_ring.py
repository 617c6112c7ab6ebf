"""Uploads that take the ring of pinned chunks: an opaque image drawn texel for pixel
comes back byte for byte, and the ring's threads have worked for the large ones only."""
import threading
from pathlib import Path

import numpy as np
import pytest

import tileink_b200 as tk

pytestmark = pytest.mark.gpu


def turns():
    """How often the ring's threads have gone to sleep: each copy wakes them."""
    n = 0
    for task in Path("/proc/self/task").iterdir():
        if (task / "comm").read_text().strip() == "tileink-upload":
            n += int(next(line for line in (task / "status").read_text().splitlines()
                          if line.startswith("voluntary_ctxt_switches")).split()[1])
    return n


def wrong_texels(r, w, h, seed):
    im = np.random.default_rng(seed).integers(0, 1 << 32, (h, w), dtype=np.uint32) | np.uint32(0xFF000000)
    c = tk.Canvas(w, h)
    c.push_image(0, 0, w, h, c.add_image(im))
    got = np.ascontiguousarray(r.render_to_image(c)).view(np.uint32).reshape(h, w)
    return int((got != im).sum())


# 16 MB to the byte, and with a last chunk of a part
@pytest.mark.parametrize("w,h", [(2048, 2048), (2311, 1831)])
def test_gpu_large_uploads_take_the_ring(w, h):
    r = tk.NativeRenderer(0)
    try:
        assert [wrong_texels(r, w, h, k) for k in range(4)] == [0] * 4  # 64 MB: the ring is there
        for k in range(3):
            before = turns()
            assert wrong_texels(r, w, h, 10 + k) == 0
            assert turns() > before
        before = turns()
        assert wrong_texels(r, 2048, 2047, 20) == 0  # below the limit
        assert turns() == before
    finally:
        r.close()


def test_gpu_contexts_share_the_ring():
    wrong = []

    def rounds(seed):
        r = tk.NativeRenderer(0)
        try:
            for k in range(7):
                wrong.append(wrong_texels(r, 2048, 2049, (seed, k)))
        finally:
            r.close()

    threads = [threading.Thread(target=rounds, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0] * 21
