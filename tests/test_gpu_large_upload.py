"""Large pageable uploads through the shared ring of pinned chunks: an opaque image
drawn texel for pixel comes back byte for byte, below and above the sizes at which
the ring is made and used, from several contexts at once."""
import threading

import numpy as np
import pytest

import tileink_b200 as tk

pytestmark = pytest.mark.gpu


def rounds(w, h, n, seed, wrong):
    r = tk.NativeRenderer(0)
    try:
        for k in range(n):
            im = np.random.default_rng((seed, k)).integers(0, 1 << 32, (h, w), dtype=np.uint32) | np.uint32(0xFF000000)
            c = tk.Canvas(w, h)
            c.push_image(0, 0, w, h, c.add_image(im))
            got = np.ascontiguousarray(r.render_to_image(c)).view(np.uint32).reshape(h, w)
            wrong.append(int((got != im).sum()))
    finally:
        r.close()


# 8 MB to the byte; a last chunk of a part; a texel below the limit
@pytest.mark.parametrize("w,h", [(2048, 1024), (1601, 1443), (2049, 1023)])
@pytest.mark.parametrize("threads", [1, 3])
def test_gpu_large_uploads(w, h, threads):
    wrong = []
    ts = [threading.Thread(target=rounds, args=(w, h, 6, s, wrong)) for s in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert wrong == [0] * (6 * threads)
