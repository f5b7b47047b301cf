"""The row pipeline of intra frames (intra_rows_kernel) against the oracle at
the sizes where it can go wrong: search areas 1 to 8 (windows narrower than the
16 columns it is laid out for), rows shorter than a group of 8 blocks, a partial
last group, rows of more than 32 groups (the word tags' lap), fewer rows than
the window, and contents from flat (every word the same) to noise (a window of
nothing but distinct words)."""
import numpy as np
import pytest

import oracle
from mptc_gb300.synth import StreamSpec

pytestmark = pytest.mark.gpu


def frame(kind, w, h, seed):
    rng = np.random.default_rng(seed)
    if kind == "flat":
        return np.full((h, w, 3), (90, 140, 30), np.uint8)
    if kind == "noise":
        return rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    if kind == "mixed":  # noise patches on a gradient: words that come and go along a row
        g = (np.arange(w)[None, :, None] + 2 * np.arange(h)[:, None, None] + np.array([0, 40, 90])) % 256
        f = np.clip(g + rng.integers(-3, 4, (h, w, 3)), 0, 255).astype(np.uint8)
        m = (np.arange(h)[:, None] // 16 + np.arange(w)[None, :] // 24) % 3 == 0
        f[m] = rng.integers(0, 256, (int(m.sum()), 3), dtype=np.uint8)
        return f
    return StreamSpec(w, h, 1, seed=seed, square_size=min(32, w, h)).generate()[0]


@pytest.mark.parametrize("w,h,sa,thr,kind", [
    (4, 4, 8, 5, "stream"), (4, 80, 8, 5, "mixed"), (28, 64, 8, 5, "mixed"), (36, 72, 1, 5, "stream"),
    (100, 60, 2, 5, "mixed"), (132, 96, 3, 0, "stream"), (256, 64, 5, -1, "stream"), (260, 100, 7, 5, "noise"),
    (1100, 40, 8, 5, "mixed"), (2200, 24, 8, 5, "stream"), (320, 200, 8, 2000, "noise"), (320, 200, 8, 5, "flat"),
    (508, 260, 8, 5, "mixed"), (508, 260, 4, 0x7FFFFFFE, "mixed"),
])
def test_intra_rows_match_oracle(w, h, sa, thr, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.encoder import Encoder
    f = frame(kind, w, h, seed=w * 1000 + h + sa)
    ref = oracle.encode_stream(f[None], sa, thr, 16)[0]
    enc = Encoder(w, h, sa, thr, 16)
    try:
        for _ in range(2):  # the second frame finds the first one's leftovers
            out = enc.encode_frame_host(f, is_intra=True)
            np.testing.assert_array_equal(out.final, ref.final)
            np.testing.assert_array_equal(out.motion, ref.motion)
            np.testing.assert_array_equal(out.unique, ref.unique)
    finally:
        enc.close()
