"""The row pipeline with two CTAs per SM (intra_rows_kernel<2>) against the oracle. It
runs the intra frames of several streams side by side: batches of two, and of three and
more streams, whose frames take fewer clusters the narrower they are, as a run and step
by step. And frames by themselves from 640 block columns and 39 block
rows on."""
import numpy as np
import pytest

import oracle
from test_gpu_intra_rows import frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,sa,kind", [
    ([(36, 72), (1100, 40)], 8, "mixed"), ([(4, 80), (260, 100), (2200, 24)], 8, "mixed"),
    ([(412, 64), (420, 60), (508, 260), (64, 200)], 8, "noise"), ([(132, 96)] * 5, 3, "stream"),
])
def test_frames_side_by_side_match_oracle(sizes, sa, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.batch import BatchEncoder
    f = [frame(kind, w, h, seed=w * 10 + h + i) for i, (w, h) in enumerate(sizes)]
    ref = [oracle.encode_stream(x[None], sa, 5, 16)[0] for x in f]
    b = BatchEncoder(sizes, sa, 5, 16)
    try:
        outs = []
        for i, x in enumerate(f):
            n, z = b.nblk(i), lambda m, t: torch.zeros((1, m), dtype=t, device="cuda")  # noqa: E731
            outs.append((torch.from_numpy(x[None].copy()).cuda(), z(n, torch.int64), z(2 * n, torch.uint8),
                         z(n, torch.int32), torch.zeros(1, dtype=torch.int32, device="cuda")))
        for _ in range(2):  # the second run finds the first one's leftovers
            b.encode_run(*zip(*outs), [[True]] * len(sizes))
            for r, (_, fin, mot, uni, nu) in zip(ref, outs):
                np.testing.assert_array_equal(fin.cpu().numpy().view(np.uint64)[0], r.final)
                np.testing.assert_array_equal(mot.cpu().numpy()[0], r.motion)
                np.testing.assert_array_equal(uni.cpu().numpy().view(np.uint32)[0, :int(nu)], r.unique)
        for i, x in enumerate(f):
            b.upload(i, x)
        b.encode([True] * len(sizes))
        for i, r in enumerate(ref):
            fin, mot, uni = b.fetch(i)
            np.testing.assert_array_equal(fin, r.final)
            np.testing.assert_array_equal(mot, r.motion)
            np.testing.assert_array_equal(uni, r.unique)
    finally:
        b.close()


@pytest.mark.parametrize("w,h,sa,kind", [(2556, 160, 8, "mixed"), (2560, 152, 8, "mixed"), (2560, 156, 8, "noise"),
                                         (2564, 340, 1, "stream"), (3840, 200, 2, "mixed")])
def test_wide_frames_match_oracle(w, h, sa, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.encoder import Encoder
    f = frame(kind, w, h, seed=w + h + sa)
    ref = oracle.encode_stream(f[None], sa, 5, 16, threads=8)[0]
    enc = Encoder(w, h, sa, 5, 16)
    try:
        for _ in range(2):
            out = enc.encode_frame_host(f, is_intra=True)
            np.testing.assert_array_equal(out.final, ref.final)
            np.testing.assert_array_equal(out.motion, ref.motion)
            np.testing.assert_array_equal(out.unique, ref.unique)
    finally:
        enc.close()
