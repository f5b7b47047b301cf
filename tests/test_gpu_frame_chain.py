"""The chain of a frame's kernels, each started while the one before it still
runs, against the oracle: frames queued back to back on one context without a
synchronisation between them, as encode_frame, as stb encode and reencode, and
captured into a CUDA graph that is replayed twice. The smallest frames have more
work words to zero than blocks; sa 12 takes the kernels of larger windows."""
import numpy as np
import pytest

import oracle
from mptc_gb300.synth import StreamSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sa", [(4, 4, 8), (8, 4, 12), (64, 64, 8), (260, 132, 8), (640, 360, 8), (320, 200, 12)])
@pytest.mark.parametrize("how", ["frames", "split", "captured"])
def test_queued_frames_match_oracle(w, h, sa, how):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.encoder import Encoder
    n, nblk = 6, w * h // 16
    intra = [True, False, False, True, False, False]
    f = StreamSpec(w, h, n, seed=w + h, square_size=min(48, w, h), n_squares=3).generate()
    ref = []
    for k in (0, 3):  # two runs of one intra and two inter frames
        ref += oracle.encode_stream(f[k:k + 3], sa, 5, 16, threads=8)
    dev = torch.from_numpy(f).cuda()
    i64 = dict(dtype=torch.int64, device="cuda")
    fin, stb = torch.zeros((n, nblk), **i64), torch.zeros((n, nblk), **i64)
    orig = torch.zeros((n, nblk), dtype=torch.int32, device="cuda")
    mot = torch.zeros((n, 2 * nblk), dtype=torch.uint8, device="cuda")
    uni = torch.zeros((n, nblk), dtype=torch.int32, device="cuda")
    nu = torch.zeros((n, 1), dtype=torch.int32, device="cuda")
    enc = Encoder(w, h, sa, 5, 16)
    s = torch.cuda.Stream()

    def queue():
        for k in range(n):
            prev = None if intra[k] else fin[k - 1]
            if how == "split":
                enc.dxt1_encode_device(dev[k], stb[k], orig[k], stream=s)
                enc.reencode_device(dev[k], stb[k], orig[k], prev, fin[k], mot[k], uni[k], nu[k], stream=s)
            else:
                enc.encode_frame_device(dev[k], prev, None, fin[k], mot[k], uni[k], nu[k], stream=s)

    try:
        torch.cuda.synchronize()
        if how == "captured":
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                queue()
            for _ in range(2):
                g.replay()
        else:
            queue()
        torch.cuda.synchronize()
        for k in range(n):
            m = int(nu[k, 0])
            np.testing.assert_array_equal(fin[k].cpu().numpy().view(np.uint64), ref[k].final, err_msg=f"frame {k}")
            np.testing.assert_array_equal(mot[k].cpu().numpy(), np.asarray(ref[k].motion).reshape(-1))
            np.testing.assert_array_equal(uni[k, :m].cpu().numpy().view(np.uint32), ref[k].unique)
    finally:
        enc.close()
