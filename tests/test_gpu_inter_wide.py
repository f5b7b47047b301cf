"""The inter search of windows wider than 16 (inter_wide_kernel) against the
oracle at the sizes where it can go wrong: search areas 9 to 63, frames narrower
than a run and than the window, runs of 1 to 8 blocks, thresholds whose ranks lie at
the ends of their 16 bits, flat blocks, near-ties of the refit, and noise (unions
of more distinct words than the table takes, alone and beside smooth content)."""
import numpy as np
import pytest

import oracle
from test_gpu_inter_runs import frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sa,thr,kind", [
    (4, 4, 9, 5, "stream"), (12, 72, 63, 5, "steps"), (36, 20, 9, 5, "steps"), (132, 96, 12, 0, "stream"),
    (256, 128, 16, -1, "stream"), (260, 100, 17, 5, "steps"), (600, 400, 9, 5, "stream"), (428, 160, 63, 5, "stream"),
    (500, 300, 24, 70000, "steps"), (320, 200, 24, 0x7FFFFFFE, "flat"), (160, 120, 24, 300, "noise"),
    (128, 64, 63, 5, "noise"), (856, 480, 24, 5, "stream"), (700, 260, 31, 40, "mixed"),
])
def test_inter_wide_matches_oracle(w, h, sa, thr, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.encoder import Encoder
    n = 2
    f = frames("stream" if kind == "mixed" else kind, w, h, n, seed=w * 1000 + h + sa)
    if kind == "mixed":  # noise in the frame's middle
        f[:, h // 3:h // 2, w // 3:2 * w // 3] = frames("noise", w, h, n, seed=3)[:, h // 3:h // 2, w // 3:2 * w // 3]
    ref = oracle.encode_stream(f, sa, thr, 16, threads=16)
    enc = Encoder(w, h, sa, thr, 16)
    try:
        for k in range(n):
            out = enc.encode_frame_host(f[k], is_intra=k == 0)
            np.testing.assert_array_equal(out.final, ref[k].final, err_msg=f"frame {k}")
            np.testing.assert_array_equal(out.motion, ref[k].motion, err_msg=f"frame {k}")
            np.testing.assert_array_equal(out.unique, ref[k].unique, err_msg=f"frame {k}")
    finally:
        enc.close()
