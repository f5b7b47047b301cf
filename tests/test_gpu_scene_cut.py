"""Inter frames after a scene cut, whose fixed-point sweeps do not converge and are
given up, against the oracle: every sweep count (one sweep cannot be given up, two
only after the first), windows of both kinds, and cuts between frames of which
some blocks still find their word."""
import numpy as np
import pytest

import oracle
from mptc_gb300.synth import StreamSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sa", [(256, 256, 8), (640, 360, 8), (320, 200, 3), (256, 160, 24)])
@pytest.mark.parametrize("sweeps", [0, 1, 2, 12])
def test_frame_after_a_cut(w, h, sa, sweeps):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.encoder import Encoder
    a, b = [StreamSpec(w, h, 2, seed=s, square_size=48, n_squares=2).generate() for s in (w, h + 1)]
    mixed = a[1].copy()
    mixed[:, w // 2:] = b[1][:, w // 2:]
    f = np.stack([a[0], b[0], mixed, b[1]])
    ref = oracle.encode_stream(f, sa, 5, 16, threads=16)
    enc = Encoder(w, h, sa, 5, 16, intra_sweeps=sweeps)
    try:
        for k in range(len(f)):
            out = enc.encode_frame_host(f[k], is_intra=k == 0)
            np.testing.assert_array_equal(out.final, ref[k].final, err_msg=f"frame {k}")
            np.testing.assert_array_equal(out.motion, ref[k].motion, err_msg=f"frame {k}")
            np.testing.assert_array_equal(out.unique, ref[k].unique, err_msg=f"frame {k}")
    finally:
        enc.close()
