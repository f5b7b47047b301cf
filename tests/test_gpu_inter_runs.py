"""The run search of inter frames (inter_run_kernel) against the oracle at the
sizes where it can go wrong: search areas 1 to 8, frames narrower than a run, of
partial runs and too small to give every warp a run of 8 blocks, thresholds
whose ranks lie at the ends of their 16 bits, flat blocks (words whose refit is
degenerate), near-ties of the refit, and noise (runs that overflow the table)."""
import numpy as np
import pytest

import oracle
from mptc_gb300.synth import StreamSpec

pytestmark = pytest.mark.gpu


def frames(kind, w, h, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "noise":
        return rng.integers(0, 256, (n, h, w, 3), dtype=np.uint8)
    if kind == "steps":  # few levels: refits that fall exactly between two values
        f = np.repeat(np.repeat(rng.integers(0, 4, (n, (h + 1) // 2, (w + 1) // 2, 3)) * 21, 2, 1), 2, 2)[:, :h, :w]
        return (f + rng.integers(0, 2, f.shape)).astype(np.uint8)
    if kind == "flat":  # constant blocks with an odd pixel now and then
        f = np.repeat(np.repeat(rng.integers(0, 256, (1, h // 4, w // 4, 3)), 4, 1), 4, 2).repeat(n, 0)
        return np.where(rng.random((n, h, w, 1)) < 0.02, rng.integers(0, 256, (n, h, w, 3)), f).astype(np.uint8)
    return StreamSpec(w, h, n, seed=seed, square_size=min(48, w, h), n_squares=2).generate()


@pytest.mark.parametrize("w,h,sa,thr,kind", [
    (4, 4, 8, 5, "stream"), (12, 72, 8, 5, "steps"), (36, 20, 1, 5, "steps"), (100, 64, 2, 5, "stream"),
    (132, 96, 3, 0, "stream"), (256, 128, 5, -1, "stream"), (260, 100, 7, 5, "steps"), (256, 256, 8, 5, "stream"),
    (256, 256, 8, 70000, "noise"), (128, 128, 8, 0x7FFFFFFE, "steps"), (320, 200, 8, 5, "flat"),
    (320, 200, 6, 40, "flat"), (508, 260, 8, 5, "steps"), (1284, 724, 8, 5, "stream"), (400, 200, 8, 300, "noise"),
])
def test_inter_runs_match_oracle(w, h, sa, thr, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.encoder import Encoder
    f = frames(kind, w, h, 3, seed=w * 1000 + h + sa)
    ref = oracle.encode_stream(f, sa, thr, 16, threads=8)
    enc = Encoder(w, h, sa, thr, 16)
    try:
        for k in range(3):
            out = enc.encode_frame_host(f[k], is_intra=k == 0)
            np.testing.assert_array_equal(out.final, ref[k].final, err_msg=f"frame {k}")
            np.testing.assert_array_equal(out.motion, ref[k].motion, err_msg=f"frame {k}")
            np.testing.assert_array_equal(out.unique, ref[k].unique, err_msg=f"frame {k}")
    finally:
        enc.close()
