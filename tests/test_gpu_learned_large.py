"""The exact test of the learned proposals on frames of more than 65,536 block
columns or rows, at the blocks past that number, against the oracle's refit."""
import ctypes

import numpy as np
import pytest

from test_gpu_inter_runs import frames
from test_gpu_learned_eval import expected

pytestmark = pytest.mark.gpu

LAST = 96  # block columns or rows checked, counted from the frame's end


@pytest.mark.parametrize("w,h,K", [(4 * (65536 + 16), 16, 8), (16, 4 * (65536 + 16), 4)])
def test_proposals_past_65536_block_columns_or_rows(w, h, K):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300._lib import check, lib
    from mptc_gb300.encoder import Encoder
    from mptc_gb300.model import ProposalModel
    sa, thr, bw, bh = 8, 100, w // 4, h // 4
    f = frames("stream", w, h, 2, seed=11)
    enc, m = Encoder(w, h, sa, thr, 16), ProposalModel(seed=7)
    try:
        enc.set_model(m, K)
        prev = enc.encode_frame_host(f[0], is_intra=True).final.copy()
        o = enc.encode_frame_host(f[1], is_intra=False, want_stb=True)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        topk = torch.empty((bw * bh, 16), dtype=torch.int16, device="cuda")
        rgb_d, stb_d, prev_d = dev(f[1]), dev(o.stb.view(np.int64)), dev(prev.view(np.int64))
        check(lib().mptc_learned_proposals(enc.handle, rgb_d.data_ptr(), stb_d.data_ptr(), prev_d.data_ptr(),
                                           topk.data_ptr(), ctypes.c_void_p(0)), enc.handle)
        # the frame's end as a frame of its own; its first sa columns or rows, whose
        # windows reach before it, are left out below
        x0, y0 = max(0, bw - LAST), max(0, bh - LAST)
        end = lambda a: np.ascontiguousarray(a.reshape(bh, bw, -1)[y0:, x0:])  # noqa: E731
        cbw = bw - x0
        want = expected(f[1][4 * y0:, 4 * x0:], end(o.stb).reshape(-1), end(prev).reshape(-1),
                        end(topk.cpu().numpy().view(np.uint16)).reshape(-1, 16), cbw, sa, K, thr)
        fin, mot = end(o.final).reshape(-1), end(o.motion).reshape(-1, 2)
        passed = 0
        for idx, x in enumerate(want):
            by, bx = divmod(idx, cbw)
            if x is None or (x0 and bx < sa) or (y0 and by < sa):
                continue
            passed += bx + x0 >= 65536 or by + y0 >= 65536
            row, col = divmod(x[0], 2 * sa)
            assert (int(mot[idx, 0]), int(mot[idx, 1])) == (col | 0x80, row | 0x80), (by, bx)
            assert int(fin[idx]) == x[1], (by, bx)
        assert passed > 0
    finally:
        enc.close()
        m.close()
