"""The exact test of the learned proposals (learned_eval_kernel) against the
oracle's refit: every block whose proposals pass gets the position and block that
the reference's selection over its proposals gives, and the others are counted as
fallbacks. Frames of one and of many groups of blocks, with a last group that is
not full, 4, 8 and 16 proposals, thresholds that pass nothing, only err_diff <= 0
and everything, and content with near ties of the refit."""
import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_inter_runs import frames

pytestmark = pytest.mark.gpu


def expected(frame, stb, prev, topk, bw, sa, K, thr):
    """Per block (position, block), or None where no proposal passes."""
    w2, out = 2 * sa, []
    for idx in range(stb.size):
        by, bx = divmod(idx, bw)
        px = frame[4 * by:4 * by + 4, 4 * bx:4 * bx + 4].reshape(48)
        orig = oracle.block_error(px, int(stb[idx]))
        m, sel, rows = None, None, set()
        for p in sorted(int(q) for q in topk[idx, :K] if q != 0xFFFF):
            row = p // w2
            if row in rows:  # the row ended at an err_diff <= 0
                continue
            word = int(prev[(by - sa + row) * bw + bx - sa + p % w2]) >> 32
            if word == int(stb[idx]) >> 32:
                e, blk = 0, int(stb[idx])
            else:
                err, e1, e2, valid = oracle.refit(px, word)
                if not valid:
                    continue
                q1, q2 = [(int(c[0]) >> 3) << 11 | (int(c[1]) >> 2) << 5 | int(c[2]) >> 3 for c in (e1, e2)]
                e, blk = err - orig, q1 | q2 << 16 | word << 32
            if m is None or e < m:
                m, sel = e, (p, blk)
                if e <= 0:
                    m = 0
                    rows.add(row)
        out.append(sel if m is not None and m <= thr else None)
    return out


@pytest.mark.parametrize("w,h,sa,K,thr,kind", [
    (4, 4, 8, 8, 5, "stream"), (36, 20, 8, 4, 5, "steps"), (132, 100, 8, 16, 5, "steps"), (260, 132, 8, 8, 0, "steps"),
    (256, 128, 6, 8, -1, "stream"), (256, 128, 3, 16, 0x7FFFFFFE, "flat"), (640, 360, 8, 8, 5, "stream"),
    (856, 480, 8, 4, 40, "flat"),
])
def test_proposals_are_tested_exactly(w, h, sa, K, thr, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300._lib import check, lib
    from mptc_gb300.encoder import Encoder
    from mptc_gb300.model import ProposalModel
    bw, n = w // 4, w * h // 16
    f = frames(kind, w, h, 2, seed=w + h + K)
    enc, m = Encoder(w, h, sa, thr, 16), ProposalModel(seed=7)
    try:
        enc.set_model(m, K)
        prev = enc.encode_frame_host(f[0], is_intra=True).final.copy()
        o = enc.encode_frame_host(f[1], is_intra=False, want_stb=True)
        fin, mot, stb, fallbacks = o.final.copy(), o.motion.copy(), o.stb.copy(), enc.stats().n_fallback
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        topk = torch.empty((n, 16), dtype=torch.int16, device="cuda")
        rgb_d, stb_d, prev_d = dev(f[1]), dev(stb.view(np.int64)), dev(prev.view(np.int64))
        check(lib().mptc_learned_proposals(enc.handle, rgb_d.data_ptr(), stb_d.data_ptr(), prev_d.data_ptr(),
                                           topk.data_ptr(), ctypes.c_void_p(0)), enc.handle)
        tk = topk.cpu().numpy().view(np.uint16)
        want = expected(f[1], stb, prev, tk, bw, sa, K, thr)
        assert fallbacks == sum(x is None for x in want)
        for idx, x in enumerate(want):
            if x is not None:
                row, col = divmod(x[0], 2 * sa)
                assert (int(mot[2 * idx]), int(mot[2 * idx + 1])) == (col | 0x80, row | 0x80), idx
                assert int(fin[idx]) == x[1], idx
    finally:
        enc.close()
        m.close()
