"""The training step's products at the sizes where their tiles, slices and
candidate groups end: one example, batches around 128 rows (a tile, and the
smallest slice of a split reduction), candidate counts around multiples of 8 and
the largest, a batch large enough for 128-column tiles and many slices. Loss and
gradients against the CPU reference within the BF16 bounds of test_gpu_learned,
and the same bits from a second step."""
import numpy as np
import pytest

from test_gpu_learned import GRAD_TOL, bf, block_features, cand_features, layers, make_batch, mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C", [(1, 2), (1, 64), (127, 3), (128, 8), (129, 9), (256, 33), (300, 64), (1000, 17),
                                 (4096, 7)])
def test_gradients_at_tile_edges(B, C):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.model import ProposalModel, param_slices
    b = make_batch(torch, w=256, h=256, B=B, C=C, seed=B + C)
    m = ProposalModel(seed=3)
    try:
        args = (b["rgb_d"], b["w"], b["stb_d"], b["blocks_d"], b["cands_d"])
        loss_gpu, g_gpu = m.grads(*args)
        assert np.array_equal(g_gpu, m.grads(*args)[1])
        p, Ws = layers(torch, m.params())
        hf, tf = mlp(torch, Ws, torch.tensor(block_features(b["frame"], b["stb"], b["blocks"], b["bw"])), [0, 1, 2])
        hg, tg = mlp(torch, Ws, torch.tensor(cand_features(b["cands"])), [3, 4])
        scores = (hf[:, None, :] * hg.view(B, C, 64)).sum(-1)
        loss = torch.nn.functional.cross_entropy(scores, torch.zeros(B, dtype=torch.long))
        loss.backward()
        ref = float(loss.detach())
        assert abs(loss_gpu - ref) <= 2.0 ** -6 * abs(ref) + 1e-4
        sl, _ = param_slices()
        with torch.no_grad():
            for chain, ids in ((tf, [0, 1, 2]), (tg, [3, 4])):
                M = chain[-1][1].grad.abs()
                for pos in range(len(ids) - 1, -1, -1):
                    inp, _ = chain[pos]
                    (a, e, shp), (c, d, _) = sl[ids[pos]]
                    ew = (torch.tensor(g_gpu[a:e]).view(*shp) - p.grad[a:e].view(*shp)).abs()
                    eb = (torch.tensor(g_gpu[c:d]) - p.grad[c:d]).abs()
                    assert bool((ew <= GRAD_TOL * (inp.abs().t() @ M) + 1e-7).all()), (ids[pos], "weight")
                    assert bool((eb <= GRAD_TOL * M.sum(0) + 1e-7).all()), (ids[pos], "bias")
                    if pos > 0:
                        M = (M @ bf(torch, Ws[ids[pos]][0]).abs().t()) * (chain[pos - 1][1] > 0).float()
    finally:
        m.close()
