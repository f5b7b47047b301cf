"""Palettes that are not 32-bit words: their length is that of their elements, so
that they do not fit as words and are refused, also as CUDA tensors, which are
read in place where they fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["cuda", "cpu"])
@pytest.mark.parametrize("dtype", ["int64", "uint8", "int16"])
def test_palettes_of_another_element_size_are_refused(dtype, where):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.decoder import Decoder
    n = 64 * 64
    motion = torch.full((2 * n,), 255, dtype=torch.uint8, device="cuda")
    coeff = torch.full((6 * n,), 128, dtype=torch.uint8, device="cuda")
    words = torch.from_numpy(np.random.default_rng(3).integers(0, 1 << 32, n, dtype=np.uint32).view(np.int32))
    dec = Decoder(256, 256, 8)
    try:
        with pytest.raises(RuntimeError):
            dec.decode_frame(motion, coeff, words.to(getattr(torch, dtype)).to(where))
        got = dec.decode_frame(motion, coeff, words.to(where)).cpu()  # the decoder is as it was
        dec.check()
        assert torch.equal((got >> 32) & 0xFFFFFFFF, words.to(torch.int64) & 0xFFFFFFFF)
    finally:
        dec.close()


def test_first_frame_on_a_stream_of_its_own():
    """A decoder's scan state is ready when the decoder is, also while the stream that
    zeroed it has earlier work queued: its first frames on a stream that does not wait
    for that one, without and with a decoder used before in the same memory."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mptc_gb300.decoder import Decoder
    w, h = 768, 512
    n = w * h // 16
    motion = torch.full((2 * n,), 255, dtype=torch.uint8, device="cuda")
    coeff = torch.full((6 * n,), 128, dtype=torch.uint8, device="cuda")
    words = torch.from_numpy(np.random.default_rng(4).integers(0, 1 << 32, n, dtype=np.uint32).view(np.int32)).cuda()
    want, s = words.cpu().to(torch.int64) & 0xFFFFFFFF, torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(6):
        torch.cuda._sleep(20_000_000)  # about 10 ms on the default stream
        dec = Decoder(w, h, 8)
        try:
            for _ in range(2):
                got = dec.decode_frame(motion, coeff, words, stream=s)
                dec.check(stream=s)
                with torch.cuda.stream(s):
                    assert torch.equal((got >> 32).cpu() & 0xFFFFFFFF, want)
        finally:
            dec.close()
