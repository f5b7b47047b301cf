"""The endpoint transform and the decoder's kernels against a plain numpy
restatement: tile values over the whole range of the words, coefficient buffers
at any byte offset, and motion codes whose copies form no chain, short chains, a
chain per row and one chain through the whole frame; several frames of a decoder
in a row (its scan state is reused), valid and invalid ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def div(a, b):  # C division
    return np.where(a < 0, -((-a) // b), a // b)


def i16(a):
    return a.astype(np.int64).astype(np.uint16).view(np.int16).astype(np.int64)


def lift(p, inverse):
    """The 5/3 wavelet of one 64x64 tile, level by level."""
    p = p.astype(np.int64)
    mirror = lambda i, n: abs(i) if i < n else 2 * n - 2 - i  # noqa: E731
    for dim in ([2, 4, 8, 16, 32, 64] if inverse else [64, 32, 16, 8, 4, 2]):
        h = dim // 2
        for axis in ((1, 0) if inverse else (0, 1)):
            v = p[:dim, :dim] if axis == 0 else p[:dim, :dim].T
            o = np.zeros_like(v)
            if inverse:
                for k in range(h):
                    o[2 * k] = i16(v[k] - div(v[h + mirror(2 * k - 1, dim) // 2] + v[h + k] + 2, 4))
                for k in range(h):
                    o[2 * k + 1] = i16(v[h + k] + div(o[2 * k] + o[mirror(2 * k + 2, dim)], 2))
            else:
                for k in range(h):
                    o[h + k] = i16(v[2 * k + 1] - div(v[2 * k] + v[mirror(2 * k + 2, dim)], 2))
                for k in range(h):
                    o[k] = i16(v[2 * k] + div(o[h + mirror(2 * k - 1, dim) // 2] + o[h + k] + 2, 4))
            p[:dim, :dim] = o if axis == 0 else o.T
    return p


def tiles(planes, f):
    out = planes.copy()
    for p in out:
        for y in range(0, p.shape[0], 64):
            for x in range(0, p.shape[1], 64):
                p[y:y + 64, x:x + 64] = f(p[y:y + 64, x:x + 64])
    return out


def i8(a):
    return a.astype(np.int64).astype(np.uint8).view(np.int8).astype(np.int64)


def forward(blocks, bw, bh):
    planes = []
    for ep in (0, 1):
        c = ((blocks >> np.uint64(16 * ep)) & np.uint64(0xFFFF)).astype(np.int64).reshape(bh, bw)
        r, g, b = c >> 11, c >> 5 & 63, c & 31
        t = r + b + (b >> 4)
        planes += [t + div(g - t, 2), r - b, g - t]
    return (i8(tiles(np.array(planes), lambda p: lift(p, False))) + 128).astype(np.uint8)


def endpoint_words(coeff, bw, bh):
    v = i8(tiles(coeff.reshape(6, bh, bw).astype(np.int64) - 128, lambda p: lift(p, True))).reshape(2, 3, -1)
    words = []
    for y, co, cg in v:
        t = i8(y - div(cg, 2))
        g = i8(cg + t)
        b = i8(div(t - co, 2))
        r = i8(b + co)
        words.append(((((r << 6) & 0xFFFF) | (g & 0xFFFF)) << 5 & 0xFFFF) | (b & 0xFFFF))
    return words


def index_words(motion, palette, prev, bw, sa):
    n, rank = motion.size // 2, 0
    out = np.zeros(n, np.int64)
    for i in range(n):
        x, y = int(motion[2 * i]), int(motion[2 * i + 1])
        if x == 255 and y == 255:
            out[i] = palette[rank]
            rank += 1
        elif x & 0x80 and y & 0x80:
            out[i] = prev[i + ((y & 0x7F) - sa) * bw + (x & 0x7F) - sa]
        else:
            out[i] = out[i + (y - 2 * sa + 1) * bw + x - sa]
    return out


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("w,h,offset", [(256, 256, 0), (256, 512, 1), (768, 256, 2), (512, 256, 3), (512, 512, 4)])
def test_forward_tiles(torch_cuda, w, h, offset):
    from mptc_gb300.decoder import endpoint_coefficients
    torch = torch_cuda
    bw, bh = w // 4, h // 4
    n = bw * bh
    blocks = np.random.default_rng(w + offset).integers(0, 1 << 63, n, dtype=np.int64)
    blocks[: n // 2] &= ~0xFFFF  # half with endpoint 1 black: flat tiles
    buf = torch.zeros(6 * n + 8, dtype=torch.uint8, device="cuda")
    endpoint_coefficients(w, h, torch.from_numpy(blocks).cuda(), buf[offset:offset + 6 * n])
    np.testing.assert_array_equal(buf[offset:offset + 6 * n].cpu().numpy(),
                                  forward(blocks.view(np.uint64), bw, bh).reshape(-1))
    assert not buf[:offset].any() and not buf[offset + 6 * n:].any()


def codes(rng, kind, bw, bh, sa, first):
    n = bw * bh
    m = np.full((n, 2), 255, np.uint8)
    bx, by = np.arange(n) % bw, np.arange(n) // bw
    if kind == "unique":
        return m
    left = np.array([sa - 1, 2 * sa - 1], np.uint8)
    if kind == "frame":  # every block copies the one before it
        m[1:] = left
    elif kind == "rows":  # a chain per row, up to the block above at its start
        m[bx > 0] = left
        m[(bx == 0) & (by % 3 > 0)] = (sa, 2 * sa - 2)
    else:
        for i in range(1, n):
            u = rng.random()
            dx, dy = int(rng.integers(-sa, sa)), int(rng.integers(0, 2 * sa))
            src = i - dy * bw + dx
            if u < 0.7 and 0 <= src < i:
                m[i] = (dx + sa, 2 * sa - 1 - dy)
            elif u < 0.9 and not first:
                dy = int(rng.integers(-sa, sa))
                if 0 <= i + dy * bw + dx < n:
                    m[i] = (dx + sa | 0x80, dy + sa | 0x80)
    return m


@pytest.mark.parametrize("w,h,sa,offset", [(256, 256, 8, 0), (768, 256, 1, 1), (512, 512, 40, 3)])
def test_decoder_frames(torch_cuda, w, h, sa, offset):
    from mptc_gb300._lib import MptcError
    from mptc_gb300.decoder import Decoder
    torch = torch_cuda
    bw, bh = w // 4, h // 4
    n = bw * bh
    rng = np.random.default_rng(w + sa)
    dec = Decoder(w, h, sa)
    prev = None
    try:
        for k, kind in enumerate(["mixed", "frame", "mixed", "rows", "invalid", "unique", "mixed"]):
            coeff = rng.integers(0, 256, 6 * n, dtype=np.uint8)
            motion = codes(rng, "mixed" if kind == "invalid" else kind, bw, bh, sa, prev is None)
            count = int((motion == 255).all(1).sum())
            palette = rng.integers(0, 1 << 32, count, dtype=np.uint32)
            buf = torch.zeros(6 * n + 8, dtype=torch.uint8, device="cuda")
            c = buf[offset:offset + 6 * n]
            c.copy_(torch.from_numpy(coeff))
            m = torch.from_numpy(motion.reshape(-1)).cuda()
            if kind == "invalid":  # a palette one entry short
                dec.decode_frame(m, c, torch.from_numpy(palette[:-1].view(np.int32)).cuda())
                with pytest.raises(MptcError):
                    dec.check()
                palette[-1] = 0
                got = dec._frames[dec._cur].cpu().numpy().view(np.uint64)
            else:
                got = dec.decode_frame(m, c, torch.from_numpy(palette.view(np.int32)).cuda())
                got = got.cpu().numpy().view(np.uint64)
                dec.check()
            words = index_words(motion.reshape(-1), palette, prev, bw, sa)
            e1, e2 = endpoint_words(coeff, bw, bh)
            want = (e1 | e2 << 16).astype(np.uint64) | words.astype(np.uint64) << np.uint64(32)
            np.testing.assert_array_equal(got, want, err_msg=f"frame {k}, {kind}")
            prev = words
    finally:
        dec.close()


@pytest.mark.parametrize("form", ["strided", "wider", "cpu", "numpy"])
def test_decoder_input_forms(torch_cuda, form):
    """Inputs that are not plain CUDA byte tensors are staged: the same blocks."""
    from mptc_gb300.decoder import Decoder
    torch = torch_cuda
    rng = np.random.default_rng(5)
    n, sa = 64 * 64, 8
    coeff = rng.integers(0, 256, 6 * n, dtype=np.uint8)
    motion = codes(rng, "mixed", 64, 64, sa, True).reshape(-1)
    palette = rng.integers(0, 1 << 32, int((motion.reshape(-1, 2) == 255).all(1).sum()), dtype=np.uint32)
    t = [torch.from_numpy(a.copy()) for a in (motion, coeff, palette.view(np.int32))]
    dec = Decoder(256, 256, sa)
    try:
        want = dec.decode_frame(*[x.cuda() for x in t]).cpu()
        if form == "strided":
            args = [x.cuda().repeat_interleave(2)[::2] for x in t]
        elif form == "wider":
            args = [t[0].cuda().to(torch.int32), t[1].cuda().to(torch.int64), t[2].cuda()]
        else:
            args = t if form == "cpu" else [motion, coeff, palette]
        assert torch.equal(dec.decode_frame(*args).cpu(), want)
        with pytest.raises(RuntimeError):
            dec.decode_frame(t[0].cuda().view(-1, 2), t[1].cuda(), t[2].cuda())
    finally:
        dec.close()


def test_decoder_on_another_stream(torch_cuda):
    """Inputs read in place on a stream that is not their own, freed and overwritten
    right after the call."""
    from mptc_gb300.decoder import Decoder
    torch = torch_cuda
    rng = np.random.default_rng(8)
    n, sa = 64 * 64, 8
    coeff = rng.integers(0, 256, 6 * n, dtype=np.uint8)
    motion = codes(rng, "mixed", 64, 64, sa, True).reshape(-1)
    palette = rng.integers(0, 1 << 32, int((motion.reshape(-1, 2) == 255).all(1).sum()), dtype=np.uint32)
    host = [torch.from_numpy(a.copy()) for a in (motion, coeff, palette.view(np.int32))]
    dec, s = Decoder(256, 256, sa), torch.cuda.Stream()
    try:
        want = dec.decode_frame(*[x.cuda() for x in host]).cpu()
        for _ in range(4):
            args = [x.cuda() for x in host]
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                torch.cuda._sleep(2000000)  # the decode starts after the inputs are gone
            got = dec.decode_frame(*args, stream=s)
            shapes = [a.shape for a in args]
            del args
            junk = [torch.full(sh, 77, dtype=x.dtype, device="cuda") for sh, x in zip(shapes, host)]
            s.synchronize()
            assert torch.equal(got.cpu(), want)
            del junk
    finally:
        dec.close()
