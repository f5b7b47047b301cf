"""Workloads of the encoder, the learned proposal and the decoder for timing.

Every case runs through the package's public entry points on seeded synthetic
video made on the GPU: per channel the sum of four low-frequency sinusoids,
square patches of noise texture that move a few pixels per frame, and uniform
noise in [-4, 4], the content the package's own workloads are defined on.
Frame sizes are those of the package's workloads (256x256 to 3840x2160) and
whatever lies between, in multiples of 4 pixels (of 256 for the endpoint
images); the encoder's parameters are its defaults (search area 8, threshold
5, intra interval 16) except where a case says otherwise.
"""
import math

import numpy as np
import torch

from mptc_gb300.batch import BatchEncoder
from mptc_gb300.decoder import Decoder, endpoint_coefficients
from mptc_gb300.encoder import Encoder, StreamOutput, intra_schedule
from mptc_gb300.model import ProposalModel

LAYERS = [(64, 128), (128, 128), (128, 64), (32, 128), (128, 64)]  # f1 f2 f3, g1 g2
THR, INTERVAL = 5, 16


def listed():
    return [
        # a thumbnail or preview stream: single calls on small frames, where launches and latency count
        dict(name="intra_256", kind="frame", w=256, h=256, sa=8, intra=True, squares=1),
        dict(name="inter_256", kind="frame", w=256, h=256, sa=8, intra=False, squares=1),
        # the call a device-resident pipeline makes per 1080p frame
        dict(name="intra_1080p", kind="frame", w=1920, h=1080, sa=8, intra=True, squares=1),
        dict(name="inter_1080p", kind="frame", w=1920, h=1080, sa=8, intra=False, squares=1),
        # a wide search area (the command line takes up to 63) on a moving, textured frame of odd size
        dict(name="inter_wide_856x480", kind="frame", w=856, h=480, sa=24, intra=False, squares=4),
        # whole runs: device-resident, and from pinned host memory with a scene cut
        dict(name="stream_1080p", kind="stream", w=1920, h=1080, sa=8, frames=32, squares=1, cut=0, k=0),
        dict(name="host_720p", kind="host", w=1280, h=720, sa=8, frames=24, squares=4, cut=12, pinned=True),
        # the learned proposal: one stream, and several of different sizes in one batch
        dict(name="learned_1080p", kind="stream", w=1920, h=1080, sa=8, frames=16, squares=1, cut=0, k=8),
        dict(name="batch_mixed", kind="batch", streams=8, scale=1.0, frames=16, squares=1, k=8),
        # the stream's endpoint images, and decoding on the GPU
        dict(name="endpoints_2048x1280", kind="endpoints", w=2048, h=1280, frames=8),
        dict(name="decode_2048x1280", kind="decode", w=2048, h=1280, frames=8, squares=2),
        # one training step's loss and gradients at the training batch
        dict(name="train_4096x32", kind="train", B=4096, C=32),
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "stream", "stream", "host", "batch", "endpoints", "decode", "train"])
    w, h = _log(rng, 64, 2560, 4), _log(rng, 64, 1440, 4)
    sa = rng.choice([8, 8, 8, 8, rng.randint(1, 7), rng.randint(9, 63)])
    sq = rng.choice([0, 1, 1, 2, 4, 8])
    if kind == "frame":
        if sa > 8:
            w, h = (min(w, 856), min(h, 480)) if sa <= 24 else (min(w, 428), min(h, 160))
        return dict(kind=kind, w=w, h=h, sa=sa, intra=rng.random() < 0.4, squares=sq)
    if kind == "stream":
        w, h, sa = min(w, 1920), min(h, 1080), min(sa, 8)
        return dict(kind=kind, w=w, h=h, sa=sa, frames=rng.randint(3, 24), squares=sq, cut=rng.choice([0, 0, 10]),
                    k=rng.choice([0, 0, 4, 8, 16]))
    if kind == "host":
        return dict(kind=kind, w=min(w, 1280), h=min(h, 720), sa=min(sa, 8), frames=rng.randint(2, 20), squares=sq,
                    cut=rng.choice([0, 7]), pinned=rng.random() < 0.6)
    if kind == "batch":
        return dict(kind=kind, streams=rng.randint(2, 8), scale=rng.choice([0.25, 0.5, 0.75, 1.0]),
                    frames=rng.randint(3, 14), squares=sq, k=rng.choice([0, 0, 8]))
    if kind in ("endpoints", "decode"):
        c = dict(kind=kind, w=256 * rng.randint(1, 8), h=256 * rng.randint(1, 5), frames=rng.randint(2, 8))
        return c if kind == "endpoints" else dict(c, squares=sq)
    return dict(kind="train", B=_log(rng, 100, 4096), C=rng.randint(2, 32))


# ---- inputs ---------------------------------------------------------------------
def _video(w, h, count, seed, squares, cut=0):
    """(count, h, w, 3) uint8 frames on the GPU."""
    dev = torch.device("cuda")
    p = np.random.default_rng(seed)
    g = torch.Generator(device=dev).manual_seed(seed)
    lo = 32 if w <= 1024 else 64 if w < 1920 or w > 1920 else 32
    y, x = torch.arange(h, device=dev)[:, None, None], torch.arange(w, device=dev)[None, :, None]

    def background():
        v = torch.full((h, w, 3), 128.0, device=dev)
        for _ in range(4):
            period, amp = p.integers(lo, 8 * lo + 1, 3), p.integers(20, 51, 3)
            phase, turn = p.random(3), p.random(3) * 2 * np.pi
            kx = torch.tensor(np.cos(turn) / period, dtype=torch.float32, device=dev)
            ky = torch.tensor(np.sin(turn) / period, dtype=torch.float32, device=dev)
            a, ph = (torch.tensor(t, dtype=torch.float32, device=dev) for t in (amp, phase))
            v += a * torch.sin(2 * math.pi * (x * kx + y * ky + ph))
        return v

    size = max(8, min(64 if w <= 1920 else 128, w // 4, h // 4))
    patch = [(int(p.integers(0, w)), int(p.integers(0, h)), p.integers(1, 5) * np.exp(2j * np.pi * p.random()),
              torch.randint(0, 256, (size, size, 3), device=dev, generator=g).float()) for _ in range(squares)]
    out = torch.empty((count, h, w, 3), dtype=torch.uint8, device=dev)
    span, v0 = torch.arange(size, device=dev), None
    for f in range(count):
        if v0 is None or (cut and f and f % cut == 0):
            v0 = background()
        v = v0.clone()
        for px, py, speed, tex in patch:
            rows = (int(py + f * speed.imag) + span) % h
            cols = (int(px + f * speed.real) + span) % w
            v[rows[:, None], cols[None, :]] = tex
        v += torch.randint(-4, 5, v.shape, device=dev, generator=g)
        out[f] = v.clamp_(0, 255).to(torch.uint8)
    return out


def _encoded(enc, frames, flags, stb=False):
    """The frames' outputs, one frame call each (device tensors per frame)."""
    got, prev, dev = [], None, frames.device
    for f, intra in zip(frames, flags):
        o = _outputs(enc.nblk)
        s = torch.empty(enc.nblk, dtype=torch.int64, device=dev) if stb else None
        enc.encode_frame_device(f, None if intra else prev, s, *o)
        prev = o[0]
        got.append((*o, s))
    return got


def _outputs(n, frames=None):
    lead = () if frames is None else (frames,)
    z = lambda m, t: torch.zeros((*lead, m), dtype=t, device="cuda")  # noqa: E731
    return (z(n, torch.int64), z(2 * n, torch.uint8), z(n, torch.int32),
            torch.zeros(frames or 1, dtype=torch.int32, device="cuda"))


def _features(rgb, stb, blocks, bw, dtype):
    """Block features: 48 channel values over the block's channel range, then
    both endpoints as 5/6/5-bit fractions, zero padded to 64."""
    h, w, _ = rgb.shape
    px = rgb.view(h // 4, 4, w // 4, 4, 3).permute(0, 2, 1, 3, 4).reshape(-1, 16, 3)[blocks].to(dtype)
    lo, hi = px.amin(1, keepdim=True), px.amax(1, keepdim=True)
    x = torch.where(hi > lo, (px - lo) / (hi - lo).clamp(min=1), torch.zeros_like(px)).reshape(-1, 48)
    b = stb[blocks]
    ends = [((b >> s) & m).to(dtype) / m for s, m in ((11, 31), (5, 63), (0, 31), (27, 31), (21, 63), (16, 31))]
    return torch.cat([x, torch.stack(ends, 1), torch.zeros(len(x), 10, dtype=dtype, device=x.device)], 1)


def _bits(words, dtype):
    return ((words[..., None].long() >> torch.arange(32, device=words.device)) & 1).to(dtype)


def _loss(params, x, bits):
    """Sampled softmax cross-entropy; candidate 0 of each row is the accepted one."""
    (w1, b1), (w2, b2), (w3, b3), (v1, c1), (v2, c2) = params
    f = torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2) @ w3 + b3
    g = torch.relu(bits @ v1 + c1) @ v2 + c2
    s = torch.einsum("be,bce->bc", f, g)
    return (torch.logsumexp(s, 1) - s[:, 0]).mean()


def _split(flat):
    out, o = [], 0
    for i, n in LAYERS:
        out.append((flat[o:o + i * n].view(i, n), flat[o + i * n:o + i * n + n]))
        o += i * n + n
    return out


def _he(seed):
    p, parts = np.random.default_rng(seed), []
    for k, (i, n) in enumerate(LAYERS):
        lim = math.sqrt(6.0 / (54 if k == 0 else i))
        w = p.uniform(-lim, lim, (i, n)).astype(np.float32)
        if k == 0:
            w[54:] = 0
        parts += [w.reshape(-1), np.zeros(n, np.float32)]
    return np.concatenate(parts)


_WEIGHTS = []


def _weights():
    """Weights of a trained proposal (the file such a program would load):
    trained once per process on the exhaustive search's decisions."""
    if _WEIGHTS:
        return _WEIGHTS[0]
    w, h, sa, nf = 1280, 720, 8, 6
    bw, bh = w // 4, h // 4
    frames = _video(w, h, nf, 5000, 1)
    enc = Encoder(w, h, sa, THR, INTERVAL)
    outs = _encoded(enc, frames, intra_schedule(nf, INTERVAL), stb=True)
    enc.close()
    g = torch.Generator(device="cuda").manual_seed(1)
    flat = torch.from_numpy(_he(1)).cuda().requires_grad_(True)
    opt = torch.optim.AdamW([flat], lr=1e-3, weight_decay=1e-4, foreach=False)
    for step in range(500):
        t = 1 + step % (nf - 1)
        m = outs[t][1].view(-1, 2).long()
        inter = torch.nonzero((m[:, 0] >= 128) & ~((m[:, 0] == 255) & (m[:, 1] == 255)))[:, 0]
        b = inter[torch.randint(0, len(inter), (2048,), device="cuda", generator=g)]
        bx, by = b % bw, b // bw
        words = outs[t - 1][0] >> 32 & 0xFFFFFFFF
        acc = words[(by + m[b, 1] - 128 - sa) * bw + bx + m[b, 0] - 128 - sa]
        dx, dy = (torch.randint(-sa, sa, (2048, 15), device="cuda", generator=g) for _ in range(2))
        neg = words[(by[:, None] + dy).clamp(0, bh - 1) * bw + (bx[:, None] + dx).clamp(0, bw - 1)]
        x = _features(frames[t], outs[t][4], b, bw, torch.float32)
        loss = _loss(_split(flat), x, _bits(torch.cat([acc[:, None], neg], 1), torch.float32))
        flat.grad = None
        loss.backward()
        opt.step()
    _WEIGHTS.append(flat.detach().cpu().numpy())
    return _WEIGHTS[0]


def _model():
    m = ProposalModel(seed=1)
    m.set_params(_weights())
    return m


def _train_inputs(case, seed):
    """One 640x360 frame, endpoints from each block's channel extremes, and
    candidate words of a few hundred distinct values, as final blocks hold."""
    w, h, B, C = 640, 360, case["B"], case["C"]
    rgb = _video(w, h, 1, seed, 2)[0]
    px = rgb.view(h // 4, 4, w // 4, 4, 3).permute(0, 2, 1, 3, 4).reshape(-1, 16, 3).long()
    pack = lambda c: (c[:, 0] >> 3 << 11) | (c[:, 1] >> 2 << 5) | (c[:, 2] >> 3)  # noqa: E731
    stb = pack(px.amax(1)) | (pack(px.amin(1)) << 16)
    p = np.random.default_rng(seed)
    pool = p.integers(0, 1 << 32, 400, dtype=np.uint64).astype(np.uint32)
    blocks = torch.from_numpy(p.integers(0, (w // 4) * (h // 4), B).astype(np.int32)).cuda()
    cands = torch.from_numpy(pool[p.integers(0, 400, (B, C))].view(np.int32)).cuda()
    return rgb, w, stb, blocks, cands


def _batch_sizes(case):
    sizes = [(856, 480), (1280, 720), (1920, 1080), (2560, 1440)]
    fit = lambda v: max(16, int(v * case["scale"]) // 4 * 4)  # noqa: E731
    return [tuple(map(fit, sizes[i % 4])) for i in range(case["streams"])]


def _model_k(case):
    return _model() if case["k"] else None


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        model = ProposalModel(seed=0)
        model.set_params(_he(seed + 1))
        return dict(kind=kind, model=model, args=_train_inputs(case, seed))
    if kind == "batch":
        sizes, F = _batch_sizes(case), case["frames"]
        model, enc = _model_k(case), BatchEncoder(sizes, 8, THR, INTERVAL)
        if model:
            enc.set_model(model, case["k"])
        frames = [_video(w, h, F, seed * 64 + i, case["squares"]) for i, (w, h) in enumerate(sizes)]
        outs = list(zip(*[_outputs(enc.nblk(i), F) for i in range(len(sizes))]))
        return dict(kind=kind, enc=enc, model=model, frames=frames, outs=outs,
                    flags=[intra_schedule(F, INTERVAL)] * len(sizes))
    w, h = case["w"], case["h"]
    if kind == "endpoints":
        n, F = (w // 4) * (h // 4), case["frames"]
        enc = Encoder(w, h, 8, THR, INTERVAL)
        final = torch.stack([o[0] for o in _encoded(enc, _video(w, h, F, seed, 1), intra_schedule(F, INTERVAL))])
        enc.close()
        return dict(kind=kind, w=w, h=h, final=final, out=torch.zeros((F, 6 * n), dtype=torch.uint8, device="cuda"))
    enc = Encoder(w, h, case.get("sa", 8), THR, INTERVAL)
    if kind == "frame":
        frames = _video(w, h, 2, seed, case["squares"])
        prev = None if case["intra"] else _encoded(enc, frames[:1], [True])[0][0]
        return dict(kind=kind, enc=enc, rgb=frames[1], prev=prev, outs=_outputs(enc.nblk))
    F = case["frames"]
    frames = _video(w, h, F, seed, case["squares"], case.get("cut", 0))
    flags = intra_schedule(F, INTERVAL)
    if kind == "decode":
        outs = _encoded(enc, frames, flags)
        enc.close()
        parts = []
        for final, motion, unique, n_unique, _ in outs:
            coeff = torch.empty(6 * final.numel(), dtype=torch.uint8, device="cuda")
            endpoint_coefficients(w, h, final, coeff)
            parts.append((motion, coeff, unique[: int(n_unique)].clone()))
        return dict(kind=kind, dec=Decoder(w, h, 8), parts=parts,
                    out=torch.zeros((F, outs[0][0].numel()), dtype=torch.int64, device="cuda"))
    if kind == "host":
        pin = (lambda t: t.pin_memory()) if case["pinned"] else (lambda t: t)
        host = lambda shape, t, as_: pin(torch.zeros(shape, dtype=t)).numpy().view(as_)  # noqa: E731
        n = enc.nblk
        out = StreamOutput(host((F, n), torch.int64, np.uint64), host((F, 2 * n), torch.uint8, np.uint8),
                           host((F, n), torch.int32, np.uint32), host((F,), torch.int32, np.uint32))
        return dict(kind=kind, enc=enc, frames=pin(frames.cpu()).numpy(), flags=flags, out=out,
                    palettes=np.zeros((F, n), np.uint32))
    model = _model_k(case)
    if model:
        enc.set_model(model, case["k"])
    return dict(kind=kind, enc=enc, model=model, frames=frames, flags=flags, outs=_outputs(enc.nblk, F))


def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["enc"].encode_frame_device(s["rgb"], s["prev"], None, *s["outs"])
        return s["outs"]
    if kind == "stream":
        s["enc"].encode_stream_device(s["frames"], *s["outs"], is_intra=s["flags"])
        return s["outs"]
    if kind == "host":
        o = s["enc"].encode_stream_host(s["frames"], s["flags"], s["out"])
        for k, keep in enumerate(s["palettes"]):  # entries past a palette's length are not outputs
            palette = o.frame(k).unique
            keep[: len(palette)] = palette
        return o.final, o.motion, o.n_unique, s["palettes"]
    if kind == "batch":
        s["enc"].encode_run(s["frames"], *s["outs"], s["flags"])
        return s["outs"]
    if kind == "endpoints":
        for final, coeff in zip(s["final"], s["out"]):
            endpoint_coefficients(s["w"], s["h"], final, coeff)
        return s["out"]
    if kind == "decode":
        for part, out in zip(s["parts"], s["out"]):
            out.copy_(s["dec"].decode_frame(*part))
        s["dec"].check()
        return s["out"]
    loss, grads = s["model"].grads(*s["args"])
    return loss, grads


def work(case):
    """Bytes: every frame and previous frame's blocks in, every output out.
    Operations: about 1,500 a block for its DXT1 encode and, for each of the
    some 33 distinct index words of its window, 200 for the refit and error."""
    kind = case["kind"]
    if kind == "train":
        mac = case["B"] * sum(i * n for i, n in LAYERS[:3]) + case["B"] * case["C"] * sum(i * n for i, n in LAYERS[3:])
        return {"bytes": case["B"] * (48 + 8 + 4 + 4 * case["C"]) + 8 * sum(i * n + n for i, n in LAYERS),
                "flops": 6 * mac}
    if kind == "batch":
        n = sum((w // 4) * (h // 4) for w, h in _batch_sizes(case)) * case["frames"]
    else:
        n = (case["w"] // 4) * (case["h"] // 4) * case.get("frames", 1)
    if kind == "endpoints":
        return {"bytes": 14 * n, "flops": 6 * 2 * 8 * n}
    if kind == "decode":
        return {"bytes": 16 * n, "flops": 6 * 2 * 8 * n}
    return {"bytes": (48 + 8 + 8 + 2) * n, "flops": (1500 + 33 * 200) * n}


def exact(case, seed):
    if case["kind"] != "train":
        return None  # whole numbers throughout
    rgb, w, stb, blocks, cands = _train_inputs(case, seed)
    flat = torch.from_numpy(_he(seed + 1)).cuda().double().requires_grad_(True)
    x = _features(rgb, stb, blocks.long(), w // 4, torch.float64)
    loss = _loss(_split(flat), x, _bits(cands, torch.float64))
    loss.backward()
    return loss.item(), flat.grad.cpu().numpy()
