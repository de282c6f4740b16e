"""What is measured: the calls that a user of this decoder makes, from a
thumbnail to a 4096 x 4096 image, a mixed batch and a large set of
code-blocks, and the stages that other programs call on their own (wavelet,
colour, encoder).

A case names a kind and its sizes:

  call    Decoder.decode: a codestream in pinned host memory in, samples in
          pinned host memory out (a viewer, a transcoder, one image at a time)
  plan    Plan.execute: codestreams already on the device (a batch that was
          parsed and uploaded while another one decoded), samples on the device
  batch   Plan.execute of images of mixed sizes, depths and coding
  blocks  code-blocks of many images in one Tier-1 call (int32 coefficients)
  dwt     one component through the forward or reverse 5/3 or 9/7 transform
  color   inverse or forward component transform of three planes
  encode  codec.encode_gpu: host samples in, codestream out

Images are the benchmark family (gradients plus Gaussian noise, seeded), coded
by the host encoder with the parameters that a file would have.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from thousandthchicken_b200 import codec
from thousandthchicken_b200._lib import TC_ROUND_FLOOR
from thousandthchicken_b200.blockbatch import BlockBatch
from thousandthchicken_b200.stages import (Context, Decoder, DWTForward53, DWTForward97, DWTReverse53, DWTReverse97,
                                           Plan, Preprocessor)
from thousandthchicken_b200.synth import c3_coefficients, c3_geometry, gradient_noise_image_device

DEV = "cuda:0"
_ctx = None


def context() -> Context:
    """The program's one context."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


def listed():
    return [
        # a preview of a catalogue page: the smallest call, all latency
        dict(name="call_thumb_160x96", kind="call", w=160, h=96, c=3, bits=8, rev=False, levels=4, step=1 / 128,
             style=0),
        # a video frame or a photo, one call at a time, host to host
        dict(name="call_hd_1920x1080", kind="call", w=1920, h=1080, c=3, bits=8, rev=False, levels=5, step=1 / 64,
             style=0),
        # a 16-bit single-component lossless image (medical, scientific): deep code-blocks
        dict(name="call_gray16_2048", kind="call", w=2048, h=2048, c=1, bits=16, rev=True, levels=5, step=0.0,
             style=0),
        # the benchmark image: 4096 x 4096 colour, lossy, near-lossless step
        dict(name="plan_lossy_4096", kind="plan", w=4096, h=4096, c=3, bits=8, rev=False, levels=6, step=1 / 128,
             style=0),
        # 12-bit lossless colour of an odd size (cinema masters, archives)
        dict(name="plan_lossless12_3001x2047", kind="plan", w=3001, h=2047, c=3, bits=12, rev=True, levels=5, step=0.0,
             style=0),
        # a stream with selective arithmetic-coding bypass, as fast encoders write it
        dict(name="plan_bypass_1536x1100", kind="plan", w=1536, h=1100, c=3, bits=8, rev=True, levels=5, step=0.0,
             style=codec.CBLK_STYLE_BYPASS),
        # one batch of a decode server: sizes, depths and coding mixed
        dict(name="batch_mixed_12", kind="batch", n=12, lo=128, hi=1600, pick=11),
        # code-blocks of many images: the batched Tier-1 workload, truncated codewords
        dict(name="blocks_24000", kind="blocks", n=24000),
        # the transform alone, as a program with its own Tier-1 calls it
        dict(name="dwt_reverse97_4096", kind="dwt", w=4096, h=4096, rev=False, inverse=True, levels=6),
        dict(name="dwt_forward53_2999x2001", kind="dwt", w=2999, h=2001, rev=True, inverse=False, levels=5),
        # colour alone: a 4K frame back to 8-bit RGB
        dict(name="color_ict_inverse_3840x2160", kind="color", w=3840, h=2160, bits=8, rev=False, inverse=True),
        # the encoder, host to host
        dict(name="encode_lossy_2048", kind="encode", w=2048, h=2048, c=3, bits=8, rev=False, levels=5, step=1 / 64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "plan", "plan", "plan", "batch", "blocks", "dwt", "dwt", "color", "encode"])
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(2, 16), lo=64, hi=_log(rng, 256, 1600), pick=rng.randint(1, 10 ** 6))
    if kind == "blocks":
        return dict(kind=kind, n=_log(rng, 64, 24000))
    rev = rng.random() < 0.5
    if kind == "dwt":
        return dict(kind=kind, w=_log(rng, 33, 4096), h=_log(rng, 33, 4096), rev=rev, inverse=rng.random() < 0.6,
                    levels=rng.randint(1, 6))
    if kind == "color":
        return dict(kind=kind, w=_log(rng, 64, 4096), h=_log(rng, 64, 2100), bits=rng.choice([8, 8, 12]), rev=rev,
                    inverse=rng.random() < 0.7)
    big = 2048 if kind == "encode" else 3000
    case = dict(kind=kind, w=_log(rng, 48, big), h=_log(rng, 48, big), c=rng.choice([1, 3, 3]),
                bits=rng.choice([8, 8, 12, 16]), rev=rev, levels=rng.randint(3, 6),
                step=0.0 if rev else 1 / rng.choice([32, 64, 128]))
    if case["bits"] == 16:
        case.update(c=1, rev=True, step=0.0)
    if kind != "encode":
        case["style"] = rng.choice([0, 0, 0, 0, codec.CBLK_STYLE_BYPASS, codec.CBLK_STYLE_TERMALL])
    return case


def _image(w, h, c, bits, seed):
    sigma = 8.0 if bits <= 12 else 0.25   # 16-bit: about 40 of 65,535
    img = gradient_noise_image_device(w, h, c, bits if bits < 16 else 15, seed, DEV, sigma).cpu().numpy()
    return img if bits <= 8 else img.view(np.uint16)


def _stream(case, seed):
    img = _image(case["w"], case["h"], case["c"], case["bits"], seed)
    return codec.encode(img, case["bits"], levels=case["levels"], reversible=case["rev"], mct=case["c"] == 3,
                        base_step=case["step"] or 1 / 128, cblk_style=case["style"])


def _batch(case):
    """The images of a batch: sides over lo..hi, half of them lossless."""
    r = np.random.default_rng(case["pick"])
    out = []
    for i in range(case["n"]):
        w, h = (int(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(2))
        rev = bool(i % 2 == 0)
        out.append(dict(w=w, h=h, c=int(r.choice([1, 3])), bits=int(r.choice([8, 12])), rev=rev, levels=5,
                        step=0.0 if rev else 1 / 64, style=0))
    return out


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _dwt_input(case, seed):
    """Samples (forward) or subband coefficients (reverse) of one component."""
    v = torch.randn((case["h"], case["w"]), generator=_gen(seed), device=DEV) * 40.0
    return torch.round(v).to(torch.int32) if case["rev"] else v


def _color_input(case, seed):
    shape, top = (case["h"], case["w"]), (1 << case["bits"]) - 1
    g = _gen(seed)
    planes = []
    for k in range(3):
        v = torch.rand(shape, generator=g, device=DEV)
        if case["inverse"]:
            # luminance and two smaller chrominance planes around zero
            v = (v - 0.5) * (top if k == 0 else 0.4 * top)
            planes.append(torch.round(v).to(torch.int32) if case["rev"] else v)
        else:
            planes.append(torch.round(v * top).to(torch.uint8 if case["bits"] <= 8 else torch.int16))
    return planes


def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    if kind == "call":
        cs = np.frombuffer(_stream(case, seed), np.uint8)
        src = _pinned(cs.size, torch.uint8)
        src.numpy()[:] = cs
        out = _pinned((case["c"], case["h"], case["w"]), torch.uint8 if case["bits"] <= 8 else torch.int16)
        return dict(kind=kind, dec=Decoder(ctx), src=src, out=out)
    if kind in ("plan", "batch"):
        images = [case] if kind == "plan" else _batch(case)
        plan = Plan(ctx, [_stream(im, seed * 1000 + i) for i, im in enumerate(images)])
        return dict(kind=kind, plan=plan, outs=plan.alloc_outputs())
    if kind == "blocks":
        geom = c3_geometry(case["n"])   # sizes and pass counts; the seed gives the coefficients
        bb = BlockBatch(ctx, geom, c3_coefficients(geom, DEV, seed=seed + 3))
        return dict(kind=kind, blocks=bb)
    if kind == "dwt":
        cls = {(True, True): DWTReverse53, (True, False): DWTForward53, (False, True): DWTReverse97,
               (False, False): DWTForward97}[case["rev"], case["inverse"]]
        x = _dwt_input(case, seed)
        return dict(kind=kind, stage=cls(ctx, TC_ROUND_FLOOR), x=x, out=torch.empty_like(x), case=case)
    if kind == "color":
        planes = _color_input(case, seed)
        if case["inverse"]:
            dt = torch.uint8 if case["bits"] <= 8 else torch.int16
        else:
            dt = torch.int32 if case["rev"] else torch.float32
        pre = Preprocessor(ctx)
        fn = {(True, True): pre.color_decoder_lossless, (False, True): pre.color_decoder_lossy,
              (True, False): pre.color_coder_lossless, (False, False): pre.color_coder_lossy}[case["rev"],
                                                                                             case["inverse"]]
        return dict(kind=kind, fn=fn, planes=planes, out=[torch.empty_like(p, dtype=dt) for p in planes],
                    bits=case["bits"])
    return dict(kind=kind, ctx=ctx, img=_image(case["w"], case["h"], case["c"], case["bits"], seed), case=case)


def run(state):
    kind = state["kind"]
    if kind == "call":
        # 16-bit samples: the same bytes, as the uint16 that the decoder writes
        out = state["out"].numpy()
        state["dec"].decode(state["src"].numpy(), out)
        return out
    if kind in ("plan", "batch"):
        return state["plan"].execute(state["outs"])
    if kind == "blocks":
        state["blocks"].decode_batched()
        return state["blocks"].out
    if kind == "dwt":
        case = state["case"]
        return state["stage"].run(state["x"], state["out"], case["w"], case["h"], case["levels"])
    if kind == "color":
        return state["fn"](state["planes"], state["out"], state["bits"])
    case = state["case"]
    cs = codec.encode_gpu(state["ctx"], state["img"], case["bits"], levels=case["levels"], reversible=case["rev"],
                          mct=case["c"] == 3, base_step=case["step"] or 1 / 128)
    # the codestream and its length, in a buffer of the size that a caller sets aside
    out = np.zeros(2 * state["img"].nbytes + 4096, np.uint8)
    out[:len(cs)] = np.frombuffer(cs, np.uint8)
    return [out, len(cs)]


def _coded_bits(case):
    """Codeword bits per sample, about: the noise (sigma 8 of 255) sets them."""
    noise = 8.0 * ((1 << case["bits"]) - 1) / 255.0 if case["bits"] <= 12 else 40.0
    if case["rev"]:
        return math.log2(noise * 4.13)
    # quantised with the base step (a fraction of the nominal range); 3.35 bits at 1/128
    return max(0.3, math.log2(8.0 / 255.0 * 4.13 / case["step"]) - 0.7)


def work(case):
    kind = case["kind"]
    if kind == "dwt":
        n = case["w"] * case["h"]
        # 8 (9/7) or 4 (5/3) operations a sample and direction; the levels add a third
        return dict(bytes=8 * n, flops=n * (16 if not case["rev"] else 8) * 4 / 3)
    if kind == "color":
        n = 3 * case["w"] * case["h"]
        return dict(bytes=n * (4 + (1 if case["bits"] <= 8 else 2)), flops=4 * n)
    if kind == "blocks":
        # 60% of 4096 samples, 30% of 1024, 10% about 1056; half of about 9 planes coded
        n = case["n"] * 2870
        return dict(bytes=n * (4 + 0.4), flops=n * 5 * 10)
    images = _batch(case) if kind == "batch" else [case]
    nbytes = flops = 0.0
    for im in images:
        n = im["w"] * im["h"] * im["c"]
        bits = _coded_bits(im)
        nbytes += n * (bits / 8 + (1 if im["bits"] <= 8 else 2))
        # about 1.1 binary decisions a coded bit, ten operations each, and the transform
        flops += n * (11 * bits + (8 if im["rev"] else 16) * 4 / 3 + 4)
    return dict(bytes=nbytes, flops=flops)


# 9/7 lifting constants and scaling (ISO/IEC 15444-1, Table F.4)
_LIFT = (-1.586134342059924, -0.052980118572961, 0.882911075530934, 0.443506852043971)
_K = 1.230174104914001


def _steps(x, steps):
    """Lifting steps (odd samples first) along the last axis of an
    interleaved signal, with whole-sample symmetric extension."""
    n = x.shape[-1]
    for parity, a in steps:
        t = x[..., parity::2]
        left = x[..., 1 - parity::2]
        if parity:   # odd sample 2i+1: neighbours 2i and 2i+2 (mirrored past the end)
            right = left[..., 1:]
            if n % 2 == 0:
                right = torch.cat([right, left[..., -1:]], -1)
            left = left[..., :t.shape[-1]]
        else:        # even sample 2i: neighbours 2i-1 (mirrored before the start) and 2i+1
            right = left
            left = torch.cat([left[..., :1], left], -1)[..., :t.shape[-1]]
            if n % 2:
                right = torch.cat([right, right[..., -1:]], -1)
        x[..., parity::2] = t + a * (left + right)
    return x


def _dwt97(x, levels, inverse):
    """9/7 of a float64 plane in Mallat layout."""
    x = x.clone()
    sizes = [x.shape]
    for _ in range(levels):
        h, w = sizes[-1]
        sizes.append(((h + 1) // 2, (w + 1) // 2))

    def analyse(v):
        if v.shape[-1] == 1:
            return v
        v = _steps(v, ((1, _LIFT[0]), (0, _LIFT[1]), (1, _LIFT[2]), (0, _LIFT[3])))
        return torch.cat([v[..., 0::2] / _K, v[..., 1::2] * _K], -1)

    def synthesise(v):
        n = v.shape[-1]
        if n == 1:
            return v
        y = torch.empty_like(v)
        y[..., 0::2], y[..., 1::2] = v[..., :(n + 1) // 2] * _K, v[..., (n + 1) // 2:] / _K
        return _steps(y, ((0, -_LIFT[3]), (1, -_LIFT[2]), (0, -_LIFT[1]), (1, -_LIFT[0])))

    for lvl in range(levels - 1, -1, -1) if inverse else range(levels):
        h, w = sizes[lvl]
        v = x[:h, :w].clone()
        if inverse:   # rows, then columns
            v = synthesise(v)
            v = synthesise(v.t().contiguous()).t()
        else:         # columns, then rows
            v = analyse(v.t().contiguous()).t().contiguous()
            v = analyse(v)
        x[:h, :w] = v
    return x


def exact(case, seed):
    """The transforms of floating-point values in 64 bits; the other cases
    return whole numbers."""
    if case["kind"] == "dwt" and not case["rev"]:
        return _dwt97(_dwt_input(case, seed).double(), case["levels"], case["inverse"])
    if case["kind"] == "color" and not case["rev"] and not case["inverse"]:
        r, g, b = (p.double() - (1 << (case["bits"] - 1)) for p in _color_input(case, seed))
        y = 0.299 * r + 0.587 * g + 0.114 * b
        return [y, 0.5 * (b - y) / (1 - 0.114), 0.5 * (r - y) / (1 - 0.299)]
    return None
