"""Tier-1 launches of more blocks than fit the GPU at once, with blocks of more
bit-planes than a block's state then has room for: the oracle's samples, whatever
the output held before, and nothing written outside the blocks."""
import numpy as np
import pytest

import oracle as O
from gpu_helpers import SLOT
from thousandthchicken_b200 import codec
from thousandthchicken_b200.synth import laplacian_block

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(64, 64), (33, 30), (5, 64), (64, 3), (1, 1), (40, 17)]


@pytest.mark.parametrize("mode", ["int", "float", "raw"])
@pytest.mark.parametrize("styled", [False, True])
@pytest.mark.parametrize("deep,bound", [(9, 9), (13, 13), (16, 0), (17, 17), (24, 0), (31, 31)])
def test_deep_blocks_of_a_full_launch(gpu_ctx, deep, bound, styled, mode):
    from thousandthchicken_b200.stages import CoefficientCoder, _dev_bytes
    rng = np.random.default_rng(deep)
    kinds, segs, off = np.zeros(4 * len(SIZES), codec.DESC_DTYPE), [], 0
    want = np.full((len(kinds), 64, 64), 0x5A5A5A5A, np.uint32)
    for i in range(len(kinds)):
        w, h = SIZES[i % len(SIZES)]
        planes = deep if i < 2 * len(SIZES) else 4
        coef = laplacian_block(rng, w, h, planes, zero_frac=0.3)
        coef[h // 2, w // 2] = (1 << planes) - 1
        seg, passes, zbp = codec.t1_encode_block(coef, i % 4, 31)
        if i % 3 == 0:
            seg, passes, zbp = codec.t1_encode_block(coef, i % 4, 31, int(rng.integers(1, passes + 1)))
        kinds[i] = (off, 0, len(seg), 64, 0.25, w, h, passes, 31, zbp, i % 4, int(mode == "float"), 0, 0, (0,))
        segs.append(seg)
        off += len(seg)
        if mode == "raw":
            want[i, :h, :w] = O.t1_decode_raw(seg, w, h, i % 4, 31, zbp, passes)
        else:
            q, u = O.t1_decode(seg, w, h, i % 4, 31 - zbp, passes)
            v = O.dequant_float(q, u, 0.5, 0.25) if mode == "float" else O.dequant_int(q, u, 0.0)
            want[i, :h, :w] = np.ascontiguousarray(v).view(np.uint32)
    pool = np.frombuffer(b"".join(segs) + b"\0" * 16, np.uint8).copy()
    copies = 25 * torch.cuda.get_device_properties(gpu_ctx.device).multi_processor_count // len(kinds) + 1
    desc = np.tile(kinds, copies)
    desc["out_off"] = np.arange(len(desc), dtype=np.uint64) * np.uint64(SLOT)
    dev = torch.device("cuda", gpu_ctx.device)
    out = torch.full((len(desc) * SLOT,), 0x5A5A5A5A, dtype=torch.int32, device=dev)
    CoefficientCoder(gpu_ctx).decode(_dev_bytes(desc, dev), _dev_bytes(pool, dev), out, len(desc),
                                     _dev_bytes(codec.sort_order(desc), dev), mode == "raw",
                                     0.5 if mode == "float" else 0.0, bound, styled)
    gpu_ctx.synchronize()
    got = out.cpu().numpy().view(np.uint32).reshape(copies, len(kinds), 64, 64)
    want = np.ascontiguousarray(np.broadcast_to(want, got.shape))
    if mode == "float":   # the magnitude, its sum with r and the oracle's result each round once, by 2^-24 at most
        np.testing.assert_allclose(got.view(np.float32), want.view(np.float32), rtol=3 * 2.0 ** -24, atol=0)
    else:
        np.testing.assert_array_equal(got, want)
