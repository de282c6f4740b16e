"""The one-warp-per-block Tier-1 decoder at the edges of its bitmaps (widths
around words of eight columns, heights around stripes of four rows, one-column
and one-row blocks) and of its bit-planes (1 to 31), in launches of few blocks
and of many (each runs a kernel of its own), against the CPU oracle: bit-exact."""
import numpy as np
import pytest

from gpu_helpers import SLOT, oracle_slots
from thousandthchicken_b200 import codec
from thousandthchicken_b200.synth import laplacian_block

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(1, 1), (1, 64), (64, 1), (2, 3), (7, 4), (8, 5), (9, 8), (31, 6), (32, 32), (33, 9), (63, 64), (64, 63),
         (64, 64)]


def _blocks(planes):
    rng = np.random.default_rng(100 + planes)
    desc = np.zeros(2 * len(SIZES), codec.DESC_DTYPE)
    segs, off = [], 0
    for i, (w, h) in enumerate(SIZES + SIZES):
        coef = laplacian_block(rng, w, h, planes, zero_frac=0.3)
        coef[h // 2, w // 2] = (1 << planes) - 1     # the block has all its planes
        orient = i % 4
        seg, total, zbp = codec.t1_encode_block(coef, orient, 31)
        passes = total if i < len(SIZES) else int(rng.integers(1, total + 1))
        if passes < total:
            seg, passes, zbp = codec.t1_encode_block(coef, orient, 31, passes)
        desc[i] = (off, i * SLOT, len(seg), 64, 1.0, w, h, passes, 31, zbp, orient, 0, 0, 0, (0,))
        segs.append(seg)
        off += len(seg)
    return desc, np.frombuffer(b"".join(segs) + b"\0" * 16, np.uint8).copy()


@pytest.mark.parametrize("copies", [1, 40])
@pytest.mark.parametrize("planes", [1, 2, 8, 9, 16, 17, 31])
def test_t1_warp_decoder_edges(gpu_ctx, planes, copies):
    from thousandthchicken_b200.stages import CoefficientCoder
    desc, pool = _blocks(planes)
    want = oracle_slots(desc, pool, "int", 0.0)
    many = np.tile(desc, copies)
    many["out_off"] = np.arange(len(many), dtype=np.uint64) * np.uint64(SLOT)
    got = CoefficientCoder(gpu_ctx).decode_blocks(many, pool, len(many) * SLOT, recon_r=0.0).cpu().numpy()
    np.testing.assert_array_equal(got.reshape(copies, *want.shape), np.broadcast_to(want, (copies, *want.shape)))
