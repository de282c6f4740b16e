"""The GPU Tier-1 encoder at the edges of its column lanes (widths around 32),
stripes (heights around multiples of four) and bit-planes, whole and truncated
codewords: the same bytes as the host encoder."""
import numpy as np
import pytest

from thousandthchicken_b200 import codec
from thousandthchicken_b200.synth import laplacian_block

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(1, 1), (1, 64), (64, 1), (3, 4), (31, 5), (32, 8), (33, 7), (63, 64), (64, 62), (64, 64)]


@pytest.mark.parametrize("planes,zero_frac", [(1, 0.0), (1, 0.97), (4, 0.6), (9, 0.15), (17, 0.9), (30, 0.3)])
def test_gpu_tier1_encoder_edges(gpu_ctx, planes, zero_frac):
    from thousandthchicken_b200.stages import T1Encoder
    rng = np.random.default_rng(planes * 7 + int(10 * zero_frac))
    jobs = [(w, h, o, tr) for w, h in SIZES for o in range(4) for tr in (False, True)]
    desc = np.zeros(len(jobs), codec.ENC_DESC_DTYPE)
    planes_in = np.zeros((len(jobs), 64, 64), np.int32)
    want = []
    for i, (w, h, o, truncate) in enumerate(jobs):
        coef = laplacian_block(rng, w, h, planes, zero_frac)
        planes_in[i, :h, :w] = coef
        total = codec.t1_encode_block(coef, o, 31)[1]
        limit = int(rng.integers(1, total + 1)) if truncate and total > 1 else 0
        desc[i] = (i * 4096, 64, 1.0, w, h, o, 31, 0, limit)
        want.append(codec.t1_encode_block(coef, o, 31, limit))
    got = T1Encoder(gpu_ctx).encode(desc, torch.from_numpy(planes_in).cuda(), cap=5 * 4096 + 256)
    for i, (g, e) in enumerate(zip(got, want)):
        assert g == e, f"block {i} {jobs[i]}"
