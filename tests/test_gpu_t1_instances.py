"""Both instances of the one-warp-per-block Tier-1 decoder (for few blocks and
for launches that fill the GPU) at the edges of its bitmaps and bit-planes,
against the CPU oracle: bit-exact.  The launches lie on either side of the
border that the dispatch draws, read from its source."""
import re

import numpy as np
import pytest

from conftest import ROOT
from gpu_helpers import SLOT, oracle_slots
from test_gpu_t1_warp import _blocks

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _border():
    text = (ROOT / "thousandthchicken_b200" / "csrc" / "t1_decode_warp.cu").read_text()
    assert "return n < kDeepBlocks * num_sms(ctx->device);" in text
    return int(re.search(r"kDeepBlocks = (\d+);", text).group(1)) * \
        torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("instance,blocks", [("few", -1), ("full", 0), ("full", 2000)])
@pytest.mark.parametrize("planes", [1, 2, 8, 9, 16, 17, 31])
def test_instances_at_the_edges(gpu_ctx, planes, instance, blocks):
    from thousandthchicken_b200.stages import CoefficientCoder
    n = _border() + blocks
    assert (n < _border()) == (instance == "few")
    desc, pool = _blocks(planes)
    want = oracle_slots(desc, pool, "int", 0.0)
    which = np.arange(n) % len(desc)
    many = desc[which]
    many["out_off"] = np.arange(n, dtype=np.uint64) * np.uint64(SLOT)
    got = CoefficientCoder(gpu_ctx).decode_blocks(many, pool, n * SLOT, recon_r=0.0).cpu().numpy()
    np.testing.assert_array_equal(got.reshape(n, 64, 64), want[which])
