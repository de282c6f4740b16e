"""The fused last level of one- to four-component images around the edges of its
tiles, of one image and of a batch (kernels of their own): lossless images come
back as they were, lossy ones within 1 of the oracle's FP64 decode."""
import numpy as np
import pytest

from conftest import synth_image
from gpu_helpers import oracle_decode_tiled
from thousandthchicken_b200 import codec

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("w,h", [(512, 240), (388, 179), (386, 128), (257, 121)])
@pytest.mark.parametrize("comps", [1, 2, 3, 4])
@pytest.mark.parametrize("reversible", [True, False])
def test_last_level_tiles(gpu_ctx, reversible, comps, w, h, batch):
    from thousandthchicken_b200.stages import Plan
    imgs = [synth_image(w, h, comps, 8, seed=comps + k) for k in range(batch)]
    streams = [codec.encode(i, 8, levels=3, reversible=reversible, mct=comps >= 3) for i in imgs]
    plan = Plan(gpu_ctx, streams)
    outs = plan.alloc_outputs()
    plan.execute(outs)
    gpu_ctx.synchronize()
    for img, cs, out in zip(imgs, streams, outs):
        got = out.cpu().numpy().astype(np.int64)
        if reversible:
            np.testing.assert_array_equal(got, img)
        else:
            diff = np.abs(got - oracle_decode_tiled(cs)[1].astype(np.int64))
            assert diff.max() <= 1 and (diff > 0).mean() < 0.01
