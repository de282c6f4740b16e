"""Tier-1 blocks of mixed depth with 8, 16 and 32 lanes per block.  With 32, one
launch takes the three depth classes in turn, the deepest first; with lane groups
they are launches of their own, of which a small 8-bit class joins the 16-bit one,
and deep blocks keep their magnitudes in their output words."""
import numpy as np
import pytest

from conftest import synth_image
from gpu_helpers import SLOT, oracle_slots
from test_gpu_t1_warp import _blocks
from thousandthchicken_b200 import codec

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(params=[8, 16, 32])
def lanes(gpu_ctx, request):
    from thousandthchicken_b200 import _lib as L
    assert L.lib().tc_ctx_set_t1_group(gpu_ctx.handle, request.param) == 0
    yield request.param
    L.lib().tc_ctx_set_t1_group(gpu_ctx.handle, 32)


@pytest.mark.parametrize("planes", [9, 16, 23])
def test_repeated_deep_launches_are_identical(gpu_ctx, lanes, planes):
    """A deep class that fills the GPU gives the oracle's samples on every run,
    from any starting contents of the output."""
    from thousandthchicken_b200.stages import CoefficientCoder, _dev_bytes
    desc, pool = _blocks(planes)
    want = oracle_slots(desc, pool, "int", 0.0)
    n = 26 * torch.cuda.get_device_properties(gpu_ctx.device).multi_processor_count
    which = np.arange(n) % len(desc)
    many = desc[which]
    many["out_off"] = np.arange(n, dtype=np.uint64) * np.uint64(SLOT)
    inside = np.zeros(want.shape, bool)
    for i, d in enumerate(desc):
        inside[i, :d["h"], :d["w"]] = True
    dev = torch.device("cuda", gpu_ctx.device)
    d_desc, d_pool, d_order = (_dev_bytes(a, dev) for a in (many, pool, codec.sort_order(many)))
    out = torch.empty(n * SLOT, dtype=torch.int32, device=dev)
    for fill in (0, -1, 0x5A5A5A5A):
        out.fill_(fill)
        CoefficientCoder(gpu_ctx).decode(d_desc, d_pool, out, n, d_order, False, 0.0, planes)
        gpu_ctx.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy().reshape(n, 64, 64), np.where(inside, want, fill)[which])


@pytest.mark.parametrize("bits", [[8, 12, 16], [12], [12, 12, 16], [8, 8, 8, 12], [16, 8]])
def test_depth_classes_of_a_plan(gpu_ctx, lanes, bits):
    """Lossless images of several sample depths, one of them with a coding style,
    in one plan: every image comes back as it was."""
    from thousandthchicken_b200.stages import Plan
    imgs = [synth_image(700 - 40 * k, 500, 3, b, seed=21 + k) for k, b in enumerate(bits)]
    streams = [codec.encode(i, b, levels=5, reversible=True, mct=True, cblk_style=0x01 if k == 1 else 0)
               for k, (i, b) in enumerate(zip(imgs, bits))]
    if bits == [12]:   # the 8-bit class joins the 16-bit one
        _, desc, _ = codec.parse(streams[0])
        nb = desc["mb"].astype(int) - desc["zero_bitplanes"].astype(int)
        assert 0 < 2 * int((nb <= 8).sum()) <= int(((nb > 8) & (nb <= 16)).sum())
    plan = Plan(gpu_ctx, streams)
    outs = plan.execute(plan.alloc_outputs())
    gpu_ctx.synchronize()
    for img, out in zip(imgs, outs):
        np.testing.assert_array_equal(out.cpu().numpy().view(img.dtype), img)
    plan.close()
