"""Raw (bypass) refinement passes, alone and with termination on every pass,
at the edges of the decoder's words and stripes: lossless round trips of
images whose code-blocks have 10 and more coding passes, bit-exact."""
import numpy as np
import pytest

from thousandthchicken_b200 import codec

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("style", [codec.CBLK_STYLE_BYPASS, codec.CBLK_STYLE_BYPASS | codec.CBLK_STYLE_TERMALL])
@pytest.mark.parametrize("w,h", [(1, 9), (9, 1), (33, 30), (64, 64), (71, 67), (129, 62)])
def test_raw_refinement_edges(gpu_ctx, w, h, style):
    from thousandthchicken_b200.stages import Decoder
    img = np.random.default_rng(w * 100 + h).integers(0, 1 << 12, (1, h, w)).astype(np.uint16)
    cs = codec.encode(img, 12, levels=1, reversible=True, mct=False, cblk_style=style)
    np.testing.assert_array_equal(Decoder(gpu_ctx).decode(cs), img)
