"""Forward and reverse transforms at sizes around the edges of their tiles
(120- and 128-column tiles of 56 and 60 rows) and with planes whose rows or
address are and are not 8-byte aligned (the reverse levels stage aligned
interior tiles with wider loads): 5/3 bit-exact, 9/7 within the fp32 tolerance
of test_gpu_dwt.py."""
import numpy as np
import pytest

import oracle as O
from test_gpu_dwt import TOL97

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# width, height, levels, extra pitch, element offset of the plane
CASES = [(520, 200, 2, 0, 0), (520, 200, 2, 1, 0), (520, 200, 2, 2, 1), (516, 190, 1, 0, 0), (518, 121, 1, 0, 0),
         (390, 185, 2, 0, 0), (386, 180, 1, 2, 0), (385, 181, 3, 1, 1), (1024, 192, 1, 0, 0)]


def _place(a, pitch_extra, offset, dt):
    h, w = a.shape
    buf = torch.zeros(offset + h * (w + pitch_extra), dtype=dt, device="cuda")
    view = buf[offset:].view(h, w + pitch_extra)
    view[:, :w] = torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype=dt)
    return view


@pytest.mark.parametrize("w,h,levels,extra,offset", CASES)
def test_tile_edges_and_alignment(gpu_ctx, w, h, levels, extra, offset):
    from thousandthchicken_b200.stages import DWTForward53, DWTForward97, DWTReverse53, DWTReverse97
    rng = np.random.default_rng(w * 7 + h + offset)
    x = rng.integers(-128, 128, (h, w)).astype(np.int32)
    for rev, fwd_cls, inv_cls, dt in ((True, DWTForward53, DWTReverse53, torch.int32),
                                      (False, DWTForward97, DWTReverse97, torch.float32)):
        coef = O.fdwt53(x, levels, 0) if rev else O.fdwt97(x.astype(np.float64), levels)
        for cls, src, want in ((fwd_cls, x, coef), (inv_cls, coef, x)):
            d = _place(src, extra, offset, dt)
            out = torch.zeros_like(d)
            cls(gpu_ctx).run(d, out, w, h, levels, in_pitch=w + extra, out_pitch=w + extra)
            got = out.cpu().numpy()[:, :w]
            if rev:
                np.testing.assert_array_equal(got, want)
            else:
                err = np.abs(got.astype(np.float64) - want).max()
                assert err <= TOL97 * max(1.0, np.abs(want).max() / 256.0), err
