"""The Tier-1 kernels' results do not depend on how far a lane runs ahead of
the others between two synchronisation points (CUDA promises no lock-step
there): the device code, run on the CPU warp emulator with its lanes taken in
several orders, gives the oracle's samples and the host encoder's codewords,
and every lane reaches the same synchronisation points."""
import ctypes as C

import numpy as np
import pytest

import warp_emulator as W
from conftest import synth_image
from gpu_helpers import SLOT, oracle_mallat, oracle_slots
from thousandthchicken_b200 import codec
from thousandthchicken_b200.synth import laplacian_block

ORDERS = [0, 1, 2, 3]   # ascending, descending, two shuffles
SIZES = [(16, 12), (9, 7), (33, 5), (1, 6), (64, 8)]


def _blocks(planes, sizes=SIZES):
    rng = np.random.default_rng(planes)
    desc = np.zeros(len(sizes), codec.DESC_DTYPE)
    segs, off = [], 0
    for i, (w, h) in enumerate(sizes):
        coef = laplacian_block(rng, w, h, planes, zero_frac=0.3)
        coef[h // 2, w // 2] = (1 << planes) - 1
        seg, passes, zbp = codec.t1_encode_block(coef, i % 4, 31)
        if i % 2:
            seg, passes, zbp = codec.t1_encode_block(coef, i % 4, 31, int(rng.integers(1, passes + 1)))
        desc[i] = (off, i * SLOT, len(seg), 64, 1.0, w, h, passes, 31, zbp, i % 4, 0, 0, 0, (0,))
        segs.append(seg)
        off += len(seg)
    return desc, np.frombuffer(b"".join(segs) + b"\0" * 16, np.uint8).copy()


@pytest.fixture(scope="module")
def emulated(tmp_path_factory):
    built = {}

    def get(kind):
        if kind not in built:
            built[kind] = W.build(kind, tmp_path_factory.mktemp("emu"))
        return built[kind]
    return get


def _p(a):
    return C.c_void_p(a.ctypes.data)


def _decode(call, desc, pool, elems):
    """call(descriptors, n, pool, its length, out, its length, mode, r, error word) -> samples"""
    out, err = np.zeros(elems, np.int32), C.c_uint32(0)
    rc = call(_p(desc), len(desc), _p(pool), C.c_uint64(len(pool)), _p(out), C.c_uint64(elems), 0, C.c_float(0.0),
              C.byref(err))
    assert (rc, err.value) == (0, 0)
    return out


def _warp(emulated, kernel, planes, order, room=None):
    """room: the bit-planes that a block's state holds (default: all)."""
    def call(*a):
        return emulated("EMU_WARP").emu_decode(int(kernel == "styled"), int(kernel == "deep"), *a[:-1], room or planes,
                                               planes, order, a[-1])
    return call


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("planes", [1, 6, 12])
@pytest.mark.parametrize("kernel", ["lean", "deep", "styled"])
def test_warp_decoder(emulated, kernel, planes, order):
    desc, pool = _blocks(planes)
    got = _decode(_warp(emulated, kernel, planes, order), desc, pool, len(desc) * SLOT)
    np.testing.assert_array_equal(got.reshape(-1, 64, 64), oracle_slots(desc, pool, "int", 0.0))


@pytest.mark.parametrize("planes,room", [(9, 8), (12, 11), (16, 8), (23, 11), (31, 8)])
@pytest.mark.parametrize("kernel", ["lean", "deep", "styled"])
def test_warp_decoder_moves_planes_on(emulated, kernel, planes, room):
    """Blocks of more bit-planes than their state has room for, whole and cut
    after any number of them: the samples that the state alone would give."""
    desc, pool = _blocks(planes, SIZES[:4])
    got = _decode(_warp(emulated, kernel, planes, 2, room), desc, pool, len(desc) * SLOT)
    np.testing.assert_array_equal(got.reshape(-1, 64, 64), oracle_slots(desc, pool, "int", 0.0))


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("style", [0x01, 0x05, 0x0A, 0x26])
def test_warp_decoder_styles(emulated, style, order):
    """Bypass, context reset, termination, causal contexts and segmentation
    symbols: the same coefficients as the plain stream's."""
    img = synth_image(45, 34, 1, 8, seed=style)
    kw = dict(levels=2, cblk_log2=5, reversible=True)
    want, _ = oracle_mallat(codec.encode(img, 8, **kw))
    _, desc, pool = codec.parse(codec.encode(img, 8, cblk_style=style, **kw))
    got = _decode(_warp(emulated, "styled", 12, order), desc, pool, want.size)
    np.testing.assert_array_equal(got.reshape(want.shape), want)


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("planes", [1, 6, 12])
@pytest.mark.parametrize("lanes", [8, 16])
def test_group_decoder(emulated, lanes, planes, order):
    """Several blocks per warp: the groups' lanes part from one another, too."""
    desc, pool = _blocks(planes)

    def call(*a):
        return emulated("EMU_GROUPS").emu_decode_groups(lanes, int(planes > 8), *a[:-1], order, a[-1])
    got = _decode(call, desc, pool, len(desc) * SLOT)
    np.testing.assert_array_equal(got.reshape(-1, 64, 64), oracle_slots(desc, pool, "int", 0.0))


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("planes", [0, 1, 6, 12])
@pytest.mark.parametrize("irreversible", [False, True])
def test_encoder(emulated, irreversible, planes, order):
    """irreversible: float samples whose magnitudes are floored, zeros of either
    sign among them; planes 0: empty blocks."""
    rng = np.random.default_rng(planes)
    cap = 8192
    desc = np.zeros(4 * len(SIZES), codec.ENC_DESC_DTYPE)   # a CTA of four warps for each block
    coefs = np.zeros(len(SIZES) * SLOT, np.float32 if irreversible else np.int32)
    want = []
    for i, (w, h) in enumerate(SIZES):
        coef = laplacian_block(rng, w, h, planes, zero_frac=0.3) if planes else np.zeros((h, w), np.int32)
        limit = int(rng.integers(1, 3 * planes - 1)) if planes and i % 2 else 0
        desc[4 * i] = (i * SLOT, w, 1.0, w, h, i % 4, 31, int(irreversible), limit)
        fraction = np.where(coef == 0, rng.choice([-0.5, -0.0, 0.5], coef.shape), np.sign(coef) * 0.5) if irreversible else 0
        coefs[i * SLOT:i * SLOT + w * h] = (coef + fraction).ravel()
        want.append(codec.t1_encode_block(coef, i % 4, 31, limit))
    out, res = np.zeros(len(desc) * cap, np.uint8), np.zeros(len(desc), codec.ENC_RESULT_DTYPE)
    assert emulated("EMU_ENCODE").emu_encode(_p(desc), len(desc), _p(coefs), _p(out), C.c_uint32(cap), _p(res), order) == 0
    for i, (seg, passes, zbp) in enumerate(want):
        r = res[4 * i]
        assert (r["status"], r["passes"], r["zero_bitplanes"]) == (0, passes, zbp)
        assert out[4 * i * cap:4 * i * cap + int(r["len"])].tobytes() == seg
