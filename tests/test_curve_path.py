"""The curve decode (linear, sRGB, ST 2084 and HLG images): its divisions by
constants on the CPU, its planes against the oracle's on the GPU."""

import numpy as np
import pytest

from tests import helpers
from vqm_b200 import ss2

F, T, M = ss2.ImageFormat, ss2.TransferCharacteristics, ss2.MatrixCoefficients


@pytest.mark.parametrize("divisor", [1.055, 12.92, 0.17883277, 12.0])
def test_division_by_constants_is_correctly_rounded(divisor):
    """q = a r, q + r (a - b q) with one rounding each is a / b for every
    significand of a (all of two octaves)."""
    b = np.float32(divisor)
    r = np.float32(1.0) / b
    a = np.arange(0x3f000000, 0x40000000, dtype=np.uint32).view(np.float32)
    q = a * r
    rest = a.astype(np.float64) - np.float64(b) * q.astype(np.float64)  # exact
    assert np.array_equal(rest, rest.astype(np.float32))
    got = (q.astype(np.longdouble) + rest.astype(np.longdouble) * np.longdouble(r)).astype(np.float32)
    assert np.array_equal(got, a / b)


def _hdr(transfer, **kw):
    base = dict(type=ss2.PixelType.Word, depth=10, family=ss2.ColorFamily.Yuv,
                range=ss2.PixelRange.Limited, matrix=M.Bt2020Ncl, transfer=transfer,
                primaries=ss2.ColorPrimaries.Bt2020, subsample_w=1, subsample_h=1)
    base.update(kw)
    return F(**base)


FORMATS = {
    "pq420p10": _hdr(T.St2084),
    "pq420p10_center": _hdr(T.St2084, chroma_location=ss2.ChromaLocation.Center),
    "hlg422p10": _hdr(T.AribB67, subsample_h=0),
    "hlg420p8": _hdr(T.AribB67, type=ss2.PixelType.Byte, depth=0),
    # No primaries matrix behind the transfer: its last product is the linear
    # value that the box sums and the opsin mix read.
    "pq420p10_bt709": _hdr(T.St2084, primaries=ss2.ColorPrimaries.Bt709),
    "hlg420p10_bt709": _hdr(T.AribB67, primaries=ss2.ColorPrimaries.Bt709),
    "pq_grey16": F(type=ss2.PixelType.Word, family=ss2.ColorFamily.Grey, matrix=M.Bt709,
                   transfer=T.St2084),
    "pq444p12": _hdr(T.St2084, depth=12, subsample_w=0, subsample_h=0),
    "ictcp_pq420p10": _hdr(T.St2084, matrix=M.Bt2100ICtCp),
    "srgb_yuv420p8": _hdr(T.Srgb, type=ss2.PixelType.Byte, depth=0, matrix=M.Bt709,
                          primaries=ss2.ColorPrimaries.Bt709),
    # The BT.2020 matrix's inverse has entries of 2^-56 for 0, so the device
    # tests this image's values for tiny ones.
    "srgb_yuv420p16_bt2020": _hdr(T.Srgb, depth=0, range=ss2.PixelRange.Full),
    "rgb16": F(type=ss2.PixelType.Word),
    "rgb10": F(type=ss2.PixelType.Word, depth=10),
    "rgba8": F(type=ss2.PixelType.Byte, alpha=ss2.AlphaType.Straight),
    "rgba16_premul": F(type=ss2.PixelType.Word, alpha=ss2.AlphaType.Premultiplied),
    "grey16": F(type=ss2.PixelType.Word, family=ss2.ColorFamily.Grey, matrix=M.Bt709),
    "rgb_float": F(),
    "rgb_half_linear": F(type=ss2.PixelType.Half, transfer=T.Linear),
    "hlg_float_bt709": _hdr(T.AribB67, type=ss2.PixelType.Float, depth=0, subsample_w=0,
                            subsample_h=0, primaries=ss2.ColorPrimaries.Bt709),
    "pq_float": _hdr(T.St2084, type=ss2.PixelType.Float, depth=0, subsample_w=0, subsample_h=0),
}


def _image(fmt, w, h, seed, wild):
    """Random samples; `wild`: also float values far outside [0, 1] (tiny,
    negative and large ones) and integer codes past the declared depth."""
    rng = np.random.default_rng(seed)
    values = [rng.random(w * h) if p in (0, 3) or fmt.family != ss2.ColorFamily.Yuv
              else rng.random(w * h) - 0.5 for p in range(4)]
    img = helpers.pack_planes(fmt, w, h, values)
    if wild and fmt.type == ss2.PixelType.Word and fmt.depth:
        v = img.data.view("<u2")
        v[::97] = rng.integers(0, 65536, v[::97].size)
    if wild and fmt.type == ss2.PixelType.Float:
        v = img.data.view("<f4")
        v[::61] = np.resize(np.float32([-0.02, 0.0, 1e-33, 3e-40, 13.0, 90.0, -1.5, 2e-7]),
                            v[::61].size)
    return img


def _check_planes(pipe, images, w, h, precision=32):
    from oracle import binding as ob
    scales = len(ss2.plan_scales(w, h))
    for image, img in enumerate(images):
        want = ob.pyramid(helpers.to_oracle(img), 0.3, precision=precision)
        for level in range(scales):
            for c in range(3):
                if not ob.channel_pruned(c, level, scales):
                    got, w_ = pipe.debug_plane(image, level, c), want[level][c]
                    # A NaN's payload is the processor's own.
                    nan = np.isnan(w_)
                    assert np.array_equal(np.isnan(got), nan)
                    assert np.array_equal(got[~nan].view(np.uint32), w_[~nan].view(np.uint32)), \
                        (image, level, c, np.nanmax(np.abs(got - w_)))


@pytest.mark.gpu
@pytest.mark.parametrize("wild", [False, True])
@pytest.mark.parametrize("name", list(FORMATS))
def test_planes_bit_exact(name, wild):
    fmt = FORMATS[name]
    assert ss2.decode_path(fmt) == "curve"
    sizes = [(200, 134), (66, 130)]
    if not fmt.subsample_w:
        sizes += [(201, 133), (67, 65)]
    for w, h in sizes:
        images = [_image(fmt, w, h, s, wild) for s in (3, 4)]
        with ss2.Ssimulacra2Pipeline(w, h) as p:
            p.compute(*images, 0.3)
            _check_planes(p, images, w, h)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(FORMATS))
def test_half_planes_bit_exact(name):
    """The binary16 stores, averages and padding blocks of the curve kernel."""
    fmt = FORMATS[name]
    sizes = [(200, 134), (66, 130)] if fmt.subsample_w else [(201, 133), (67, 65)]
    for w, h in sizes:
        images = [_image(fmt, w, h, s, False) for s in (3, 4)]
        with ss2.Ssimulacra2Pipeline(w, h, half_planes=True) as p:
            p.compute(*images, 0.3)
            _check_planes(p, images, w, h, precision=16)


@pytest.mark.gpu
@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("name,w,h", [("pq420p10", 1664, 1472), ("rgb16", 1663, 1471)])
def test_large_single_pair_bit_exact(name, w, h, half):
    """One pair of 1,196 tiles, more than two waves (1,184): the one-pair
    kernel of 128 threads, as a graph's first launch and its next replay."""
    fmt = FORMATS[name]
    images = [_image(fmt, w, h, s, False) for s in (6, 7)]
    with ss2.Ssimulacra2Pipeline(w, h, half_planes=half) as p:
        p.compute(images[1], images[0], 0.3)
        p.compute(*images, 0.3)
        _check_planes(p, images, w, h, precision=16 if half else 32)


@pytest.mark.gpu
def test_one_pair_replays_with_two_decodes():
    """Images of different decode groups give a captured call two prepare
    launches; each replay takes its own pair's record in both."""
    w, h = 258, 130
    names = [("pq420p10", "rgb8"), ("rgb8", "pq420p10"), ("rgba8", "yuv"), ("yuv", "rgb8"),
             ("pq420p10", "hlg422p10")]
    formats = dict(FORMATS, rgb8=F(type=ss2.PixelType.Byte),
                   yuv=_hdr(T.Bt709, matrix=M.Bt709, primaries=ss2.ColorPrimaries.Bt709))
    pairs = [tuple(_image(formats[n], w, h, 10 * k + i, False) for i, n in enumerate(pair))
             for pair in names for k in range(2)]
    with ss2.Ssimulacra2Pipeline(w, h) as p, ss2.Ssimulacra2Pipeline(w, h) as plain:
        plain.set_graphs(False)
        for images in pairs + pairs[::-1]:
            got = p.compute(*images, 0.3)
            _check_planes(p, images, w, h)
            assert np.array_equal(got.norms, plain.compute(*images, 0.3).norms)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["pq420p10", "rgba8", "rgb16"])
def test_unaligned_device_rows(name):
    """Rows off the 4-byte boundary take the samples one by one."""
    import torch
    fmt, (w, h) = FORMATS[name], (130, 98)
    images, views, keep = [], [], []
    for seed in (5, 6):
        img = _image(fmt, w, h, seed, False)
        planes, strides = [0] * 4, [0] * 4
        for p, geo in enumerate(ss2.plane_layout(fmt, w, h)):
            if geo is None:
                continue
            off, pw, ph, sb = geo
            pitch = (pw + 3) * sb
            dst = np.zeros((ph, pitch), dtype=np.uint8)
            dst[:, :pw * sb] = img.data[off:off + pw * ph * sb].reshape(ph, pw * sb)
            buf = torch.zeros(dst.size + 8, dtype=torch.uint8, device="cuda")
            buf[sb:sb + dst.size] = torch.from_numpy(dst.reshape(-1)).cuda()
            planes[p], strides[p] = buf.data_ptr() + sb, pitch
            keep.append(buf)
        images.append(img)
        views.append(ss2.DeviceImage(w, h, fmt, planes, strides, keep))
    torch.cuda.synchronize()
    with ss2.Ssimulacra2Pipeline(w, h) as p:
        p.compute(*views, 0.3)
        _check_planes(p, images, w, h)


@pytest.mark.gpu
def test_large_launches_are_bit_exact():
    """128-thread CTAs (4:2:0 windows, large launches), 256-thread ones and a
    launch held to the large window by a 4:2:2 image write the same planes."""
    w, h = 1920, 1080
    fmt = FORMATS["pq420p10"]
    pairs = [(_image(fmt, w, h, 2 * i, False), _image(fmt, w, h, 2 * i + 1, False))
             for i in range(2)]
    wide = FORMATS["hlg422p10"]
    odd = (_image(wide, 130, 98, 8, False), _image(wide, 130, 98, 9, False))
    with ss2.Ssimulacra2Batch(variant=0) as b:
        alone = [b.compute_many([p])[0] for p in pairs]
        together = b.compute_many(pairs)
        mixed = b.compute_many(pairs + [odd])
    for a, t, m in zip(alone, together, mixed):
        assert np.array_equal(a.norms, t.norms) and np.array_equal(a.norms, m.norms)
