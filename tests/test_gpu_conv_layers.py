"""Every convolution shape of the U-Net, one layer at a time, through the C ABI
(kv_conv3_bf16): the tcgen05 / TMA implicit GEMM against the mma.sync kernel
(the same products summed in the same K order: bit-identical) and against an
FP64 conv3d of the same BF16 inputs and weights.  Against FP64 the output
differs by the final rounding to BF16 (half an ulp) plus the error of the
FP32 accumulation on the tensor cores, which align the products of each MMA
step to the largest and truncate: measured 1e-6 .. 6e-6 absolute on sums of
5184 products whose magnitudes add to ~50, so the bound is
2^-8 |ref| + 2^-20 sum|w x|, and at least 99 % of the outputs must equal
the FP64 value rounded to nearest even."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (level, c1, c2, cout, relu) at a 16 x 32 x 128 input (level l: each side
# halved l times): the encoder, the bottleneck, the decoder's concatenated
# inputs (upsampled ++ skip) and the backward-data convolutions (transposed
# weights: c_out = the forward layer's input channels)
SHAPES = [
    (0, 16, 0, 16, True), (1, 16, 0, 32, True), (1, 32, 0, 32, True), (2, 32, 0, 64, True),
    (2, 64, 0, 64, True), (3, 64, 0, 128, True), (3, 128, 0, 128, True),
    (2, 128, 64, 64, True), (1, 64, 32, 32, True), (0, 32, 16, 16, True),
    (3, 128, 0, 64, False), (2, 64, 0, 192, False), (1, 32, 0, 96, False), (0, 16, 0, 48, False),
]
BASE = (16, 32, 128)


def _bf16_bits(x):
    """float32 array -> BF16 bit patterns (round to nearest even) and their float32 values."""
    u = np.ascontiguousarray(x, np.float32).view(np.uint32)
    r = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)
    return r, (r.astype(np.uint32) << 16).view(np.float32)


def _conv(ctx, a, c1, b, c2, w, bias, relu, cout, dims, kernel):
    import torch
    from kevernals_gb300 import _lib
    D, H, W = dims
    dev = torch.device("cuda")
    ta = torch.from_numpy(a.view(np.int16)).to(dev)
    tb = torch.from_numpy(b.view(np.int16)).to(dev) if c2 else None
    tw = torch.from_numpy(w.view(np.int16)).to(dev)
    tbias = torch.from_numpy(bias).to(dev)
    out = torch.empty((D, H, W, cout), dtype=torch.int16, device=dev)
    ctx.use_torch_stream()
    st = _lib.lib().kv_conv3_bf16(ctx.handle, C.c_void_p(ta.data_ptr()), c1,
                                  C.c_void_p(tb.data_ptr() if tb is not None else 0), c2,
                                  C.c_void_p(tw.data_ptr()), C.c_void_p(tbias.data_ptr()), int(relu),
                                  C.c_void_p(out.data_ptr()), cout, D, H, W, kernel)
    assert st == 0, ctx.last_error()
    ctx.sync()
    return out.cpu().numpy().view(np.uint16)


@pytest.fixture(scope="module")
def ctx():
    from kevernals_gb300 import build, engine
    build.build()
    return engine.Context(0)


@pytest.mark.parametrize("shape", SHAPES, ids=[f"L{s[0]}_{s[1]}+{s[2]}to{s[3]}" for s in SHAPES])
def test_conv_layer_tcgen05_vs_mma_sync_and_fp64(ctx, shape):
    torch = pytest.importorskip("torch")
    import torch.nn.functional as F
    lvl, c1, c2, cout, relu = shape
    dims = tuple(d >> lvl for d in BASE)
    D, H, W = dims
    rng = np.random.default_rng(lvl * 1000 + c1 * 7 + c2 * 3 + cout)
    a, af = _bf16_bits(rng.standard_normal((D, H, W, c1)).astype(np.float32))
    b, bf = _bf16_bits(rng.standard_normal((D, H, W, max(c2, 1))).astype(np.float32))
    cin = c1 + c2
    scale = 1.0 / np.sqrt(27 * cin)
    w, wf = _bf16_bits((rng.standard_normal((cout, 27, cin)) * scale).astype(np.float32))
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    tc = _conv(ctx, a, c1, b, c2, w, bias, relu, cout, dims, 1)
    ms = _conv(ctx, a, c1, b, c2, w, bias, relu, cout, dims, 2)
    assert np.array_equal(tc, ms)
    # FP64 reference on the same BF16 values
    x = af if c2 == 0 else np.concatenate([af, bf], axis=3)
    xt = torch.from_numpy(x.astype(np.float64)).permute(3, 0, 1, 2)[None]
    wt = torch.from_numpy(wf.astype(np.float64)).permute(0, 2, 1).reshape(cout, cin, 3, 3, 3)
    ref = F.conv3d(xt, wt, torch.from_numpy(bias.astype(np.float64)), padding=1)
    mag = F.conv3d(xt.abs(), wt.abs(), torch.from_numpy(np.abs(bias).astype(np.float64)), padding=1)
    if relu:
        ref = F.relu(ref)
    ref = ref[0].permute(1, 2, 3, 0).numpy()
    mag = mag[0].permute(1, 2, 3, 0).numpy()
    got = (tc.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    err = np.abs(got - ref)
    bound = 2 ** -8 * np.abs(ref) + 2 ** -20 * mag
    worst = np.unravel_index(np.argmax(err - bound), err.shape)
    assert np.all(err <= bound), (worst, got[worst], ref[worst], mag[worst])
    _, rne = _bf16_bits(ref.astype(np.float32))
    assert np.mean(got == rne) > 0.99
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 4e-3


# column shapes of the z-marching kernel: rows left over in y, one plane, a
# share that starts inside a column, several rows of a narrow volume per
# sub-tile (128, 64, 48, 32 and 16 voxels wide, and 192), weights that stay in
# shared memory and weights that stream, channel groups of 16, 32, 48 and 64
COLUMNS = [
    (1, 1, 128, 16, 0, 16), (3, 11, 128, 16, 0, 16), (37, 23, 128, 32, 16, 16), (5, 3, 256, 16, 0, 48),
    (7, 14, 64, 64, 32, 32), (3, 6, 64, 32, 0, 96), (2, 20, 32, 128, 64, 64), (4, 24, 16, 128, 0, 128),
    (2, 5, 192, 32, 0, 32), (3, 7, 48, 64, 0, 64), (1, 2, 16, 64, 0, 192), (9, 1, 384, 64, 128, 80),
]


@pytest.mark.parametrize("shape", COLUMNS, ids=["x".join(map(str, s[:3])) + f"_{s[3]}+{s[4]}to{s[5]}" for s in COLUMNS])
def test_conv_columns_equal_mma_sync(ctx, shape):
    """The default route against the mma.sync kernel: the same sums in the same order, equal bits."""
    pytest.importorskip("torch")
    D, H, W, c1, c2, cout = shape
    rng = np.random.default_rng(sum(shape))
    a, _ = _bf16_bits(rng.standard_normal((D, H, W, c1)).astype(np.float32))
    b, _ = _bf16_bits(rng.standard_normal((D, H, W, max(c2, 1))).astype(np.float32))
    w, _ = _bf16_bits((rng.standard_normal((cout, 27, c1 + c2)) / np.sqrt(27 * (c1 + c2))).astype(np.float32))
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    got = _conv(ctx, a, c1, b, c2, w, bias, True, cout, (D, H, W), 0)
    assert np.array_equal(got, _conv(ctx, a, c1, b, c2, w, bias, True, cout, (D, H, W), 2))


@pytest.mark.parametrize("c1,c2,cout", [(128, 16, 16), (16, 128, 32), (128, 128, 256), (48, 0, 16)])
def test_conv_limits_are_refused(ctx, c1, c2, cout):
    """Channel counts outside the operator's limits on a volume of whole tiles: an error, nothing run."""
    torch = pytest.importorskip("torch")
    from kevernals_gb300 import _lib
    t = torch.zeros(2 * 128 * 256 * 27, dtype=torch.int16, device="cuda")
    f = torch.zeros(256, device="cuda")
    p = C.c_void_p(t.data_ptr())
    for kernel in (0, 1):
        st = _lib.lib().kv_conv3_bf16(ctx.handle, p, c1, p if c2 else None, c2, p, C.c_void_p(f.data_ptr()), 1, p,
                                      cout, 1, 2, 128, kernel)
        assert _lib.STATUS_NAMES[st] == "KV_ERR_UNSUPPORTED"


@pytest.mark.parametrize("dims", [(1, 3, 24), (2, 5, 8), (1, 1, 100), (3, 2, 136), (1, 1, 1)])
@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_conv_widths_are_refused(ctx, dims, kernel):
    """Widths that are not multiples of 16, on volumes that are not whole tiles: an error, nothing run."""
    torch = pytest.importorskip("torch")
    from kevernals_gb300 import _lib
    t = torch.zeros(2 * 128 * 256 * 27, dtype=torch.int16, device="cuda")
    f = torch.zeros(256, device="cuda")
    p = C.c_void_p(t.data_ptr())
    st = _lib.lib().kv_conv3_bf16(ctx.handle, p, 16, None, 0, p, C.c_void_p(f.data_ptr()), 1, p, 16, *dims, kernel)
    assert _lib.STATUS_NAMES[st] == "KV_ERR_UNSUPPORTED"


@pytest.mark.parametrize("dims", [(2, 16, 8), (4, 32, 4), (64, 2, 1), (1, 64, 2)])
def test_conv_narrow_whole_tiles(ctx, dims):
    """Whole tiles of volumes narrower than 16 voxels, against FP64 at the bound of the layers above."""
    torch = pytest.importorskip("torch")
    import torch.nn.functional as F
    rng = np.random.default_rng(sum(dims))
    a, af = _bf16_bits(rng.standard_normal((*dims, 32)).astype(np.float32))
    w, wf = _bf16_bits((rng.standard_normal((16, 27, 32)) / np.sqrt(27 * 32)).astype(np.float32))
    bias = (rng.standard_normal(16) * 0.1).astype(np.float32)
    xt = torch.from_numpy(af.astype(np.float64)).permute(3, 0, 1, 2)[None]
    wt = torch.from_numpy(wf.astype(np.float64)).permute(0, 2, 1).reshape(16, 32, 3, 3, 3)
    bt = torch.from_numpy(bias.astype(np.float64))
    ref = F.conv3d(xt, wt, bt, padding=1)[0].permute(1, 2, 3, 0).numpy()
    mag = F.conv3d(xt.abs(), wt.abs(), bt.abs(), padding=1)[0].permute(1, 2, 3, 0).numpy()
    for kernel in (0, 1):
        bits = _conv(ctx, a, 32, a, 0, w, bias, False, 16, dims, kernel)
        got = (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
        assert np.all(np.abs(got - ref) <= 2 ** -8 * np.abs(ref) + 2 ** -20 * mag)


@pytest.mark.parametrize("shape", [(16, 16, 128, 16, 0, 16), (4, 32, 32, 64, 0, 64), (3, 5, 128, 16, 16, 48), (1, 8, 16, 32, 0, 32),
                                   (2, 9, 64, 64, 32, 32), (5, 4, 256, 128, 64, 64)],
                         ids=lambda s: "x".join(map(str, s[:3])) + f"_{s[3]}+{s[4]}to{s[5]}")
@pytest.mark.parametrize("tap", [4, 13, 22])   # of the plane before, this one, the one after
def test_conv_weights_that_are_not_finite(ctx, shape, tap):
    """An infinity and a NaN among the weights, one a channel: the zeros outside the volume make NaN of them, as in the
    mma.sync kernel; every other channel is untouched."""
    pytest.importorskip("torch")
    D, H, W, c1, c2, cout = shape
    rng = np.random.default_rng(sum(shape))
    a, _ = _bf16_bits(np.abs(rng.standard_normal((D, H, W, c1))).astype(np.float32) + 0.1)
    b, _ = _bf16_bits(np.abs(rng.standard_normal((D, H, W, max(c2, 1)))).astype(np.float32) + 0.1)
    w, _ = _bf16_bits((rng.standard_normal((cout, 27, c1 + c2)) / np.sqrt(27 * (c1 + c2))).astype(np.float32))
    w[3, tap, 5], w[cout - 2, tap, c1 + c2 - 1] = 0x7f80, 0x7fc0
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    want = _conv(ctx, a, c1, b, c2, w, bias, False, cout, (D, H, W), 2)
    got = _conv(ctx, a, c1, b, c2, w, bias, False, cout, (D, H, W), 0)
    nan_w, nan_g = (want & 0x7fff) > 0x7f80, (got & 0x7fff) > 0x7f80
    assert nan_w.any() and np.array_equal(nan_g, nan_w)
    assert np.array_equal(got[~nan_w], want[~nan_w])
