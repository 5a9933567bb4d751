"""The forms of MatMulInteger / ConvInteger / QLinearConv that reach the tensor cores through a pass of their own -- ragged K, NCHW maps, zero
points that pad or live on the device -- and the small problems whose K blocks are shared by a cluster, at the edges of their tiles.  Integer
results: every comparison is exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _t(a, dev):
    return torch.from_numpy(np.array(a)).to(dev)


def _rand(rng, shape, dtype):
    i = np.iinfo(dtype)
    return rng.integers(i.min, i.max + 1, shape).astype(dtype)


@pytest.mark.parametrize("M,N,K", [(1, 1, 17), (7, 3, 31), (8, 63, 100), (9, 65, 127), (129, 64, 65), (130, 257, 1283), (64, 1000, 1000), (33, 130, 2049)])
@pytest.mark.parametrize("a_dtype,b_dtype", [(np.uint8, np.int8), (np.int8, np.uint8)])
def test_matmul_ragged_k(ops, orc, dev, M, N, K, a_dtype, b_dtype):
    rng = np.random.default_rng(M + N + K)
    a, b = _rand(rng, (M, K), a_dtype), _rand(rng, (K, N), b_dtype)
    za, zb = _rand(rng, K, a_dtype), _rand(rng, N, b_dtype)
    buf = torch.zeros(M * K + 3, dtype=torch.uint8 if a_dtype == np.uint8 else torch.int8, device=dev)
    buf[3:] = _t(a, dev).reshape(-1)  # rows that start on odd addresses
    for at in (_t(a, dev), buf[3:].reshape(M, K)):
        for z0, z1 in ((None, None), (za[:1], None), (None, zb), (za, zb[:1]), (za[:1], zb)):
            y = ops.MatMulInteger(at, _t(b, dev), None if z0 is None else _t(z0, dev), None if z1 is None else _t(z1, dev))
            assert np.array_equal(y.cpu().numpy(), orc.matmul_integer(a, b, z0, z1)), (z0 is None, z1 is None)


def test_matmul_ragged_k_batched(ops, orc, dev):
    rng = np.random.default_rng(5)
    a, b = _rand(rng, (3, 5, 37), np.uint8), _rand(rng, (3, 37, 21), np.int8)
    y = ops.MatMulInteger(_t(a, dev), _t(b, dev), _t(np.array([9], np.uint8), dev), None)
    assert np.array_equal(y.cpu().numpy(), orc.matmul_integer(a, b, np.array([9], np.uint8), None))


def test_pair_kernel_column_groups(ops, dev):
    """More than eight 256-column blocks, the last group and the last pair of position tiles partial.  |sum| < 2^24: the fp32 product is exact."""
    M, N, K = 1100, 2305, 128
    gen = torch.Generator(device=dev).manual_seed(3)
    a = torch.randint(0, 256, (M, K), dtype=torch.uint8, device=dev, generator=gen)
    b = torch.randint(-127, 128, (K, N), dtype=torch.int8, device=dev, generator=gen)
    want = (a.double() @ b.double()).to(torch.int32)
    assert torch.equal(ops.MatMulInteger(a, b, None, None), want)


# (N, C, H, W, M, k, stride, pad)
CONVS = [
    (1, 5, 9, 7, 3, 3, 1, 1),        # few channels, odd everything
    (2, 17, 13, 11, 33, 3, 2, 1),
    (3, 64, 8, 16, 64, 1, 1, 0),     # 1x1: flattened positions; the plane is one 128-position tile
    (1, 65, 12, 43, 70, 5, 1, 2),    # second channel tile of one channel, four positions that cross rows of the padded map
    (2, 130, 7, 7, 257, 3, 1, 1),    # several channel shares of the pixel sums
    (1, 16, 23, 23, 16, 1, 2, 0),    # strided 1x1
    (2, 48, 10, 9, 24, 3, 2, 1),     # NHWC rows the tensor-core kernel reads as they are
    (2, 20, 6, 6, 40, 3, 1, 4),      # padding wider than the kernel
]


@pytest.mark.parametrize("case", CONVS)
@pytest.mark.parametrize("x_dtype,w_dtype", [(np.uint8, np.int8), (np.int8, np.uint8)])
def test_conv_integer_nchw_zero_points(ops, orc, dev, case, x_dtype, w_dtype):
    N, C, H, W, M, k, s, p = case
    rng = np.random.default_rng(C + M)
    x, w = _rand(rng, (N, C, H, W), x_dtype), _rand(rng, (M, C, k, k), w_dtype)
    zws = (None, _rand(rng, M, w_dtype), _rand(rng, 1, w_dtype))
    xt = _t(x, dev)
    odd = torch.zeros(xt.numel() + 1, dtype=xt.dtype, device=dev)
    odd[1:] = xt.reshape(-1)
    for zx in (0, 77):
        for zw in zws:
            want = orc.conv_integer(x, w, zx, zw, (s, s), (p, p))
            zwt = None if zw is None else _t(zw, dev)
            zxd = _t(np.array(zx, x_dtype), dev)
            for xin in (xt, odd[1:].reshape(xt.shape), xt.contiguous(memory_format=torch.channels_last)):
                for z in (x_dtype(zx), zxd):
                    y = ops.ConvInteger(xin, _t(w, dev), z, zwt, (s, s), (p, p))
                    assert np.array_equal(y.cpu().numpy(), want), (zx, zw is None, xin.stride(), type(z))


@pytest.mark.parametrize("case", CONVS)
def test_qlinear_conv_nchw_zero_points(ops, orc, dev, case):
    N, C, H, W, M, k, s, p = case
    rng = np.random.default_rng(C * M)
    x, w = _rand(rng, (N, C, H, W), np.uint8), _rand(rng, (M, C, k, k), np.int8)
    ws = rng.uniform(0.001, 0.002, M).astype(np.float32)
    bias = rng.integers(-500, 500, M).astype(np.int32)
    ys = float(0.02 * 0.0015 * 74 * 73 * np.sqrt(C * k * k) / 40)
    for zx in (0, 77):
        for zw in (np.zeros(M, np.int8), _rand(rng, M, np.int8)):
            acc = orc.conv_integer(x, w, zx, zw, (s, s), (p, p))
            want = orc.requantize(acc, 0.02, ws, ys, 11, bias=bias, channel_axis=1)
            y = ops.QLinearConv(_t(x, dev), 0.02, np.uint8(zx), _t(w, dev), _t(ws, dev), _t(zw, dev), ys, np.uint8(11), _t(bias, dev), (s, s), (p, p))
            assert np.array_equal(y.cpu().numpy(), want), (zx, zw.any())


# small batches: few tiles (boxes that do not divide the map) and K blocks shared by clusters of two and four
@pytest.mark.parametrize("N,C,H,W,M,k,s", [(1, 512, 7, 7, 512, 3, 1), (1, 1024, 14, 14, 256, 1, 1), (3, 256, 14, 14, 72, 3, 2), (1, 576, 5, 9, 64, 1, 1),
                                           (1, 256, 28, 28, 1100, 3, 1), (2, 80, 11, 5, 17, 3, 1)])
def test_small_batch_split_k(ops, pkg, orc, dev, N, C, H, W, M, k, s):
    rng = np.random.default_rng(C + H)
    x, w = _rand(rng, (N, C, H, W), np.uint8), _rand(rng, (M, C, k, k), np.int8)
    p = k // 2
    ws = rng.uniform(0.001, 0.002, M).astype(np.float32)
    zw = np.zeros(M, np.int8)
    ys = float(0.02 * 0.0015 * 74 * 73 * np.sqrt(C * k * k) / 40)
    acc = orc.conv_integer(x, w, 0, None, (s, s), (p, p))
    res = _rand(rng, acc.shape, np.uint8)
    cl = lambda a: _t(a, dev).contiguous(memory_format=torch.channels_last)  # noqa: E731
    pk = ops.PackedConv(_t(w, dev), _t(zw, dev), x.shape, (s, s), (p, p))
    assert np.array_equal(ops.ConvIntegerPacked(cl(x), pk).cpu().numpy(), acc)
    for fold in (False, True):
        want = orc.qadd_relu(orc.requantize(acc, 0.02, ws, ys, 121, channel_axis=1, fold=fold), ys, 121, res, 0.05, 9, 0.11, 0, relu=True, fold=fold)
        got = []
        for variant in (0, 1):
            assert pkg.lib().chxq_tc_variant(variant) == 0
            try:
                got.append(ops.QLinearConvPacked(cl(x), pk, 0.02, np.uint8(0), _t(ws, dev), _t(zw, dev), ys, np.uint8(121), residual=cl(res), res_scale=0.05,
                                                 res_zero_point=9, out_scale=0.11, out_zero_point=0, fold_scales=fold).cpu().numpy())
            finally:
                pkg.lib().chxq_tc_variant(0)
        assert np.array_equal(got[0], want) and np.array_equal(got[1], want)


# the position box of a strided convolution has to fit a TMA box: 256 input rows
@pytest.mark.parametrize("N,H,W,k,s,p", [(2, 382, 19, 3, (3, 3), (1, 1)), (2, 509, 1, 1, (4, 1), (0, 0)), (1, 1017, 3, 1, (8, 8), (0, 0))])
def test_strided_conv_tall_box(ops, orc, dev, N, H, W, k, s, p):
    rng = np.random.default_rng(H)
    x, w = _rand(rng, (N, 16, H, W), np.uint8), _rand(rng, (8, 16, k, k), np.int8)
    zw = _rand(rng, 8, np.int8)
    wt, xt = _t(w, dev), _t(x, dev)
    for zx in (0, 9):
        for zp in (None, zw):
            want = orc.conv_integer(x, w, zx, zp, s, p)
            for xin in (xt, xt.contiguous(memory_format=torch.channels_last)):
                for path in (ops.PATH_AUTO, ops.PATH_TENSOR):
                    y = ops.ConvInteger(xin, wt, np.uint8(zx), None if zp is None else _t(zp, dev), s, p, path=path)
                    assert np.array_equal(y.cpu().numpy(), want), (zx, zp is None, xin.stride(), path)


# no zero point of x, zero points of w: fewer position tiles than with a border, so more channel shares of the pixel sums
@pytest.mark.parametrize("N,C,H,W,M,k,p", [(6, 80, 112, 112, 16, 3, 1), (78, 128, 128, 8, 64, 3, (1, 0))])
def test_conv_pixel_sums_fit_the_reported_workspace(ops, dev, N, C, H, W, M, k, p):
    gen = torch.Generator(device=dev).manual_seed(C)
    kw = k if isinstance(p, int) else 1
    pads = (p, p) if isinstance(p, int) else p
    x = torch.randint(0, 256, (N, C, H, W), dtype=torch.uint8, device=dev, generator=gen)
    w = torch.randint(-127, 128, (M, C, k, kw), dtype=torch.int8, device=dev, generator=gen)
    zw = torch.randint(-9, 10, (M,), dtype=torch.int8, device=dev, generator=gen)
    ws = torch.rand(M, device=dev, generator=gen) * 1e-3 + 1e-3
    args = (x, 0.02, np.uint8(0), w, ws, zw, 0.9, np.uint8(100), None, (1, 1), pads)
    assert torch.equal(ops.QLinearConv(*args, path=ops.PATH_TENSOR), ops.QLinearConv(*args, path=ops.PATH_SIMT))


# (batch, M, N, K, launches): the copy and the product (two launches a matrix) where they are faster than the one of the CUDA cores
@pytest.mark.parametrize("batch,M,N,K,launches", [(1, 1, 1, 249, 2), (1, 7, 3, 259, 2), (1, 8, 63, 265, 2), (1, 9, 65, 255, 2), (1, 129, 64, 321, 2), (2, 5, 21, 561, 4),
                                                  (3, 130, 257, 1283, 6), (1, 49, 49, 50, 1), (512, 49, 49, 50, 1), (5, 70, 33, 197, 1)])
def test_matmul_ragged_k_launches(ops, pkg, orc, dev, batch, M, N, K, launches):
    rng = np.random.default_rng(batch + M + N + K)
    lead = () if batch == 1 else (batch,)
    a, b = _rand(rng, lead + (M, K), np.uint8), _rand(rng, lead + (K, N), np.int8)
    za, zb = _rand(rng, K, np.uint8), _rand(rng, N, np.int8)
    at, bt = _t(a, dev), _t(b, dev)
    for z0, z1 in ((None, None), (za[:1], zb), (za, zb[:1])):
        before = pkg.lib().chxq_launch_count()
        y = ops.MatMulInteger(at, bt, None if z0 is None else _t(z0, dev), None if z1 is None else _t(z1, dev))
        assert pkg.lib().chxq_launch_count() - before == launches
        assert np.array_equal(y.cpu().numpy(), orc.matmul_integer(a, b, z0, z1)), (z0 is None, z1 is None)


# (N, C, H, W, M, k, launches): with a device zero point, one launch of the CUDA-core kernel, or two where the tensor cores are faster
@pytest.mark.parametrize("N,C,H,W,M,k,launches", [(1, 3, 7, 7, 16, 3, 1), (1, 16, 2, 2, 4, 1, 1), (1, 5, 32, 32, 16, 1, 1), (1, 24, 7, 7, 16, 3, 2), (2, 100, 5, 6, 16, 1, 2),
                                                  (16, 3, 24, 23, 32, 3, 2)])
def test_conv_integer_device_zero_point_launches(ops, pkg, orc, dev, N, C, H, W, M, k, launches):
    rng = np.random.default_rng(C + M)
    x, w = _rand(rng, (N, C, H, W), np.uint8), _rand(rng, (M, C, k, k), np.uint8)
    zw = _rand(rng, M, np.uint8)
    args = (_t(x, dev), _t(w, dev), _t(np.array([77], np.uint8), dev), _t(zw, dev), (1, 1), (k // 2, k // 2))
    before = pkg.lib().chxq_launch_count()
    y = ops.ConvInteger(*args)
    assert pkg.lib().chxq_launch_count() - before == launches
    assert np.array_equal(y.cpu().numpy(), orc.conv_integer(x, w, 77, zw, (1, 1), (k // 2, k // 2)))


# requantized products of ragged K: the general epilogue (int8 outputs here) moves the line
@pytest.mark.parametrize("M,N,K,launches_u8,launches_s8", [(64, 208, 188, 2, 1), (280, 171, 44, 1, 1), (996, 901, 447, 2, 2), (2, 4, 725, 2, 2)])
def test_qlinear_matmul_ragged_k_launches(ops, pkg, orc, dev, M, N, K, launches_u8, launches_s8):
    rng = np.random.default_rng(M + K)
    a, b = _rand(rng, (M, K), np.uint8), _rand(rng, (K, N), np.int8)
    ys = float(0.02 * 0.0015 * 74 * 73 * np.sqrt(K) / 40)
    acc = orc.matmul_integer(a, b, np.array([9], np.uint8), None)
    for oz, launches in ((np.uint8(11), launches_u8), (np.int8(-5), launches_s8)):
        before = pkg.lib().chxq_launch_count()
        y = ops.QLinearMatMul(_t(a, dev), 0.02, np.uint8(9), _t(b, dev), 0.0015, np.int8(0), ys, oz)
        assert pkg.lib().chxq_launch_count() - before == launches
        want = orc.requantize(acc, 1.0, np.array([np.float32(0.02) * np.float32(0.0015)], np.float32), ys, int(oz), y_dtype=type(oz))
        assert np.array_equal(y.cpu().numpy(), want)


# as many clusters of four CTAs as are resident at once, one more (pairs then), and around the last pair
@pytest.mark.parametrize("tiles", [33, 34, 37, 74, 75])
def test_split_k_last_cluster(ops, dev, tiles):
    """|sum| < 2^24: the fp64 product is exact."""
    M, N, K = 8, 64 * tiles - 3, 1232
    gen = torch.Generator(device=dev).manual_seed(tiles)
    a = torch.randint(0, 256, (M, K), dtype=torch.uint8, device=dev, generator=gen)
    b = torch.randint(-127, 128, (K, N), dtype=torch.int8, device=dev, generator=gen)
    assert torch.equal(ops.MatMulInteger(a, b, None, None), (a.double() @ b.double()).to(torch.int32))
