"""A 3x3 depthwise cell and the 1x1 cell behind it as one kernel, against the oracle (whole numbers: no tolerance)."""
import numpy as np
import pytest

from gpu_common import compare_net, kernels_of_host_call
from n2d2_b200 import netdesc, runtime
from oracle import oracle

pytestmark = pytest.mark.gpu
ENGINE = 'depthwise-1x1-tcgen05'


def pair_net(C, H, W, N, stride, pad, mode, act='relu', clipped=False, seed=11):
    b = netdesc.NetBuilder('pair', 16, H, W, seed, mode, weight_dist=('normal', 30), clipped=clipped)
    x = b.conv(-1, C, 1, name='front')   # the depthwise cell does not read the caller's buffer
    x = b.conv(x, C, 3, stride=stride, pad=pad, groups=C, name='dw')
    b.conv(x, N, 1, act=act, name='pw')
    return b.net


# (C, H, W, N, stride, pad, batch): K blocks of 32, 64 and 128 channels, one to four of them; output rows of one to several segments; tiles
# that end inside an image and span up to five; maps of one pixel and one row; columns that do not fill an accumulator; weights resident and
# streamed; column ranges on several CTAs; one, two and more tiles per CTA
CASES = [(32, 112, 112, 64, 1, 1, 3), (64, 30, 30, 128, 2, 1, 5), (128, 28, 28, 128, 1, 1, 2), (128, 28, 28, 256, 2, 1, 33), (256, 14, 14, 512, 2, 1, 40),
         (512, 14, 14, 512, 1, 1, 1), (512, 14, 14, 512, 1, 1, 150), (512, 14, 14, 1024, 2, 1, 37), (1024, 7, 7, 1024, 1, 1, 50), (1024, 7, 7, 1024, 1, 1, 1),
         (96, 9, 13, 32, 1, 1, 3), (192, 5, 7, 96, 2, 0, 9), (160, 3, 3, 160, 1, 2, 70), (256, 1, 1, 64, 1, 1, 300), (64, 1, 17, 64, 1, 1, 2),
         (32, 6, 300, 96, 1, 1, 2), (64, 5, 259, 128, 2, 1, 3), (128, 4, 127, 64, 1, 1, 3), (480, 6, 5, 576, 2, 2, 11),
         (256, 14, 14, 512, 2, 1, 140), (96, 40, 41, 64, 1, 1, 5), (192, 33, 31, 96, 2, 0, 40), (256, 1, 1, 64, 1, 1, 30), (64, 7, 7, 32, 1, 1, 140),
         (256, 13, 9, 160, 1, 1, 2), (384, 5, 5, 384, 1, 1, 2), (512, 3, 3, 512, 1, 2, 300), (384, 9, 13, 384, 1, 1, 60), (128, 3, 3, 96, 1, 2, 9),
         (32, 6, 300, 64, 1, 1, 8), (64, 5, 259, 128, 2, 1, 20), (128, 28, 28, 128, 1, 1, 1), (64, 1, 97, 64, 1, 1, 70)]

# two kernels are faster: a few rows per multiprocessor, many outputs, more than four K blocks or three of few rows
SEPARATE = [(32, 6, 300, 96, 1, 1, 2), (64, 30, 30, 128, 2, 1, 5), (512, 14, 14, 1024, 2, 1, 37),
            (1024, 7, 7, 1024, 1, 1, 50), (96, 9, 13, 32, 1, 1, 3), (192, 5, 7, 96, 2, 0, 9), (160, 3, 3, 160, 1, 2, 70), (256, 1, 1, 64, 1, 1, 300), (480, 6, 5, 576, 2, 2, 11), (384, 5, 5, 384, 1, 1, 2)]


@pytest.mark.parametrize('case', CASES, ids=lambda c: 'C%d_%dx%d_N%d_s%d_p%d_b%d' % c)
@pytest.mark.parametrize('mode', ['single', 'fixed', 'float'])
def test_depthwise_and_pointwise(case, mode):
    C, H, W, N, s, p, batch = case
    n, eng = compare_net(pair_net(C, H, W, N, s, p, mode), batch, flags=0)
    assert (ENGINE in eng) == (case not in SEPARATE and mode != 'float')


@pytest.mark.parametrize('mode, clipped, act', [('double', False, 'linear'), ('fixed', True, 'relu'), ('float', True, 'linear')])
def test_depthwise_and_pointwise_forms(mode, clipped, act):
    net = pair_net(128, 13, 11, 160, 1, 1, mode, act, clipped)
    n, eng = compare_net(net, 3, flags=0)
    assert (ENGINE in eng) == (mode != 'float')


def test_calls_of_any_size_on_one_network():
    net = netdesc.mobilenet_v1(size=64, classes=100)
    x = netdesc.make_input(net, 40)
    ref = oracle.run_net(net, x, 'i64')[-1].reshape(40, -1)
    qn = runtime.QuantizedNet(net, 40)
    try:
        assert qn.engines().count(ENGINE) == 5   # (the maps behind them are a few rows per multiprocessor)
        for batch in (40, 1, 7, 39, 2, 40):
            assert np.array_equal(qn.forward_host(x[:batch]).astype(np.int64), ref[:batch])
    finally:
        qn.close()


# The leading cells of a host call run slice by slice while their outputs have 2048 pixels and more: one segment to a row and several, a patch of one tile
# and of several, slices of one image and of three (weights 2, 2, 2, 1)
@pytest.mark.parametrize('case', [(32, 56, 56, 64, 1), (64, 112, 112, 128, 2), (128, 48, 50, 160, 1), (32, 16, 260, 64, 1)], ids=lambda c: 'C%d_%dx%d_N%d_s%d' % c)
@pytest.mark.parametrize('mode', ['single', 'fixed'])
def test_slices_of_the_upload(case, mode):
    C, H, W, N, s = case
    net = pair_net(C, H, W, N, s, 1, mode)
    x = netdesc.make_input(net, 11)
    ref = oracle.run_net(net, x, 'i64')[-1].reshape(11, -1)
    qn = runtime.QuantizedNet(net, 11)
    try:
        assert qn.engines()[2] == ENGINE
        qn.set_slices(4)
        for batch in (11, 7, 10):
            out, kernels = kernels_of_host_call(qn, x[:batch])
            assert sum('dwpw' in k for k in kernels) == 4
            assert np.array_equal(out.astype(np.int64), ref[:batch])
    finally:
        qn.close()
