"""The two convolutions in front of a residual sum as one kernel, against the oracle (whole numbers: no tolerance)."""
import numpy as np
import pytest

from gpu_common import compare_net, kernels_of
from n2d2_b200 import netdesc, runtime
from oracle import oracle

pytestmark = pytest.mark.gpu
ENGINE = 'tcgen05-dual'


def unit_net(C, mid, H, W, O, k, stride, mode, unsigned_relu=True, clipped=False, act='linear', weight_bits=8, seed=5, projection_first=False):
    """A residual block's first unit: conv -> branch (k x k) beside a 1x1 projection of its input, their sum, and a cell that reads it.  The later one of
    branch and projection carries the sum.  mid = 0: both read the same tensor."""
    dist = ('normal', 30) if weight_bits == 8 else ('uniform', 7)
    b = netdesc.NetBuilder('unit', 16, H, W, seed, mode, unsigned_relu=unsigned_relu, weight_dist=dist, clipped=clipped, weight_bits=weight_bits)
    x = b.conv(-1, C, 1, name='front')
    y = b.conv(x, mid, 1, name='reduce') if mid else x
    if projection_first:
        p = b.conv(x, O, 1, stride=stride, act=act, name='projection')
    y = b.conv(y, O, k, stride=stride, pad=k // 2, act=act, name='branch')
    if not projection_first:
        p = b.conv(x, O, 1, stride=stride, act=act, name='projection')
    b.conv(b.sum([y, p], act='relu', name='sum'), 32, 1, name='reader')
    return b.net


# (channels of the projection, of the branch, H, W, outputs, filter, stride, batch): K blocks of 32, 64 and 128 bytes on either side, weights
# resident and streamed, columns of 64, 128 and 256 with a part of a tile, rows that end inside a tile, one tile and many per CTA
CASES = [(64, 64, 13, 11, 256, 1, 1, 3), (64, 64, 28, 28, 256, 1, 1, 40), (256, 128, 14, 14, 512, 1, 2, 7), (512, 256, 9, 9, 1024, 1, 2, 20),
         (1024, 512, 8, 7, 2048, 1, 2, 33), (128, 256, 14, 14, 256, 3, 2, 5), (256, 512, 7, 7, 512, 3, 1, 1), (256, 512, 7, 7, 512, 3, 1, 160),
         (32, 64, 20, 20, 96, 3, 1, 9), (96, 48, 15, 15, 160, 3, 2, 6), (32, 32, 5, 3, 32, 1, 1, 2), (64, 128, 28, 28, 128, 3, 1, 30),
         (512, 256, 14, 14, 1024, 1, 1, 110), (512, 512, 9, 7, 1120, 1, 2, 300), (256, 512, 7, 7, 288, 3, 1, 400), (64, 64, 30, 30, 480, 1, 1, 90)]

# a 64-channel 3x3 branch whose projection reads other channels stays on the patch kernel
# the clusters of a branch of few tiles and long K are faster by themselves
SEPARATE = [(32, 64, 20, 20, 96, 3, 1, 9), (256, 512, 7, 7, 512, 3, 1, 1)]


@pytest.mark.parametrize('case', CASES, ids=lambda c: 'C%d_%d_%dx%d_O%d_k%d_s%d_b%d' % c)
@pytest.mark.parametrize('mode', ['double', 'fixed', 'float'])
def test_branch_and_projection(case, mode):
    C, mid, H, W, O, k, s, batch = case
    n, eng = compare_net(unit_net(C, mid, H, W, O, k, s, mode), batch, flags=0)
    assert (ENGINE in eng) == (case not in SEPARATE), eng


@pytest.mark.parametrize('mode, unsigned_relu, clipped, act', [('double', False, False, 'linear'), ('fixed', True, True, 'linear'), ('float', True, True, 'relu'),
                                                               ('single', True, False, 'relu'), ('fixed', False, False, 'linear')])
def test_branch_and_projection_forms(mode, unsigned_relu, clipped, act):
    compare_net(unit_net(128, 64, 12, 10, 256, 1, 1, mode, unsigned_relu, clipped, act), 9, flags=0, want_engine=ENGINE)


# The 3x3 layer carries the sum; a 3x3 and a 1x1 layer of one tensor; both
@pytest.mark.parametrize('mid, projection_first', [(64, True), (0, False), (0, True)])
@pytest.mark.parametrize('case', [(128, 14, 14, 256, 1, 5), (128, 15, 13, 160, 2, 40), (256, 7, 7, 512, 1, 90)], ids=lambda c: 'C%d_%dx%d_O%d_s%d_b%d' % c)
@pytest.mark.parametrize('mode', ['double', 'fixed', 'float'])
def test_order_and_inputs(case, mid, projection_first, mode):
    C, H, W, O, s, batch = case
    compare_net(unit_net(C, mid, H, W, O, 3, s, mode, projection_first=projection_first), batch, flags=0, want_engine=ENGINE)


def test_packed_weights_and_calls_of_any_size_on_one_network():
    # widened weights of both cells stand in the scratch block at once; calls below the line of the widened form run the two cells one by one
    net = unit_net(128, 128, 14, 14, 256, 3, 1, 'fixed', weight_bits=4, clipped=True)
    x = netdesc.make_input(net, 400)
    ref = oracle.run_net(net, x, 'i64')[-1].reshape(400, -1)
    qn = runtime.QuantizedNet(net, 400)
    try:
        assert ENGINE in qn.engines()
        assert any('igemm_dual' in k for k in kernels_of(qn, 400)) and not any('igemm_dual' in k for k in kernels_of(qn, 2))
        for batch in (400, 3, 399, 60):
            assert np.array_equal(qn.forward_host(x[:batch]).astype(np.int64), ref[:batch])
    finally:
        qn.close()


def test_slices_of_the_upload():
    net = unit_net(64, 64, 56, 56, 256, 1, 1, 'double')
    compare_net(net, 11, flags=0, slices=4, want_engine=ENGINE)


# bands of one to eleven rows, images of one band, many bands per CTA, maps wider than a tile's share of a row
@pytest.mark.parametrize('case', [(55, 55, 3), (55, 55, 40), (13, 9, 5), (30, 28, 60), (3, 61, 2), (40, 5, 7)], ids=lambda c: '%dx%d_b%d' % c)
@pytest.mark.parametrize('mode, clipped, unsigned_relu, act', [('fixed', False, True, 'linear'), ('fixed', True, True, 'linear'), ('float', False, True, 'linear'),
                                                               ('float', True, False, 'relu'), ('fixed', False, False, 'relu'),
                                                               ('double', False, True, 'linear'), ('single', False, False, 'relu')])
def test_patch_branch_and_projection(case, mode, clipped, unsigned_relu, act):
    H, W, batch = case
    compare_net(unit_net(64, 64, H, W, 64, 3, 1, mode, unsigned_relu, clipped, act), batch, flags=0, want_engine='patch-tcgen05-dual')


def test_patch_branch_and_projection_with_packed_weights_and_slices():
    net = unit_net(64, 64, 56, 56, 64, 3, 1, 'fixed', weight_bits=4, clipped=True)
    x = netdesc.make_input(net, 9)
    ref = oracle.run_net(net, x, 'i64')[-1].reshape(9, -1)
    qn = runtime.QuantizedNet(net, 9)
    try:
        assert 'patch-tcgen05-dual' in qn.engines()
        for batch in (9, 1, 8):
            assert np.array_equal(qn.forward_host(x[:batch]).astype(np.int64), ref[:batch])
        qn.set_slices(3)
        assert np.array_equal(qn.forward_host(x).astype(np.int64), ref)
    finally:
        qn.close()


def _bytes_held(net, batch):
    import torch
    torch.zeros(1, device='cuda')
    runtime.QuantizedNet(net, 1).close()   # (what the process itself takes)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    qn = runtime.QuantizedNet(net, batch)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    eng = qn.engines()
    qn.close()
    return held, eng


# The branch's output has no buffer where the pair is one kernel in every call (packed weights: where a single image is enough to widen them); a pair
# that stays two kernels (a 64-channel 3x3 branch whose projection reads 128 channels) does not keep the branch's input until the sum, which takes its place.
@pytest.mark.parametrize('case, weight_bits, engine', [((256, 256, 256, 1), 8, ENGINE), ((256, 256, 256, 1), 4, ENGINE), ((128, 64, 64, 3), 8, None)],
                         ids=['fused', 'packed', 'separate'])
def test_only_what_is_stored_has_a_buffer(case, weight_bits, engine):
    C, mid, O, k = case
    images = 56 * 56 * 120
    held, eng = _bytes_held(unit_net(C, mid, 56, 56, O, k, 1, 'fixed', weight_bits=weight_bits, clipped=weight_bits == 4), 120)
    assert (ENGINE in eng) == (engine is not None)
    # the front, the reduction and the sum, or the branch's output and the sum in place of the reduction; the staging of the host's calls (16 channels in, 32
    # out); weights, constants and the steps of 2 MiB that the device hands out
    assert held <= (C + mid + O + 16 + 32) * images + (24 << 20)


def _packed_layers():
    b = netdesc.NetBuilder('packed', 64, 1, 1, 3, 'fixed', weight_dist=('uniform', 7), weight_bits=4, clipped=True)
    x = b.conv(-1, 64, 1, name='front')
    x = b.fc(x, 16384, act='relu', name='wide')
    b.fc(x, 960, act='relu', name='narrow')
    return b.net


# Widened weights (one byte each) are held where a call widens them: 2^29 multiply-accumulates are 32 images of this network
@pytest.mark.parametrize('images, widened', [(4, False), (64, True)])
def test_widened_weights_are_held_where_a_call_widens_them(images, widened):
    net = _packed_layers()
    weights = sum(l['weights'].size for l in net['layers'])
    held, eng = _bytes_held(net, images)
    assert ('tcgen05-widened' in eng) == widened
    assert (held > weights * 1.25) == widened   # packed: half a byte a weight
    compare_net(net, images, flags=0)


def test_packed_pair_that_no_call_widens():
    net = unit_net(256, 256, 8, 8, 256, 1, 1, 'fixed', weight_bits=4, clipped=True)
    n, eng = compare_net(net, 3, flags=0)
    assert ENGINE not in eng and 'tcgen05-widened' not in eng
    compare_net(net, 60, flags=0, want_engine=ENGINE)
