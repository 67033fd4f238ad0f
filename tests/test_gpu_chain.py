"""An expansion with its residual sum and the 1x1 layer behind it as one kernel, against the oracle (whole numbers: no tolerance)."""
import numpy as np
import pytest

from gpu_common import compare_net
from n2d2_b200 import netdesc, runtime
from oracle import oracle

pytestmark = pytest.mark.gpu
ENGINE = 'tcgen05-chain'


def seam_net(C, N2, H, W, mode, unsigned_relu=True, clipped=False, next_act='relu', seed=19):
    """Two readers of the sum: the layer behind, which is fused, and the next sum, which reads it from memory."""
    b = netdesc.NetBuilder('seam', 16, H, W, seed, mode, unsigned_relu=unsigned_relu, weight_dist=('normal', 30), clipped=clipped)
    x = b.conv(-1, 256, 1, name='front')
    y = b.conv(b.conv(x, C, 1, name='reduce'), 256, 1, act='linear', name='expand')
    x = b.sum([y, x], act='relu', name='sum')
    z = b.conv(x, N2, 1, act=next_act, name='behind')
    b.sum([b.conv(z, 256, 1, act='linear', name='expand2'), x], act='relu', name='sum2')
    return b.net


# (channels in, outputs of the layer behind, H, W, batch): a part of a tile, one tile and many per CTA, three and four regions
CASES = [(64, 64, 13, 9, 1), (64, 128, 55, 55, 3), (128, 64, 28, 28, 30), (128, 32, 30, 29, 41), (64, 32, 7, 5, 2), (64, 96, 56, 56, 25), (64, 64, 13, 9, 25), (64, 32, 7, 5, 90)]
SEPARATE = [(64, 64, 13, 9, 1), (64, 32, 7, 5, 2)]   # few row tiles: two kernels are faster


@pytest.mark.parametrize('case', CASES, ids=lambda c: 'C%d_N%d_%dx%d_b%d' % c)
@pytest.mark.parametrize('mode', ['double', 'fixed', 'float'])
def test_expansion_and_the_layer_behind(case, mode):
    C, N2, H, W, batch = case
    n, eng = compare_net(seam_net(C, N2, H, W, mode), batch, flags=0)
    assert (ENGINE in eng) == (case not in SEPARATE)


@pytest.mark.parametrize('mode, unsigned_relu, clipped, act', [('double', False, False, 'linear'), ('single', True, False, 'linear'), ('fixed', True, True, 'relu'),
                                                               ('float', False, True, 'relu')])
def test_expansion_and_the_layer_behind_forms(mode, unsigned_relu, clipped, act):
    compare_net(seam_net(64, 64, 17, 19, mode, unsigned_relu, clipped, act), 9, flags=0, want_engine=ENGINE)


def test_calls_of_any_size_and_slices():
    net = seam_net(64, 128, 48, 48, 'double')
    x = netdesc.make_input(net, 21)
    ref = oracle.run_net(net, x, 'i64')[-1].reshape(21, -1)
    qn = runtime.QuantizedNet(net, 21)
    try:
        assert ENGINE in qn.engines()
        for batch in (21, 1, 10, 21):
            assert np.array_equal(qn.forward_host(x[:batch]).astype(np.int64), ref[:batch])
        qn.set_slices(4)
        assert np.array_equal(qn.forward_host(x).astype(np.int64), ref)
    finally:
        qn.close()
