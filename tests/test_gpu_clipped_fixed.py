"""Clipped fixed-point scalings whose products leave 32 bits, on the kernel families they used to be kept from, against the oracle (whole numbers:
no tolerance)."""
import pytest

from gpu_common import KEEP, compare_net, single_conv_net
from n2d2_b200 import netdesc
from n2d2_b200 import runtime as R

pytestmark = pytest.mark.gpu

# (C, H, W, O, k, stride, pad, groups, batch, flags, engine): first layers (gather, space-to-depth), patches, the implicit GEMM with one and two tiles per
# weight slab and with a cluster per tile, a depthwise layer, a fully-connected shape
CASES = [(3, 40, 44, 32, 7, 1, 3, 1, 2, 0, 'stem-tcgen05'), (3, 40, 44, 32, 7, 2, 3, 1, 2, 0, 'stem-tcgen05'), (64, 17, 19, 64, 3, 1, 1, 1, 3, 0, 'patch-tcgen05'),
         (128, 13, 9, 96, 3, 1, 1, 1, 2, 0, 'patch-tcgen05'), (256, 9, 9, 256, 3, 1, 1, 1, 3, 0, 'tcgen05'), (1024, 6, 5, 64, 1, 1, 0, 1, 3, 0, 'tcgen05'),
         (512, 9, 9, 256, 3, 1, 1, 1, 2, R.FORCE_PAIR, 'tcgen05-pair'), (512, 7, 7, 512, 3, 1, 1, 1, 1, 0, 'tcgen05'),
         (64, 15, 13, 64, 3, 1, 1, 64, 2, 0, 'depthwise'), (2048, 1, 1, 1000, 1, 1, 0, 1, 5, 0, 'tcgen05')]


@pytest.mark.parametrize('case', CASES, ids=lambda c: 'C%d_%dx%d_O%d_k%d_s%d_g%d_f%d' % (c[:6] + (c[7], c[9])))
@pytest.mark.parametrize('act', ['relu', 'linear'])
@pytest.mark.parametrize('signed_relu', [False, True])
def test_clipped_fixed_point(case, act, signed_relu):
    C, H, W, O, k, s, p, g, batch, flags, engine = case
    net = single_conv_net(C, H, W, O, k, s, p, act=act, mode='fixed', groups=g, clipped=True, unsigned_relu=not signed_relu)
    compare_net(net, batch, flags=KEEP | flags, want_engine=engine)


@pytest.mark.parametrize('batch', [1, 5, 40])
def test_clipped_residual_network(batch):
    net = netdesc.resnet18(size=64, classes=100, clipped=True)
    n, eng = compare_net(net, batch, flags=0)
    assert eng[0] == 'stem-pool-tcgen05' and 'simt' not in eng
