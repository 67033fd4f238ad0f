"""Streamed 3x3 layers of 128 channels: the patch kernel and, in calls of up to a tile per SM, the implicit GEMM on the same weights.  Whole numbers against the
oracle: no tolerance."""
import numpy as np
import pytest

from gpu_common import kernels_of
from n2d2_b200 import netdesc, runtime
from oracle import oracle

pytestmark = pytest.mark.gpu


# (H, W, outputs): 96 outputs leave a part of a tile; batches on both sides of the line of a tile of 128 rows per multiprocessor
@pytest.mark.parametrize('case', [(28, 28, 128), (13, 9, 96), (30, 31, 128)], ids=lambda c: '%dx%d_O%d' % c)
@pytest.mark.parametrize('mode', ['double', 'fixed', 'float'])
def test_both_kernels_on_one_network(case, mode):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    H, W, O = case
    b = netdesc.NetBuilder('patch', 16, H, W, 17, mode, weight_dist=('normal', 30))
    b.conv(b.conv(-1, 128, 1, name='front'), O, 3, pad=1, name='c')
    net = b.net
    line = sms * 128 // (H * W)   # images of one tile per multiprocessor
    capacity = min(line + 20, 200)
    x = netdesc.make_input(net, capacity)
    picks = sorted({0, 1, capacity // 2, capacity - 1})
    want = oracle.run_net(net, x[picks], 'i64')[-1].reshape(len(picks), -1)
    qn = runtime.QuantizedNet(net, capacity)
    try:
        whole = qn.forward_host(x)
        assert np.array_equal(whole[picks].astype(np.int64), want)
        for batch in (1, 2, min(line, capacity), capacity):
            assert np.array_equal(qn.forward_host(x[:batch]), whole[:batch])
        if line < capacity:
            assert any('patch_conv' in k for k in kernels_of(qn, capacity)) and not any('patch_conv' in k for k in kernels_of(qn, 2))
    finally:
        qn.close()
