"""Top-N of 8-bit scores around the class counts at which the kernel changes, against the oracle (whole numbers: no tolerance)."""
import numpy as np
import pytest

from gpu_common import single_conv_net
from n2d2_b200 import netdesc, runtime
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('classes', [128, 129, 256, 257, 512, 513, 1000, 1024, 1025])
@pytest.mark.parametrize('act', ['linear', 'relu'])
def test_class_counts(classes, act):
    net = single_conv_net(16, 5, 4, classes, 1, mode='single', act=act)
    batch, top_n = 3, 7
    x = netdesc.make_input(net, batch)
    ref = oracle.run_net(net, x, 'i64')[-1]
    want_l, want_v = oracle.estimated_labels_topn(ref.reshape(-1, classes), top_n)
    qn = runtime.QuantizedNet(net, batch)
    try:
        qn.forward_host(x)
        labels, values = (a.transpose(0, 2, 3, 1).reshape(-1, top_n) for a in qn.estimated_labels_topn_host(batch, top_n))
        assert np.array_equal(values, want_v) and np.array_equal(labels, want_l)
    finally:
        qn.close()
