"""The last cell writes the caller's output buffer and the network's own tensor: padded and unpadded columns, calls that store from the registers and calls that
do not, output buffers at any address.  Whole numbers against the oracle: no tolerance."""
import numpy as np
import pytest

from n2d2_b200 import netdesc, runtime
from oracle import oracle

pytestmark = pytest.mark.gpu


def classifier(outputs, weight_bits=8):
    b = netdesc.NetBuilder('classifier', 64, 1, 1, 13, 'fixed', weight_dist=('normal', 30) if weight_bits == 8 else ('uniform', 7), weight_bits=weight_bits)
    x = b.conv(-1, 2048, 1, name='features')
    b.fc(x, outputs, act='linear', name='fc')
    return b.net


# (classes, capacity, weight bits): the last one has more than two tiles per SM at its capacity
@pytest.mark.parametrize('case', [(1000, 300, 8), (104, 40, 8), (100, 300, 8), (10, 5, 8), (64, 130, 8), (1000, 200, 4), (2048, 6000, 8)], ids=lambda c: 'O%d_b%d_w%d' % c)
def test_last_cell_writes_both_outputs(case):
    import torch
    outputs, capacity, bits = case
    net = classifier(outputs, bits)
    data = netdesc.make_input(net, capacity)
    want = oracle.run_net(net, data, 'i64')[-1].reshape(capacity, -1)
    qn = runtime.QuantizedNet(net, capacity)
    try:
        for batch in sorted({1, min(129, capacity), capacity}):
            x = torch.from_numpy(data[:batch].view(np.uint8)).cuda()
            n = batch * outputs
            for shift in (0, 1, 4, 8):
                room = torch.full((n + 64,), 0x5a, dtype=torch.uint8, device='cuda')
                qn.forward_device(x.data_ptr(), batch, room.data_ptr() + shift)
                qn.check()
                got = room.cpu().numpy()
                assert np.array_equal(got[shift:shift + n].view(qn.out_dtype).astype(np.int64).reshape(batch, -1), want[:batch]), (batch, shift)
                assert (got[:shift] == 0x5a).all() and (got[shift + n:] == 0x5a).all()
            assert np.array_equal(qn.read_layer(len(net['layers']) - 1, batch).astype(np.int64).reshape(batch, -1), want[:batch])
    finally:
        qn.close()
