"""The first-layer convolution entry point that allocates no device memory
(n2d2b_first_conv_noalloc).

Who needs it: code that runs where cudaMalloc is off limits - a plugin inside a framework that owns
the device heap, a latency-bound loop that cannot take an allocation's device-wide synchronisation,
a process at its memory budget.  Its scratch is a fixed array inside the library, so the batch is
bounded and calls share state; this file checks that it returns exactly what the regular,
allocating path returns, on two calls in a row with different layers and inputs (the second call
must not see anything of the first), and that oversize requests are refused.

Collected last on purpose: if it fails, every other test has already run.
"""
import numpy as np
import pytest

from n2d2_b200 import netdesc, runtime
from oracle import oracle

from gpu_common import single_conv_net

pytestmark = pytest.mark.gpu


def _both_paths(net, batch, seed):
    import torch
    layer = net['layers'][0]
    i = net['input']
    x = netdesc.make_input(net, batch, seed=seed)
    # the existing entry points: a one-cell network, finalized (allocates), run on host buffers
    qn = runtime.QuantizedNet(net, batch)
    assert qn.engines() == ['stem-tcgen05']
    want = qn.forward_host(x)
    qn.close()
    # the allocation-free entry point on caller-owned device buffers
    d_in = torch.from_numpy(x.view(np.uint8)).cuda()
    d_out = torch.full((batch, want.shape[1]), 0x5A, dtype=torch.uint8, device='cuda')
    torch.cuda.synchronize()
    runtime.first_conv_noalloc(d_in.data_ptr(), batch, i['H'], i['W'], i['C'], i['unsigned'], layer, d_out.data_ptr())
    torch.cuda.synchronize()
    got = d_out.cpu().numpy().view(want.dtype)
    # both against the CPU restatement of the reference as well, not only against each other
    ref = oracle.run_net(net, x, 'i64')[-1].reshape(batch, -1)
    assert np.array_equal(want.astype(np.int64), ref), 'the allocating path differs from the oracle'
    assert np.array_equal(got.astype(np.int64), ref), 'the allocation-free entry point differs from the oracle'
    return got, want


def test_noalloc_first_conv_matches_the_allocating_path_twice_in_a_row():
    # call 1: a ResNet-style stem (3 channels, 7x7 stride 2, unsigned output after ReLU)
    net1 = single_conv_net(3, 64, 64, 64, 7, 2, 3, in_unsigned=True, mode='double', seed=21)
    got, want = _both_paths(net1, 4, seed=5)
    assert np.array_equal(got, want)          # integer path: bit-exact, no tolerance
    # call 2, straight after: other geometry, channel count, signedness, scaling mode and a smaller
    # output - anything left over from call 1 in the shared scratch would show
    net2 = single_conv_net(4, 19, 23, 32, 3, 1, 1, in_unsigned=False, act='linear', mode='single', seed=22)
    got, want = _both_paths(net2, 3, seed=6)
    assert np.array_equal(got, want)
    # and the first layer again, to make sure call 2 left nothing behind either
    got, want = _both_paths(net1, 2, seed=7)
    assert np.array_equal(got, want)


def test_noalloc_first_conv_rejects_what_it_cannot_hold():
    import torch
    net = single_conv_net(3, 64, 64, 64, 7, 2, 3, mode='double')
    layer = net['layers'][0]
    d = torch.zeros(16, dtype=torch.uint8, device='cuda')
    too_many = runtime.NOALLOC_MAX_PIXELS // (64 * 64) + 1
    with pytest.raises(runtime.N2D2BError, match='exceeds the fixed scratch'):
        runtime.first_conv_noalloc(d.data_ptr(), too_many, 64, 64, 3, True, layer, d.data_ptr())
    wide = single_conv_net(16, 16, 16, 64, 3, 1, 1, mode='double')['layers'][0]
    with pytest.raises(runtime.N2D2BError, match='first-layer kernel'):
        runtime.first_conv_noalloc(d.data_ptr(), 1, 16, 16, 16, True, wide, d.data_ptr())


# stride 2 and stride 1: both forms of the layer refuse an output they cannot store to, and the next call runs
@pytest.mark.parametrize('stride', [2, 1])
def test_noalloc_first_conv_refuses_a_misaligned_output(stride):
    import torch
    net = single_conv_net(3, 30, 28, 64, 3, stride, 1, mode='double', seed=23)
    out = torch.zeros(2 * 30 * 28 * 64 + 16, dtype=torch.uint8, device='cuda')
    x = torch.zeros(2 * 30 * 28 * 3, dtype=torch.uint8, device='cuda')
    for shift in (1, 4, 8):
        with pytest.raises(runtime.N2D2BError, match='16-byte aligned'):
            runtime.first_conv_noalloc(x.data_ptr(), 2, 30, 28, 3, True, net['layers'][0], out.data_ptr() + shift)
    got, want = _both_paths(net, 2, seed=8)
    assert np.array_equal(got, want)


# (C, H, W, O, k, stride, pad, batch): the space-to-depth form with its layer as kernel parameters (whole words per row and not, 32 to
# 128 outputs, the widest filters) and, for what does not fit it (wide rows, weights beyond the parameters), the copied form
NOALLOC_CASES = [(3, 224, 224, 64, 7, 2, 3, 3), (3, 97, 99, 32, 3, 2, 1, 5), (1, 40, 44, 96, 5, 2, 2, 2), (4, 64, 60, 128, 7, 2, 3, 2),
                 (4, 33, 30, 128, 8, 2, 3, 1), (3, 254, 256, 64, 7, 2, 3, 2), (3, 30, 28, 64, 3, 1, 1, 2)]


@pytest.mark.parametrize('case', NOALLOC_CASES, ids=lambda c: 'C%d_%dx%d_O%d_k%d_s%d_p%d_b%d' % c)
@pytest.mark.parametrize('mode', ['double', 'single'])
def test_noalloc_first_conv_forms(case, mode):
    C, H, W, O, k, s, p, batch = case
    got, want = _both_paths(single_conv_net(C, H, W, O, k, s, p, mode=mode, seed=23), batch, seed=8)
    assert np.array_equal(got, want)


def test_noalloc_first_conv_takes_an_input_at_any_address():
    import torch
    for C, stride in ((4, 2), (4, 1), (3, 2)):
        net = single_conv_net(C, 32, 32, 64, 3, stride, 1, mode='double', seed=25)
        x = netdesc.make_input(net, 2, seed=8)
        want = oracle.run_net(net, x, 'i64')[-1]
        room = torch.zeros(x.size + 16, dtype=torch.uint8, device='cuda')
        out = torch.empty(want.size, dtype=torch.uint8, device='cuda')
        for shift in (1, 2, 4, 0):
            room[shift:shift + x.size] = torch.from_numpy(x.view(np.uint8).reshape(-1)).cuda()
            runtime.first_conv_noalloc(room.data_ptr() + shift, 2, 32, 32, C, True, net['layers'][0], out.data_ptr())
            assert np.array_equal(out.cpu().numpy().astype(np.int64), want.reshape(-1))


# A bounded wait that runs out in one call's kernels (here in a one-CTA kernel that raises the same status word) is reported by the next
# call, which launches nothing; the call after it runs.
@pytest.mark.parametrize('stride', [2, 1])
def test_noalloc_first_conv_reports_a_wait_that_ran_out(stride):
    import torch
    net = single_conv_net(3, 30, 28, 64, 3, stride, 1, mode='double', seed=23)
    _both_paths(net, 2, seed=8)
    out = torch.full((2 * 30 * 28 * 64,), 0x5A, dtype=torch.uint8, device='cuda')
    x = torch.zeros(2 * 30 * 28 * 3, dtype=torch.uint8, device='cuda')
    for stream in (0, torch.cuda.Stream().cuda_stream):
        torch.cuda.synchronize()
        runtime.first_conv_noalloc_selftest_wait_timeout(1000, stream=stream)
        with pytest.raises(runtime.N2D2BError, match='status -4.*gave up waiting'):
            runtime.first_conv_noalloc(x.data_ptr(), 2, 30, 28, 3, True, net['layers'][0], out.data_ptr(), stream=stream)
        torch.cuda.synchronize()
        assert bool((out == 0x5A).all())
        got, want = _both_paths(net, 2, seed=9)
        assert np.array_equal(got, want)
    for limit in (0, 100001):
        with pytest.raises(runtime.N2D2BError, match='limit_us'):
            runtime.first_conv_noalloc_selftest_wait_timeout(limit)
