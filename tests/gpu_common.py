"""Helpers shared by the GPU parity tests: run a network description through the C ABI and compare
every readable tensor with the CPU oracle, bit for bit."""
import ctypes

import numpy as np

from n2d2_b200 import netdesc, runtime
from oracle import oracle

KEEP = runtime.KEEP_ALL_OUTPUTS | runtime.NO_FUSION


def single_conv_net(C, H, W, O, k, stride=1, pad=0, in_unsigned=True, act='relu', mode='single', seed=7, dil=1,
                    groups=1, bias=True, **builder_kw):
    b = netdesc.NetBuilder('single', C, H, W, seed, mode, input_unsigned=in_unsigned, weight_dist=('normal', 30),
                           **builder_kw)
    b.conv(-1, O, k, stride=stride, pad=pad, act=act, dil=dil, groups=groups, bias=bias, name='c')
    return b.net


class _KernelNode(ctypes.Structure):   # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [('func', ctypes.c_void_p), ('sizes', ctypes.c_uint * 7), ('params', ctypes.c_void_p), ('extra', ctypes.c_void_p),
                ('kern', ctypes.c_void_p), ('ctx', ctypes.c_void_p)]


def kernels_of(qn, batch):
    """Names of the kernels that a forward pass of `batch` images launches: the nodes of its captured graph."""
    import torch
    i = qn.desc['input']
    x = torch.zeros((batch, i['H'], i['W'], i['C']), dtype=torch.uint8, device='cuda')
    y = torch.zeros((batch, qn.out_elems * np.dtype(qn.out_dtype).itemsize), dtype=torch.uint8, device='cuda')
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    cuda = ctypes.CDLL('libcuda.so.1')

    def call(name, *args):
        rc = getattr(cuda, name)(*args)
        assert rc == 0, f'{name}: {rc}'

    graph, count = ctypes.c_void_p(), ctypes.c_size_t()
    call('cuStreamBeginCapture_v2', ctypes.c_void_p(stream.cuda_stream), 1)   # thread-local
    qn.forward_device(x.data_ptr(), batch, y.data_ptr(), stream.cuda_stream)
    call('cuStreamEndCapture', ctypes.c_void_p(stream.cuda_stream), ctypes.byref(graph))
    call('cuGraphGetNodes', graph, None, ctypes.byref(count))
    nodes = (ctypes.c_void_p * count.value)()
    call('cuGraphGetNodes', graph, nodes, ctypes.byref(count))
    names = []
    for node in nodes:
        kind, params, name = ctypes.c_int(), _KernelNode(), ctypes.c_char_p()
        call('cuGraphNodeGetType', ctypes.c_void_p(node), ctypes.byref(kind))
        if kind.value == 0:   # a kernel
            call('cuGraphKernelNodeGetParams_v2', ctypes.c_void_p(node), ctypes.byref(params))
            call('cuFuncGetName', ctypes.byref(name), ctypes.c_void_p(params.func))
            names.append(name.value.decode())
    call('cuGraphDestroy', graph)
    return names


def kernels_of_host_call(qn, x):
    """The output of a call on host buffers and the names of the kernels that ran for it."""
    import torch
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out = qn.forward_host(x)
        torch.cuda.synchronize()
    return out, [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]


def compare_net(net, batch, flags=KEEP, flavour='i64', x=None, want_engine=None, slices=0, ref=None, kernels=False):
    """Returns (number of compared layers, engines), or with `kernels` the kernels that ran. Asserts bit-exact equality with the
    oracle."""
    if x is None:
        x = netdesc.make_input(net, batch)
    if ref is None:
        ref = oracle.run_net(net, x, flavour)
    qn = runtime.QuantizedNet(net, max(batch, 1), flags=flags)
    try:
        if slices:
            qn.set_slices(slices)
        out = qn.forward_host(x)
        eng = qn.engines()
        if want_engine is not None:
            wanted = (want_engine,) if isinstance(want_engine, str) else tuple(want_engine)
            assert any(w in eng for w in wanted), f'expected a {wanted} cell, got {sorted(set(eng))}'
        n = 0
        last = len(net['layers']) - 1
        assert np.array_equal(out.astype(np.int64), ref[last].reshape(batch, -1)), 'final output differs'
        for i, l in enumerate(net['layers']):
            if not qn.tensor_info(qn.tensor_of_layer[i]).readable:
                continue
            got = qn.read_layer(i, batch).astype(np.int64)
            bad = int((got != ref[i]).sum())
            assert bad == 0, f"layer {i} {l['name']} ({eng[i]}): {bad} of {ref[i].size} values differ"
            n += 1
        return kernels_of(qn, batch) if kernels else (n, eng)
    finally:
        qn.close()
