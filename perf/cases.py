"""The work that a user of this library has it do, as measurable cases.

A case is a dict of plain values.  `task` names the calls a user's program makes for one batch:

  forward     n2d2b_net_forward on device buffers
  host        n2d2b_net_forward_host: blocking, pinned host buffers in and out
  stream      n2d2b_net_submit_host for `batches` batches back to back, then n2d2b_net_wait
  classify    float stimuli on the GPU -> n2d2b_quantize_stimuli -> n2d2b_net_forward -> top-N labels
  scaling     n2d2b_scaling_propagate: a rescale on its own, int32 accumulators to 8 bits
  first_conv  n2d2b_first_conv_noalloc: a first layer for callers that may not allocate

The network tasks run the topologies of the reference's model files (netdesc.py): `model`, the scaling mode
PTQ leaves in it (`scaling`), weight storage (`weight_bits`), clipping, image `size`, `classes`, the `batch`
of the call and the `capacity` the network was finalized for (a ragged last batch is smaller than it).

The network itself (weights, scalings) is a fixed model: it depends on the case, not on the seed.  The seed draws
the stimuli.  Every result is made of whole numbers and has to come out the same to the last bit.
"""
import functools
import math

import numpy as np
import torch

from n2d2_b200 import netdesc, runtime

MODELS = {'mnist24': (1, 24), 'resnet18': (2, 224), 'mobilenet_v1': (3, 224), 'resnet50': (4, 224)}


def _net_case(task, model, batch, scaling, capacity=None, size=None, classes=1000, weight_bits=8, clipped=False, **more):
    return dict(task=task, model=model, scaling=scaling, batch=batch, capacity=capacity or batch, size=size or MODELS[model][1],
                classes=classes, weight_bits=weight_bits, clipped=clipped, **more)


def listed():
    return [dict(c, name=name) for name, c in (
        # the small MNIST network, 64 stimuli a call; four tiny layers, so launches count
        ('mnist24_b64', _net_case('forward', 'mnist24', 64, 'single', classes=10)),
        # one image at a time, as an interactive or control-loop user has it: latency
        ('resnet50_b1', _net_case('forward', 'resnet50', 1, 'double')),
        # the benchmark batch of 1024 split over 8 GPUs: what each of them runs
        ('resnet50_b128', _net_case('forward', 'resnet50', 128, 'double')),
        # BASELINE configuration 4 on one GPU: the benchmark
        ('resnet50_b1024', _net_case('forward', 'resnet50', 1024, 'double')),
        # the benchmark's end-to-end form: batch after batch from pinned host memory, uploads under the forward passes
        ('resnet50_stream_4x256', _net_case('stream', 'resnet50', 256, 'double', batches=4)),
        # fixed-point scaling
        ('resnet18_b128', _net_case('forward', 'resnet18', 128, 'fixed')),
        # floating-point scaling (the scaling mode PTQ leaves unless asked to approximate it), and the ragged last
        # batch of an evaluation run: 100 images on a network finalized for 128
        ('resnet18_float_b100', _net_case('forward', 'resnet18', 100, 'float', capacity=128)),
        # packed 4-bit weights, clipped fixed-point scaling
        ('resnet18_w4_b2048', _net_case('forward', 'resnet18', 2048, 'fixed', weight_bits=4, clipped=True)),
        # depthwise layers, single-shift scaling
        ('mobilenet_b256', _net_case('forward', 'mobilenet_v1', 256, 'single')),
        # a classification service: float stimuli in, the five best classes out, an odd number of requests at once
        ('mobilenet_classify_b33', _net_case('classify', 'mobilenet_v1', 33, 'single', top_n=5)),
        # a Scaling cell run by itself by a host that keeps its own convolutions: 128 images of a 28 x 28 x 128 map
        ('scaling_fixed_28x28x128', dict(task='scaling', scaling='fixed', pixels=128 * 28 * 28, channels=128)),
        # the first layer inside a plugin that owns no device memory: a ResNet stem on eight images
        ('first_conv_b8', dict(task='first_conv', scaling='double', batch=8, size=224, kernel=7, outputs=64)),
    )]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    task = rng.choice(['forward'] * 6 + ['host', 'stream', 'classify', 'classify', 'scaling', 'first_conv'])
    if task == 'scaling':
        # maps of the networks' layers, from one image of a late stage to a large batch of an early one
        channels = rng.choice([16, 24, 32, 64, 96, 128, 150, 256, 512, 1000, 1024, 2048])
        return dict(task='scaling', scaling=rng.choice(['fixed', 'single', 'double', 'float']), channels=channels,
                    pixels=_log_int(rng, 49, 100_000_000 // channels))
    if task == 'first_conv':
        kernel, outputs = rng.choice([(7, 64), (3, 32), (3, 64), (5, 64)])
        size = rng.randrange(96, 257)
        return dict(task='first_conv', scaling=rng.choice(['double', 'single']), batch=_log_int(rng, 1, 96), size=size,
                    kernel=kernel, outputs=outputs)
    model = rng.choice(['mnist24', 'resnet18', 'resnet18', 'resnet50', 'resnet50', 'mobilenet_v1'])
    if model == 'mnist24':
        return _net_case(task, model, _log_int(rng, 1, 4096), rng.choice(['single', 'double', 'fixed', 'float']), classes=10,
                         **_extra(rng, task, 10))
    size = rng.choice([224, 224, rng.randrange(96, 257)])
    classes = rng.choice([1000, 1000, 100, 10])
    # no more images than the benchmark batch, and no more work for a larger image or a heavier way in
    most = int(950 * (224 / size) ** 2 / {'forward': 1, 'host': 2, 'stream': 4, 'classify': 4}[task])
    batch = _log_int(rng, 1, min(most, 1024))
    capacity = batch if rng.random() < 0.7 else min(1024, batch + _log_int(rng, 1, batch + 1))
    weight_bits, clipped = 8, False
    if model == 'resnet18':
        scaling = rng.choice(['fixed', 'fixed', 'float', 'double', 'single'])
        if rng.random() < 0.3:
            weight_bits, scaling = 4, 'fixed'
        clipped = scaling in ('fixed', 'float') and rng.random() < 0.5
    else:
        scaling = rng.choice(['double', 'double', 'single', 'fixed', 'float'] if model == 'resnet50' else ['single', 'double', 'fixed', 'float'])
    return _net_case(task, model, batch, scaling, capacity=capacity, size=size, classes=classes, weight_bits=weight_bits,
                     clipped=clipped, **_extra(rng, task, classes))


def _extra(rng, task, classes):
    if task == 'stream':
        return dict(batches=rng.randrange(2, 5))
    if task == 'classify':
        return dict(top_n=rng.choice([1, 5, min(10, classes)]))
    return {}


@functools.lru_cache(maxsize=3)
def _network(model, scaling, size, classes, weight_bits, clipped):
    seed = MODELS[model][0]
    if model == 'mnist24':
        return netdesc.mnist24(seed=seed, scaling=scaling, calibrate=scaling != 'single')
    if model == 'resnet18':
        return netdesc.resnet18(seed=seed, size=size, scaling=scaling, weight_bits=weight_bits, classes=classes, clipped=clipped)
    if model == 'resnet50':
        return netdesc.resnet50(seed=seed, size=size, scaling=scaling, classes=classes)
    return netdesc.mobilenet_v1(seed=seed, size=size, scaling=scaling, classes=classes)


def _network_of(case):
    return _network(*(case[k] for k in ('model', 'scaling', 'size', 'classes', 'weight_bits', 'clipped')))


def _first_layer(case):
    b = netdesc.NetBuilder('first', 3, case['size'], case['size'], 7, case['scaling'], weight_dist=('normal', 30))
    b.conv(-1, case['outputs'], case['kernel'], stride=2, pad=case['kernel'] // 2, act='relu', name='conv1')
    return b.net


def _scaling_quant(case):
    """Per-channel scalings that bring accumulators of about 20000 down to 8 bits, with a ReLU."""
    rng, n = np.random.default_rng(7), case['channels']
    quant = {'mode': case['scaling'], 'act': 'relu', 'out_bits': 8, 'out_unsigned': True}
    if case['scaling'] == 'fixed':
        quant.update(mode='fixed32', mult=rng.integers(1 << 14, 1 << 15, size=n).astype(np.int32), frac_bits=23)
    elif case['scaling'] == 'single':
        quant['shift0'] = rng.integers(8, 11, size=n).astype(np.uint8)
    elif case['scaling'] == 'double':
        quant['shift0'] = rng.integers(1, 5, size=n).astype(np.uint8)
        quant['shift1'] = (quant['shift0'] + rng.integers(8, 11, size=n)).astype(np.uint8)
    else:
        quant['fscale'] = (rng.uniform(0.7, 1.4, size=n) / 450.0).astype(np.float32)
    return quant


def prepare(case, seed):
    gen = torch.Generator(device='cuda').manual_seed(seed)

    def stimuli(batch, i):
        return torch.randint(0, 256, (batch, i['H'], i['W'], i['C']), dtype=torch.uint8, device='cuda', generator=gen)

    stream = torch.cuda.current_stream().cuda_stream
    state = {'case': case, 'stream': stream}
    if case['task'] == 'scaling':
        n = (case['pixels'], case['channels'])
        state['in'] = (torch.randn(n, device='cuda', generator=gen) * 20000.0).round().to(torch.int32)
        state['out'] = torch.zeros(n, dtype=torch.uint8, device='cuda')
        state['quant'] = _scaling_quant(case)
        return state
    if case['task'] == 'first_conv':
        net = _first_layer(case)
        state['layer'] = net['layers'][0]
        state['in'] = stimuli(case['batch'], net['input'])
        side = netdesc.layer_macs(net)[1][0]
        state['out'] = torch.zeros((case['batch'], side[1], side[2], side[0]), dtype=torch.uint8, device='cuda')
        return state

    net = _network_of(case)
    i, batch = net['input'], case['batch']
    state['net'] = qn = runtime.QuantizedNet(net, case['capacity'])
    out_type = torch.uint8 if qn.out_dtype == np.uint8 else torch.int8
    if case['task'] in ('host', 'stream'):
        n = case.get('batches', 1)
        state['in'] = [stimuli(batch, i).cpu().pin_memory() for _ in range(n)]
        state['out'] = [torch.zeros((batch, qn.out_elems), dtype=out_type).pin_memory() for _ in range(n)]
        return state
    state['out'] = torch.zeros((batch, qn.out_elems), dtype=out_type, device='cuda')
    if case['task'] == 'classify':
        state['float'] = torch.rand((batch, i['C'], i['H'], i['W']), device='cuda', generator=gen)
        state['in'] = torch.zeros((batch, i['H'], i['W'], i['C']), dtype=torch.uint8, device='cuda')
        state['labels'] = torch.zeros((batch, case['top_n']), dtype=torch.int32, device='cuda')
        state['values'] = torch.zeros((batch, case['top_n']), dtype=torch.int32, device='cuda')
    else:
        state['in'] = stimuli(batch, i)
    return state


def run(state):
    case, stream = state['case'], state['stream']
    task = case['task']
    if task == 'forward':
        state['net'].forward_device(state['in'].data_ptr(), case['batch'], state['out'].data_ptr(), stream)
        return state['out']
    if task == 'host':
        state['net'].forward_host_ptr(state['in'][0].data_ptr(), case['batch'], state['out'][0].data_ptr(), stream)
        return state['out']
    if task == 'stream':
        net = state['net']
        for x, y in zip(state['in'], state['out']):
            net.submit_host_ptr(x.data_ptr(), case['batch'], y.data_ptr(), stream)
        net.wait()
        return state['out']
    if task == 'classify':
        net, batch, x = state['net'], case['batch'], state['float']
        runtime.quantize_stimuli(x.data_ptr(), batch, x.shape[1], x.shape[2], x.shape[3], state['in'].data_ptr(), stream=stream)
        net.forward_device(state['in'].data_ptr(), batch, state['out'].data_ptr(), stream)
        net.estimated_labels_topn(batch, case['top_n'], state['labels'].data_ptr(), state['values'].data_ptr(), stream)
        return {'logits': state['out'], 'labels': state['labels'], 'values': state['values']}
    if task == 'scaling':
        runtime.scaling_propagate(state['in'].data_ptr(), state['out'].data_ptr(), case['pixels'], state['quant'], case['channels'],
                                  stream=stream)
        return state['out']
    x = state['in']
    runtime.first_conv_noalloc(x.data_ptr(), x.shape[0], x.shape[1], x.shape[2], x.shape[3], True, state['layer'],
                               state['out'].data_ptr(), stream=stream)
    return state['out']


def work(case):
    """Inputs and weights read once, outputs written once; operations = 2 per multiply-accumulate."""
    if case['task'] == 'scaling':
        n = case['pixels'] * case['channels']
        return {'bytes': 5 * n, 'flops': 2 * n}
    net = _first_layer(case) if case['task'] == 'first_conv' else _network_of(case)
    macs, shapes = netdesc.layer_macs(net)
    last = shapes[len(net['layers']) - 1]
    images = case['batch'] * case.get('batches', 1)
    i = net['input']
    pixels = i['C'] * i['H'] * i['W']
    weights = sum(l['weights'].size * l['weight_bits'] // 8 + 4 * l['Cout'] for l in net['layers'] if 'weights' in l)
    per_image = pixels * (4 if case['task'] == 'classify' else 1) + last[0] * last[1] * last[2] + 8 * case.get('top_n', 0)
    return {'bytes': images * per_image + weights, 'flops': 2 * images * sum(macs)}


def tolerance(case):
    return 'exact'
