"""Stand-alone Scaling::propagate on the GPU (n2d2b_scaling_propagate) against the golden vectors the
reference's own Scaling_Kernels produced, and against the hand-derived known answers."""
import json
import os

import numpy as np
import pytest

from n2d2_b200 import runtime

pytestmark = pytest.mark.gpu

GOLD = np.load(os.path.join(os.path.dirname(__file__), 'golden', 'ref_vectors.npz'))
CASES = [c for c in json.loads(bytes(GOLD['cases']).decode()) if c['kind'] == 'scaling']


def _gpu_scaling(x_nchw, q):
    import torch
    x = np.ascontiguousarray(np.transpose(x_nchw, (0, 2, 3, 1))).astype(np.int32)   # NHWC
    B, H, W, C = x.shape
    d_in = torch.from_numpy(x).cuda()
    d_out = torch.zeros((B, H, W, C), dtype=torch.int8, device='cuda')
    runtime.scaling_propagate(d_in.data_ptr(), d_out.data_ptr(), B * H * W, q, C)
    out = d_out.cpu().numpy()
    out = out.view(np.uint8) if q.get('out_unsigned') else out
    return np.transpose(out.astype(np.int64), (0, 3, 1, 2))


@pytest.mark.parametrize('case', CASES, ids=lambda c: f"{c['mode']}{c['id']}_u{c['unsigned']}_b{c['bits']}")
def test_scaling_matches_reference_vectors(case):
    i = case['id']
    q = {'mode': case['mode'], 'out_bits': case['bits'], 'out_unsigned': bool(case['unsigned']), 'act': 'linear',
         'frac_bits': case['frac_bits'], 'is_clipped': case['is_clipped']}
    for key in ('shift0', 'shift1', 'mult', 'fscale', 'clip'):
        if f'scal{i}_{key}' in GOLD:
            q[key] = GOLD[f'scal{i}_{key}']
    want = GOLD[f"scal{i}_{case['unsigned']}_{case['bits']}_y"].astype(np.int64)
    got = _gpu_scaling(GOLD['scal_x'], q)
    assert np.array_equal(got, want)


def test_scaling_known_answers_on_gpu():
    from test_oracle_golden import KAT
    for q, unsigned, xs, want in KAT:
        q = dict(q, out_bits=8, out_unsigned=unsigned, act='linear')
        x = np.array(xs).reshape(len(xs), 1, 1, 1)
        assert _gpu_scaling(x, q).reshape(-1).tolist() == want


# channel counts whose constants repeat over 1, 2 or 4 pixels, the limits of one launch, several launches; odd pixel counts
@pytest.mark.parametrize('channels,pixels', [(1, 7), (3, 1001), (37, 23), (128, 5000), (150, 33), (150, 64), (1000, 9), (1024, 3),
                                             (1025, 5), (2048, 17), (2500, 2)])
@pytest.mark.parametrize('mode', ['single', 'double', 'fixed32', 'fixed_exact', 'float', 'float_clipped', 'saturation'])
def test_scaling_shapes_and_forms(channels, pixels, mode):
    from oracle import oracle
    rng = np.random.default_rng(channels * 31 + pixels)
    q = {'mode': mode.split('_')[0], 'act': 'relu', 'out_bits': 8, 'out_unsigned': True}
    if mode in ('single', 'saturation'):
        q.update(mode='single', shift0=rng.integers(0, 12, channels).astype(np.uint8))
    elif mode == 'double':
        q.update(shift0=rng.integers(1, 5, channels).astype(np.uint8), shift1=rng.integers(8, 15, channels).astype(np.uint8))
    elif mode.startswith('fixed'):
        # 2^23: the 32-bit form; 2^30: products only the 64-bit one holds
        q.update(mode='fixed32', mult=rng.integers(1 << 14, 1 << 15, channels).astype(np.int32), frac_bits=23 if mode == 'fixed32' else 30)
    else:
        q['fscale'] = (rng.uniform(0.5, 2.0, channels) / 300.0).astype(np.float32)
        if mode == 'float_clipped':
            q.update(is_clipped=True, clip=(rng.uniform(-1.0, 3.0, channels) * 20000.0).astype(np.float32), act='linear', out_unsigned=False)
    if mode == 'saturation':
        q.update(act='saturation', sat_thr=5, out_unsigned=False)
    x = np.rint(rng.normal(0.0, 20000.0, (1, channels, 1, pixels)) * rng.choice([1.0, 1.0, 1e4], (1, channels, 1, pixels)))
    x.reshape(-1)[:3] = [-2.0 ** 31, 2.0 ** 31 - 1, 0][:x.size]
    x = x.astype(np.int64)
    assert np.array_equal(_gpu_scaling(x, q), np.asarray(oracle.scaling(x, q, 'i64')).astype(np.int64))
