"""The backward pass where the segment's intermediates do not fit (the stage by
stage reverse), that each pass decides by the memory there is then, that a tape
may take what a pass kept, and traces of more than 2^31 values."""
import ctypes

import numpy as np
import pytest

from swe_fvm_gb300 import _lib, scenarios
from swe_fvm_gb300.adjoint import Rollout

pytestmark = pytest.mark.gpu


def backward(ro, prim, gauges, segment):
    """Gradients of one pass, and the launches it took (nothing is replayed: no segment is full)."""
    ro.sd.SetVolField(prim)
    ro.sd.prime()
    tr = ro.forward(1, 6, segment, gauges, 2)
    n = ro.sd.launch_count()
    g = ro.backward(np.cos(np.arange(tr.size)).reshape(tr.shape))
    return g, ro.sd.launch_count() - n


def alike(a, b):
    # (node sums are atomic: their order varies by rounding)
    return all(np.allclose(x, y, rtol=1e-9, atol=1e-11 * np.abs(y).max()) for x, y in zip(a, b))


def test_each_pass_decides_by_the_memory_there_is(gpu):
    import torch

    m, prim = scenarios.sloped_bump_case(101, 3)
    gauges = np.random.default_rng(0).integers(0, m.num_cells, 5)
    C, ns = m.num_cells, 2
    # a segment whose stage inputs (24 B a cell) are under the 1 GiB that is kept
    # between passes and whose intermediates (about 290 B a cell) are not
    segment = int(0.9 * 2 ** 30 / (24 * C * ns))
    base, plain = Rollout(m, prim), Rollout(m, prim)
    want, n_kept = backward(plain, prim, gauges, segment)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    leave = 16 << 30  # most of the device stands for other programs' data; untouched, and far from all of it
    hold = torch.empty(max(free - leave, 1), dtype=torch.uint8, device="cuda")
    got, n_staged = backward(base, prim, gauges, segment)
    assert alike(got, want)
    assert n_staged != n_kept
    del hold
    torch.cuda.empty_cache()
    got, n = backward(base, prim, gauges, segment)
    assert n == n_kept
    assert alike(got, want)


def test_large_traces(gpu):
    """More trace values than an int counts, and a tape that fits beside the rest
    only without the workspace that a backward pass kept."""
    import torch

    m, prim = scenarios.sloped_bump_case(101, 3)
    L = _lib.load()
    n_gauges, n_obs, last = 1 << 27, 17, 7777
    cells = np.arange(n_gauges, dtype=np.int64) % m.num_cells
    cells[-1] = last
    ro, small = Rollout(m, prim), Rollout(m, prim)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ro.backward(np.ones_like(ro.forward(1, 40, 20, cells[:4], 10)))
    ro.sd.SetVolField(prim)
    ro.sd.prime()
    torch.cuda.synchronize()
    kept = free - torch.cuda.mem_get_info()[0]
    assert 2 ** 28 < kept < 2 ** 30
    traces = torch.empty((n_obs, n_gauges), dtype=torch.float64, device="cuda")
    tape = traces.numel() * 8 + n_gauges * 4
    hold = torch.empty(max(torch.cuda.mem_get_info()[0] - tape + kept // 2, 1), dtype=torch.uint8, device="cuda")
    ro.sd._check(L.swe_adjoint_forward_device(ro.sd.ctx, 1, n_obs, 4, n_gauges, cells.ctypes.data, 1,
                                              ctypes.c_void_p(traces.data_ptr())))
    del hold
    torch.cuda.empty_cache()
    want = small.forward(1, n_obs, 4, np.array([last]), 1)
    assert np.array_equal(traces[:, -1].cpu().numpy(), want[:, 0])
    weights = np.cos(np.arange(n_obs))
    grads = traces.zero_()
    grads[:, -1] = torch.as_tensor(weights, device="cuda")
    torch.cuda.synchronize()
    gp = torch.empty((m.num_cells, 3), dtype=torch.float64, device="cuda")
    gz = torch.empty((m.num_nodes,), dtype=torch.float64, device="cuda")
    ro.sd._check(L.swe_adjoint_backward_device(ro.sd.ctx, ctypes.c_void_p(grads.data_ptr()),
                                               ctypes.c_void_p(gp.data_ptr()), ctypes.c_void_p(gz.data_ptr())))
    ro.sd.synchronize()
    assert alike((gp.cpu().numpy(), gz.cpu().numpy()), small.backward(weights[:, None]))
