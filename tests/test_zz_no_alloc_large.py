"""mqb_apply_static on a register that keeps a schedule of its own for it (complex64, 24 qubits), against mqb_apply.

Tolerance of the smaller registers' test: a few hundred gates of 6e-8 each on amplitudes of a random unit vector.
"""
import ctypes

import numpy as np
import pytest
import torch

from mindquantum_b200 import _native as N
from mindquantum_b200.simulator import lowering
from reference_circuits import hea_circuit


@pytest.mark.gpu
def test_static_schedule_matches_the_generated_one():
    n = 24
    circ = hea_circuit(n, 3)
    prog = lowering.Program(circ, n, N.MQB_PREC_C64, circ.params_name)
    p = torch.as_tensor(np.random.default_rng(2).uniform(0, 2 * np.pi, (1, len(circ.params_name))), device='cuda')
    got = torch.randn(1, 1 << n, dtype=torch.complex64, device='cuda', generator=torch.Generator('cuda').manual_seed(1))
    got /= got.abs().pow(2).sum().sqrt()
    ref = got.clone()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    size = ctypes.c_size_t()
    N.call('mqb_apply_workspace_size', prog.handle, 1, ctypes.byref(size))
    ws = torch.empty(size.value, dtype=torch.uint8, device='cuda')
    N.call('mqb_apply', prog.handle, ptr(ref), 1, ptr(p), p.shape[1], None, ptr(ws), size.value, stream)
    N.call('mqb_apply_static', prog.handle, ptr(got), 1, ptr(p), p.shape[1], None, stream)
    torch.cuda.synchronize()
    assert (got - ref).abs().max().item() <= 1e-6
