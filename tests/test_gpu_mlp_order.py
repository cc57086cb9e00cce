"""A network call writes its output array in the order of the handle's stream: a copy out of the array
that was queued before the call reads what the array held then.  The stream is kept busy for some
milliseconds, so that the call is made, and its host side done, while the copy still waits.
"""
import ctypes as C

import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def test_queued_copy_of_the_output_array(mps_lib):
    import torch
    from polymps_gb300 import mps
    n = 65537
    rng = np.random.default_rng(4)
    norm = np.concatenate([np.zeros(16), np.ones(16), [0.0, 1.0]]).astype(np.float32)
    with mps.MpsGpu(cases.config(3, scale=8.0)) as g:
        g.mlp_set_weights((0.2 * rng.standard_normal(abi.MLP_NPARAM)).astype(np.float32), norm)
        f = rng.standard_normal((n, abi.MLP_NFEAT)).astype(np.float32)
        want = g.mlp_forward(f)
        out = torch.ones(n, dtype=torch.float32).pin_memory()
        dev = torch.zeros(n, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        raw = C.c_void_p()
        assert mps.lib().mpsgpu_stream(g.h, C.byref(raw)) == 0
        stream = torch.cuda.ExternalStream(raw.value)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)   # about 10 ms
            dev.copy_(out, non_blocking=True)
        assert mps.lib().mpsgpu_mlp_forward(g.h, abi.fptr(f), n, abi.fptr(out.numpy())) == 0
        torch.cuda.synchronize()
        copied, result = dev.cpu(), out.numpy().copy()
        del out, dev   # their allocator notes the stream when they are freed: before the handle goes
    assert torch.equal(copied, torch.ones(n))
    assert np.array_equal(result, want)
