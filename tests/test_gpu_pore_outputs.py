"""Pore properties into memory of any kind that the copies reach: fresh and used host
arrays, odd addresses within a page, pinned host memory, memory of the GPU."""
import ctypes as C

import numpy as np
import pytest

from mantiis_gb300 import generate_disks, lib, pore_properties_gpu

pytestmark = pytest.mark.gpu


def call(pore, n, lp, kn):
    # by addresses, past the bindings' array types
    f = lib().mgpu_pore_properties_gpu
    types, f.argtypes = f.argtypes, [C.c_void_p, C.c_int, C.c_double, C.c_double] + [C.c_void_p] * 4
    try:
        return f(pore.ctypes.data, n, 1e-9, 5e-9, lp, kn, None, None)
    finally:
        f.argtypes = types


@pytest.mark.parametrize("where", ["fresh", "used", "offset", "pinned", "gpu"])
@pytest.mark.parametrize("n", [16, 300])
def test_outputs(n, where):
    import torch

    pore = np.ascontiguousarray(generate_disks(n, 2, 9, 0.6, 5))
    want = pore_properties_gpu(pore, 1e-9, 5e-9)
    if where in ("fresh", "used", "offset"):
        off = 3 if where == "offset" else 0
        make = np.empty if where == "fresh" else np.ones
        bufs = [make(n * n + 2 * off) for _ in range(2)]
        outs = [b[off:off + n * n] for b in bufs]
        assert call(pore, n, *(o.ctypes.data for o in outs)) == 0
        for b in bufs:  # nothing around the outputs is written
            assert (b[:off] == 1.0).all() and (b[off + n * n:] == 1.0).all()
    else:
        outs = [torch.ones(n * n, dtype=torch.float64, pin_memory=where == "pinned",
                           device="cuda" if where == "gpu" else "cpu") for _ in range(2)]
        assert call(pore, n, *(o.data_ptr() for o in outs)) == 0
        outs = [o.cpu().numpy() for o in outs]
    for o, w in zip(outs, want):
        assert np.array_equal(o.reshape(n, n), w)
