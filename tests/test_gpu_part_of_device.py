"""Streams of a green context, whose kernels have a part of the device's SMs: every
engine steps there, to the same bits as on the whole device."""
import ctypes as C

import numpy as np
import pytest

from mantiis_gb300 import SIM_ADSORPTION, Batch, Solver, default_params, generate_disks

pytestmark = pytest.mark.gpu

SM_RESOURCE, DEFAULT_STREAM, NON_BLOCKING = 1, 1, 1  # cuda.h


@pytest.fixture(scope="module")
def part():
    """A stream of a green context of about half of the device."""
    import torch

    torch.zeros(1, device="cuda")  # the primary context
    cu = C.CDLL("libcuda.so.1")
    if not hasattr(cu, "cuGreenCtxStreamCreate"):
        pytest.skip("no green contexts in this driver")
    # CUdevResource is 144 bytes; room for more
    whole, first, rest = (C.create_string_buffer(512) for _ in range(3))
    desc, green, stream, n = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_uint(1)
    half = torch.cuda.get_device_properties(0).multi_processor_count // 2
    for rc in (cu.cuDeviceGetDevResource(0, whole, SM_RESOURCE),
               cu.cuDevSmResourceSplitByCount(first, C.byref(n), whole, rest, 0, half),
               cu.cuDevResourceGenerateDesc(C.byref(desc), first, 1),
               cu.cuGreenCtxCreate(C.byref(green), desc, 0, DEFAULT_STREAM),
               cu.cuGreenCtxStreamCreate(C.byref(stream), green, NON_BLOCKING, 0)):
        if rc != 0:
            pytest.skip(f"green contexts: CUDA error {rc}")
    yield stream.value
    torch.cuda.synchronize()
    cu.cuStreamDestroy_v2(stream)
    cu.cuGreenCtxDestroy(green)


def solver(n=128, levels=1, **kw):
    pore = generate_disks(n, 4, 10, 0.65, 3, open_x_edges=True)
    p = default_params(tol=0.0, multiblock=int(levels > 1), max_allowed_level=2, edge_fine=int(levels > 1), **kw)
    return Solver(pore, np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0), p)


@pytest.mark.parametrize("n,levels,sim", [(128, 1, 0), (128, 2, 0), (300, 1, SIM_ADSORPTION)])
def test_context(part, n, levels, sim):
    out, launches = [], []
    for stream in (None, part):
        s = solver(n, levels, simulation=sim)
        if stream:
            s.set_stream(stream)
        assert s.run(20) == 20
        s.advance_graph(21)
        s.advance(3)
        s.sync()
        launches.append(s.launches)
        out.append(s.cells(with_f=True)["f"])
        s.set_stream(0)
        s.advance_graph(4)
        s.close()
    assert np.isfinite(out[0]).all() and np.array_equal(*out)
    assert sim or launches[1] > launches[0]  # launches per phase in the part


def test_batch(part):
    out = []
    for stream in (None, part):
        ss = [solver(n) for n in (64, 128, 100)]
        b = Batch(ss)
        if stream:
            b.set_stream(stream)
        b.advance(21)
        b.sync()
        out.append([s.cells(with_f=True)["f"] for s in ss])
        b.close()
    assert all(np.array_equal(x, y) for x, y in zip(*out))
