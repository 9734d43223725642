"""The network's passes over activations: pooling, upsampling and adjoints at
even, odd and unaligned sizes, the passes fused into convolutions and adjoints,
and the parameter lists, against the plain torch expression of each.  Each
result is one rounded sum in a fixed order or a selection, so they are equal
bit for bit; the convolution inside a fused call is that of the plain call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tensors(*shapes, seed=0, offset=0):
    """Normal tensors; `offset` floats after an aligned address."""
    import torch

    rng = np.random.default_rng(seed)
    out = []
    for s in shapes:
        flat = torch.zeros(offset + int(np.prod(s)), device="cuda")
        flat[offset:] = torch.tensor(rng.standard_normal(int(np.prod(s))).astype(np.float32), device="cuda")
        out.append(flat[offset:].view(*s))
    return out


def block_sum(f):
    return ((f[..., ::2, ::2] + f[..., ::2, 1::2]) + f[..., 1::2, ::2]) + f[..., 1::2, 1::2]


def repeat(c):
    return c.repeat_interleave(2, -1).repeat_interleave(2, -2)


# planes, coarse height and width, floats off the aligned address
SIZES = [(1, 1, 1, 0), (3, 5, 2, 0), (2, 3, 7, 0), (4, 8, 16, 0), (6, 9, 128, 0), (3, 4, 6, 1), (2, 8, 8, 2), (5, 33, 20, 0)]


@pytest.mark.parametrize("nc, h, w, offset", SIZES)
def test_pool_and_upsample(nc, h, w, offset):
    import torch

    from mantiis_gb300 import surrogate as S

    L, st, ptr = S.cnn_lib(), S._stream(), S._ptr
    coarse, relu_c, fine, relu_f, grad = tensors((nc, h, w), (nc, h, w), (nc, 2 * h, 2 * w), (nc, 2 * h, 2 * w),
                                                 (nc, 2 * h, 2 * w), seed=nc + h + w, offset=offset)
    zero = torch.zeros((), device="cuda")

    def out(like):
        return torch.full_like(like, float("nan"))

    y = out(coarse)
    assert L.cnn_avgpool2_forward(ptr(fine), ptr(y), nc, 2 * h, 2 * w, st) == 0
    assert torch.equal(y, 0.25 * block_sum(fine))
    y = out(fine)
    assert L.cnn_avgpool2_backward(ptr(coarse), ptr(y), nc, 2 * h, 2 * w, st) == 0
    assert torch.equal(y, 0.25 * repeat(coarse))
    y = grad.clone()
    assert L.cnn_avgpool2_backward_add_relu(ptr(coarse), ptr(relu_f), ptr(y), nc, 2 * h, 2 * w, st) == 0
    assert torch.equal(y, torch.where(relu_f > 0, grad + 0.25 * repeat(coarse), zero))
    y = out(fine)
    assert L.cnn_upsample2_forward(ptr(coarse), ptr(y), nc, h, w, st) == 0
    assert torch.equal(y, repeat(coarse))
    y, m, m2 = out(coarse), out(coarse), out(coarse)
    assert L.cnn_upsample2_backward(ptr(fine), ptr(y), nc, h, w, st) == 0
    assert torch.equal(y, block_sum(fine))
    y = out(coarse)
    assert L.cnn_upsample2_backward_relu(ptr(fine), ptr(y), ptr(relu_c), ptr(m), nc, h, w, st) == 0
    assert L.cnn_upsample2_backward_relu(ptr(fine), None, ptr(relu_c), ptr(m2), nc, h, w, st) == 0
    masked = torch.where(relu_c > 0, block_sum(fine), zero)
    assert torch.equal(y, block_sum(fine)) and torch.equal(m, masked) and torch.equal(m2, masked)


@pytest.mark.parametrize("n, cin, cout, h, w, offset", [(1, 2, 3, 5, 7, 0), (2, 9, 17, 8, 8, 0), (1, 40, 33, 18, 20, 1),
                                                        (3, 32, 32, 64, 64, 0), (8, 64, 64, 8, 8, 0)])
def test_fused_convolutions(n, cin, cout, h, w, offset):
    import torch

    from mantiis_gb300 import surrogate as S

    layer = S.Conv3x3(cin, cout, np.random.default_rng(3))
    x, act, dy, skip = tensors((n, cin, h, w), (n, cin, h, w), (n, cout, h, w), (n, cout, h, w), seed=h, offset=offset)
    plain = layer.forward(x, True)
    y, d = layer.forward(x, True, skip=skip)
    none, d2 = layer.forward(x, True, skip=skip, keep=False)
    assert none is None and torch.equal(y, plain) and torch.equal(d, plain + skip) and torch.equal(d2, d)
    dx = layer.backward(x, dy)
    y, m = layer.backward(x, dy, relu=act)
    none, m2 = layer.backward(x, dy, relu=act, keep=False)
    assert none is None and torch.equal(y, dx) and torch.equal(m2, m)
    assert torch.equal(m, torch.where(act > 0, dx, torch.zeros((), device="cuda")))
    with pytest.raises(ValueError):
        layer.forward(x, True, skip=skip[..., :-1].contiguous())
    with pytest.raises(ValueError):
        layer.backward(x, dy, relu=act[..., :-1].contiguous())


@pytest.mark.parametrize("count", [1, 31, 32, 33, 70])
def test_parameter_lists(count):
    """Lists around the 32 tensors of a launch, sizes around a block of 256."""
    import torch

    from mantiis_gb300 import surrogate as S

    L, st, ptr = S.cnn_lib(), S._stream(), S._ptr
    sizes = [(1, 255, 256, 257, 1000)[k % 5] for k in range(count)]
    sets = [tensors(*[(s,)] * 4, seed=k) for k, s in enumerate(sizes)]
    for t in sets:
        t[3].abs_()
    lists = [[t.clone() for t in s] for s in sets]
    w16 = [torch.zeros(s, dtype=torch.int16, device="cuda") if k % 2 else None for k, s in enumerate(sizes)]
    v16 = [None if t is None else t.clone() for t in w16]
    array = (S._Tensor * count)(*[(*map(ptr, s), ptr(h), s[0].numel()) for s, h in zip(lists, w16)])
    assert L.cnn_adam_many(array, count, 1e-2, 0.9, 0.999, 1e-8, 3, st) == 0
    assert L.cnn_adam_many(array, count, 1e-2, 0.9, 0.999, 1e-8, 0, st) == -1
    for s, l, a, b in zip(sets, lists, v16, w16):
        assert L.cnn_adam(*map(ptr, s), ptr(a), s[0].numel(), 1e-2, 0.9, 0.999, 1e-8, 3, st) == 0
        assert all(torch.equal(p, q) for p, q in zip(s, l)) and (a is None or torch.equal(a, b))
    assert L.cnn_zero_grad_many(array, count, st) == 0
    for s, l in zip(sets, lists):
        assert not l[1].any() and all(torch.equal(s[k], l[k]) for k in (0, 2, 3))
