"""The FP32 3x3 convolutions of libmantiis_cnn.so (forward, data gradient,
weight and bias gradients) against FP64 at the edges of their register tiles:
channel counts that are not multiples of a tile or a chunk, images smaller than
a tile and not multiples of it, rows that do not start on 16 bytes, and sizes
that choose each of the tiles.  Bounds: the standard one of an FP32 sum of K
products in any order, K 2^-24 times the sum of their magnitudes, per output."""
import numpy as np
import pytest

from test_gpu_conv_tc import bf16_round, conv_ref, wgrad_ref

pytestmark = pytest.mark.gpu

# (n, cin, cout, h, w)
SHAPES = [
    (1, 1, 1, 1, 1),
    (1, 2, 3, 5, 7),
    (2, 9, 17, 8, 8),
    (3, 33, 40, 9, 6),
    (1, 40, 70, 17, 19),
    (2, 31, 33, 34, 47),
    (4, 32, 3, 64, 64),
    (8, 64, 64, 8, 8),
    (8, 128, 256, 16, 16),
    (8, 20, 32, 130, 129),
]


def setup(shape, transpose=False):
    n, cin, cout, h, wd = shape
    rng = np.random.default_rng(sum(shape))
    w16 = bf16_round((rng.standard_normal((cout, cin, 3, 3)) / np.sqrt(9 * cin)).astype(np.float32))
    wq = (w16.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    b = rng.standard_normal(cout).astype(np.float32)
    x = rng.standard_normal((n, cout if transpose else cin, h, wd)).astype(np.float32)
    return w16, wq, b, x


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("transpose", [False, True])
def test_forward_and_data_gradient(shape, transpose):
    import torch

    from mantiis_gb300 import surrogate as S

    n, cin, cout, h, wd = shape
    w16, wq, b, x = setup(shape, transpose)
    X = torch.tensor(x, device="cuda")
    W = torch.tensor(w16.view(np.int16).reshape(-1), device="cuda")
    B = torch.tensor(b, device="cuda")
    Y = torch.full((n, cin if transpose else cout, h, wd), np.nan, device="cuda")
    L, st = S.cnn_lib(), S._stream()
    if transpose:
        assert L.cnn_conv3x3_backward_data(S._ptr(X), S._ptr(W), S._ptr(Y), n, cin, cout, h, wd, st) == 0
        ref = conv_ref(x.astype(np.float64), wq, None, transpose=True)
        size = conv_ref(np.abs(x).astype(np.float64), np.abs(wq), None, transpose=True)
        terms = 9 * cout
    else:
        assert L.cnn_conv3x3_forward(S._ptr(X), S._ptr(W), S._ptr(B), S._ptr(Y), n, cin, cout, h, wd, 1, st) == 0
        ref = np.maximum(conv_ref(x.astype(np.float64), wq, b.astype(np.float64)), 0.0)
        size = conv_ref(np.abs(x).astype(np.float64), np.abs(wq), np.abs(b).astype(np.float64))
        terms = 9 * cin + 1
    err = np.abs(Y.cpu().numpy() - ref)
    assert (err <= (terms + 1) * 2.0 ** -24 * size).all(), (err / size).max() * 2.0 ** 24 / terms


@pytest.mark.parametrize("shape", SHAPES)
def test_weight_and_bias_gradient(shape):
    import torch

    from mantiis_gb300 import surrogate as S

    n, cin, cout, h, wd = shape
    _, _, _, x = setup(shape)
    dy = np.random.default_rng(3).standard_normal((n, cout, h, wd)).astype(np.float32)
    X, DY = torch.tensor(x, device="cuda"), torch.tensor(dy, device="cuda")
    L, st = S.cnn_lib(), S._stream()
    # the gradients are added to what is there
    dw, db = torch.ones(cout * cin * 9, device="cuda"), torch.ones(cout, device="cuda")
    assert L.cnn_conv3x3_backward_weight(S._ptr(X), S._ptr(DY), S._ptr(dw), S._ptr(db), n, cin, cout, h, wd, st) == 0
    ref_w, ref_b = wgrad_ref(x.astype(np.float64), dy.astype(np.float64))
    size_w, size_b = wgrad_ref(np.abs(x).astype(np.float64), np.abs(dy).astype(np.float64))
    terms = n * h * wd + 1
    for got, ref, size in ((dw.reshape(cout, cin, 3, 3), ref_w, size_w), (db, ref_b, size_b)):
        err = np.abs(got.cpu().numpy() - (ref + 1.0))
        assert (err <= (terms + 1) * 2.0 ** -24 * (size + 1.0)).all(), err.max()
