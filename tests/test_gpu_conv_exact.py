"""The 3x3 convolutions on small whole numbers, whose sums FP32 holds exactly whatever
their order: every output equals FP64's, so a pixel, channel, tile or image left out
or counted twice shows, at remainders of every tile of the weight gradient."""
import numpy as np
import pytest

from test_gpu_conv_tc import conv_ref, wgrad_ref

pytestmark = pytest.mark.gpu

# (n, cin, cout, h, w), by the weight gradient's tile (pixels, output x input channels)
SHAPES = [
    (1, 1, 1, 1, 1), (2, 9, 17, 8, 8), (2, 40, 7, 9, 8),  # 16 x 8, 4 x 8
    (3, 33, 40, 9, 6), (3, 100, 6, 40, 41), (3, 3, 20, 33, 35), (8, 2, 5, 129, 129),  # 16 x 8, 8 x 8
    (5, 11, 34, 57, 57), (2, 50, 50, 30, 31), (4, 87, 93, 9, 9),  # 16 x 8, 16 x 16
    (8, 70, 64, 7, 8), (6, 251, 12, 20, 20), (2, 12, 90, 20, 21),  # 8 x 8, 16 x 16
    (8, 20, 32, 130, 129), (4, 64, 64, 70, 71),  # 16 x 8, 32 x 32
    (8, 256, 256, 8, 8),  # 8 x 8, 32 x 32
    (8, 3, 40, 60, 61),  # 16 x 8, 32 x 4
    (4, 32, 3, 63, 65), (8, 256, 8, 40, 41),  # 16 x 8, 4 x 32
    (8, 200, 6, 7, 7),  # 8 x 8, 4 x 32
]


@pytest.mark.parametrize("shape", SHAPES)
def test_whole_numbers(shape):
    import torch

    from mantiis_gb300 import surrogate as S

    n, cin, cout, h, wd = shape
    rng = np.random.default_rng(sum(shape))
    # sums of at most 9 n cout h w products of magnitude 4: below 2^24
    x, dy = (rng.integers(-2, 3, (n, c, h, wd)).astype(np.float32) for c in (cin, cout))
    w, b = (rng.integers(-2, 3, s).astype(np.float32) for s in ((cout, cin, 3, 3), cout))
    assert 4 * n * h * wd + 4 < 2 ** 24 and 4 * 9 * max(cin, cout) < 2 ** 24
    dev = lambda a: torch.tensor(a, device="cuda")
    X, DY, B = dev(x), dev(dy), dev(b)
    W = dev(w).bfloat16().view(torch.int16).reshape(-1).contiguous()
    Y, DX = torch.full_like(DY, np.nan), torch.full_like(X, np.nan)
    dw, db = torch.ones(w.size, device="cuda"), torch.ones(cout, device="cuda")  # added to what is there
    L, st, p = S.cnn_lib(), S._stream(), S._ptr
    assert L.cnn_conv3x3_forward(p(X), p(W), p(B), p(Y), n, cin, cout, h, wd, 0, st) == 0
    assert L.cnn_conv3x3_backward_data(p(DY), p(W), p(DX), n, cin, cout, h, wd, st) == 0
    assert L.cnn_conv3x3_backward_weight(p(X), p(DY), p(dw), p(db), n, cin, cout, h, wd, st) == 0
    x, dy, w, b = (a.astype(np.float64) for a in (x, dy, w, b))
    ref_w, ref_b = wgrad_ref(x, dy)
    for got, ref in ((Y, conv_ref(x, w, b)), (DX, conv_ref(dy, w, None, transpose=True)), (dw, ref_w + 1), (db, ref_b + 1)):
        assert np.array_equal(got.cpu().numpy().reshape(ref.shape), ref)
