"""The convolutions under the settings of glnn_set_conv_tma: tile kernels (2, the default)
against the thread-gather and mma.sync kernels (0)."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _layer(setting, x1, x2, w, b, dy):
    """y, dx1, dx2, dW, db of one layer (ReLU forward, dy as it is)."""
    from svirl_gb300 import _lib
    lib = _lib.load()
    p = lambda t: None if t is None else C.c_void_p(t.data_ptr())  # noqa: E731
    n, h, wd, c1 = x1.shape
    c2, cout = 0 if x2 is None else x2.shape[3], w.shape[0]
    dev = {"device": "cuda"}
    err = torch.zeros(1, dtype=torch.int32, **dev)
    wb, wt = [torch.empty(cout * 9 * (c1 + c2), dtype=torch.bfloat16, **dev) for _ in range(2)]
    y = torch.empty((n, h, wd, cout), dtype=torch.bfloat16, **dev)
    dx1, dx2 = torch.empty_like(x1), None if x2 is None else torch.empty_like(x2)
    dw, db = torch.empty((cout, 3, 3, c1 + c2), **dev), torch.empty(cout, **dev)
    nwork = lib.glnn_conv3x3_bwd_weight_work(n, h, wd, c1 + c2, cout)
    work = torch.empty(nwork, **dev)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    try:
        assert lib.glnn_set_conv_tma(setting) == 0
        assert lib.glnn_prep_weights(p(w), p(wb), p(wt), cout, c1 + c2, s) == 0
        assert lib.glnn_conv3x3_fwd(p(x1), c1, p(x2), c2, p(wb), p(b), p(y), n, h, wd, cout, 1, p(err), s) == 0
        assert lib.glnn_conv3x3_bwd_data(p(dy), p(y), 0, p(wt), p(dx1), c1, p(dx2), c2, n, h, wd, cout, p(err), s) == 0
        assert lib.glnn_conv3x3_bwd_weight(p(dy), p(y), 0, p(x1), c1, p(x2), c2, p(dw), p(db), p(work), nwork, n, h, wd,
                                           cout, p(err), s) == 0
    finally:
        lib.glnn_set_conv_tma(2)
    assert int(err.item()) == 0
    return y, dx1, dx2, dw, db


def _inputs(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, h, w, c1, c2, cout = shape
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    return (r(n, h, w, c1).bfloat16(), r(n, h, w, c2).bfloat16() if c2 else None, 0.1 * r(cout, 3, 3, c1 + c2), r(cout),
            r(n, h, w, cout).bfloat16())


@pytest.mark.parametrize("shape", [(1, 1, 1, 8, 0, 8), (1, 17, 9, 8, 0, 32), (2, 31, 23, 64, 32, 32), (1, 12, 10, 96, 40, 64),
                                   (1, 10, 10, 24, 0, 200), (1, 16, 13, 32, 0, 32), (1, 13, 16, 32, 0, 32)])
def test_pixels_outside_the_image_add_nothing_to_the_weight_gradient(shape):
    """Infinite activations on the image's last row and column: a weight gets an infinity or a
    NaN exactly where a pixel of the image brings it one."""
    x1, x2, w, b, dy = _inputs(shape, 11)
    x1[:, -1, :, 0] = float("inf")
    x1[:, :, -1, -1] = float("-inf")
    if x2 is not None:
        x2[:, -1, -1, 3] = float("inf")
    got, ref = [_layer(s, x1, x2, w, b, dy)[3] for s in (2, 0)]
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    assert torch.equal(torch.where(torch.isinf(got), got, 0.0), torch.where(torch.isinf(ref), ref, 0.0))
    f = torch.isfinite(ref)
    assert torch.allclose(got[f], ref[f], rtol=0.0, atol=5e-3 * float(ref[f].abs().max()) if f.any() else 0.0)


@pytest.mark.parametrize("shape", [(1, 1, 1, 8, 0, 8), (2, 16, 8, 32, 0, 32), (1, 17, 9, 8, 0, 32), (2, 31, 23, 64, 32, 32),
                                   (3, 24, 56, 16, 0, 48), (1, 9, 11, 128, 0, 128), (1, 20, 18, 128, 128, 128),
                                   (1, 33, 7, 32, 16, 96), (24, 48, 40, 32, 0, 64), (2, 64, 64, 64, 0, 64),
                                   (8, 128, 128, 32, 0, 8), (2, 64, 60, 32, 0, 72), (2, 40, 33, 40, 24, 24)])
def test_settings_give_the_same_values(shape):
    """The forward bit for bit; the data gradient too where cout is a multiple of 16 (a K
    step of the tile kernel then holds the products that it holds in the gather kernel).
    Elsewhere its FP32 sums are grouped differently: at most the rounding of the sums
    (K = 9 cout terms, each side off by K 2^-24 times the terms' sum) and one rounding to
    bfloat16 (2^-8 of a value, either side) apart."""
    x1, x2, w, b, dy = _inputs(shape, 3)
    tile, gather = [_layer(s, x1, x2, w, b, dy) for s in (2, 0)]
    assert torch.equal(tile[0], gather[0])
    cout = shape[5]
    k = 9 * cout
    terms = k * float(dy.float().abs().max()) * float(w.abs().max())
    for t, g in zip(tile[1:3], gather[1:3]):
        if t is None:
            continue
        if cout % 16 == 0:
            assert torch.equal(t, g)
        else:
            t, g = t.float(), g.float()
            assert bool(((t - g).abs() <= 2.0 ** -7 * g.abs().maximum(t.abs()) + 2 * k * 2.0 ** -24 * terms).all())


@pytest.mark.parametrize("c1,c2", [(16, 16), (32, 32), (48, 16), (64, 16), (64, 48), (80, 0), (112, 0), (32, 96), (96, 64), (48, 80),
                                   (144, 0), (240, 0), (64, 176)])
def test_chunks_of_any_length_in_any_order(c1, c2):
    """Input channels in two to four chunks of one to four K steps: the same bits as the
    gather kernel's."""
    x1, x2, w, b, dy = _inputs((1, 19, 12, c1, c2, 32), 5)
    tile, gather = [_layer(s, x1, x2, w, b, dy) for s in (2, 0)]
    for t, g in zip(tile[:3], gather[:3]):
        assert t is None or torch.equal(t, g)
