"""The 8 x 16-pixel tile convolutions (any width, channel counts that are not
multiples of 64): forward and both gradients against the NumPy reference
(oracle/nn_np.py) on bfloat16-rounded operands, at the tolerances of the other
convolution tests (2e-2 of max for bfloat16 outputs, 5e-3 for the FP32 weight and bias
gradients).  Shapes at the edges: images smaller than a tile, one pixel more than a
tile, the network's 8- and 32-channel level with the 64 + 32 skip, partial chunks of 64
channels, output channels of every CTA width, several output tiles, more tiles than
CTAs, 256 input channels.  No bounded wait may run out."""
import numpy as np
import pytest

from oracle import nn_np as R

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(1, 1, 1, 8, 0, 8), (2, 16, 8, 32, 0, 32), (1, 17, 9, 8, 0, 32), (2, 31, 23, 64, 32, 32),
          (1, 5, 40, 32, 0, 8), (1, 12, 10, 96, 40, 64), (1, 9, 11, 128, 0, 128), (1, 20, 18, 128, 128, 128),
          (1, 33, 7, 32, 16, 96), (24, 48, 40, 32, 0, 64), (1, 10, 10, 24, 0, 200)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("relu", [0, 1])
def test_tile_convolution(shape, relu):
    from svirl_gb300 import learned as L
    n, h, w, c1, c2, cout = shape
    rng = np.random.default_rng(23)
    bf = lambda *s: R.bf16_round(rng.standard_normal(s).astype(np.float32))  # noqa: E731
    x1, x2 = bf(n, h, w, c1), bf(n, h, w, c2) if c2 else None
    W = (rng.standard_normal((cout, 3, 3, c1 + c2)) * 0.1).astype(np.float32)
    b = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    dy = bf(n, h, w, cout)
    xc = x1 if x2 is None else np.concatenate([x1, x2], axis=3)
    on = lambda a: torch.from_numpy(a).to("cuda", torch.bfloat16)  # noqa: E731
    tx1, tx2 = on(x1).requires_grad_(), None if x2 is None else on(x2).requires_grad_()
    tW, tb = torch.from_numpy(W).cuda().requires_grad_(), torch.from_numpy(b).cuda().requires_grad_()
    y = L.Conv3x3.apply(tx1, tx2, tW, tb, relu)
    g = torch.autograd.grad(y, [tW, tb, tx1] + ([tx2] if c2 else []), grad_outputs=on(dy))
    L.check_kernel_errors()
    f = lambda t: t.detach().float().cpu().numpy().astype(np.float64)  # noqa: E731
    dx_ref, dw_ref, db_ref = R.conv3x3_bwd(xc, R.bf16_round(W), f(y), dy, relu)
    dx = f(g[2]) if x2 is None else np.concatenate([f(g[2]), f(g[3])], axis=3)
    for got, ref, tol in ((f(y), R.conv3x3(xc, R.bf16_round(W), b, relu), 2e-2), (dx, dx_ref, 2e-2),
                          (f(g[0]), dw_ref, 5e-3), (f(g[1]), db_ref, 5e-3)):
        assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
