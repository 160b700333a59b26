"""The warm-start network's tile GEMM and training pass at the edges of their
tiles, K chunks and cluster splits.

GEMM: against torch in FP64 on the same BF16 operands; FP32 accumulation of
k exact products stays within k 2^-23 of the sum of absolute products, and a
BF16 output adds half a unit of its last place (2^-8). Training pass: against
the FP64 oracle with BF16 storage rounding (the tolerances of the network's
other tests: 1e-2 forward, 2e-2 gradients)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _operand(rows, cols, transposed, pad, gen):
    """A [rows, cols] bf16 matrix stored row- or column-major with a padded
    leading dimension: (values, tensor, stride of a row, stride of a column)."""
    shape = (cols, rows + pad) if transposed else (rows, cols + pad)
    store = torch.randn(shape, device="cuda", generator=gen).bfloat16()
    values = (store[:, :rows].T if transposed else store[:, :cols]).double()
    return values, store, (1 if transposed else shape[1]), (shape[1] if transposed else 1)


@pytest.mark.parametrize("m,n,k", [(1, 8, 1), (64, 64, 64), (65, 72, 66), (300, 256, 256),
                                   (63, 255, 257), (66, 256, 4096), (256, 256, 1023),
                                   (40, 16, 520)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("odd", [False, True])
def test_gemm(m, n, k, a_t, b_t, odd):
    from picca_gb300 import learned
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    net = learned.WarmStartMLP(seed=1)

    def pad(size):  # odd leading dimensions stay on the staged kernel
        return 1 + size % 2 if odd else -size % 8

    a, at, sam, sak = _operand(m, k, a_t, pad(m if a_t else k), gen)
    b, bt, sbk, sbn = _operand(k, n, b_t, pad(k if b_t else n), gen)
    bias = torch.randn(n, device="cuda", generator=gen)
    zin = torch.randn(m, n, device="cuda", generator=gen)
    exact = a @ b
    tol = k * 2.0**-23 * (a.abs() @ b.abs()) + 1e-6
    c = torch.full((m, n), 2.0, device="cuda")
    net.gemm(at, sam, sak, bt, sbk, sbn, m, n, k, cf=c, ldc=n, beta=0.5)
    assert bool(((c.double() - (exact + 1.0)).abs() <= tol + 2e-7 * exact.abs()).all())
    z, h = torch.empty_like(c), torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    net.gemm(at, sam, sak, bt, sbk, sbn, m, n, k, bias=bias, epilogue=learned.EPI_GELU, zout=z,
             ldz=n, c=h, ldc=n)
    exact = exact + bias.double()
    assert bool(((z.double() - exact).abs() <= tol + 2e-7 * exact.abs()).all())
    want = torch.nn.functional.gelu(z.double())
    assert bool(((h.double() - want).abs() <= 2.0**-8 * want.abs() + 1e-6).all())
    net.gemm(at, sam, sak, bt, sbk, sbn, m, n, k, epilogue=learned.EPI_GELU_GRAD, zin=zin, ldz=n,
             c=h, ldc=n)
    zd = zin.double().requires_grad_(True)
    grad = torch.autograd.grad(torch.nn.functional.gelu(zd).sum(), zd)[0]
    want = (exact - bias.double()) * grad
    assert bool(((h.double() - want).abs() <= 2.0**-8 * want.abs() + 1.2 * tol + 1e-5).all())


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("m", [1, 7, 63, 65, 512, 513, 4099])
def test_training_pass(m):
    from oracle import mlp as om
    from picca_gb300 import learned
    net = learned.WarmStartMLP(seed=3)
    rng = np.random.default_rng(m)
    x = np.full((m, learned.FEATURE_STRIDE), np.nan, dtype=np.float32)  # unused columns
    x[:, :learned.NUM_FEATURES] = rng.normal(0, 0.5, (m, learned.NUM_FEATURES))
    t = rng.normal(0, 0.3, (m, 2)).astype(np.float32)
    y, acts = net.forward(torch.tensor(x, device="cuda").bfloat16(), keep=True)
    loss = net.backward(acts, y, torch.tensor(t, device="cuda"))
    views = net._views(net.params.cpu().double())
    weights = [(w.numpy().reshape(a, b), bb.numpy()) for (w, bb), (a, b) in
               zip(views, learned.WarmStartMLP.SHAPES)]
    xin = x[:, :learned.NUM_FEATURES].astype(np.float64)
    y_ref, acts_ref = om.forward(xin, weights, quantize=True)
    assert _rel(y.cpu().numpy(), y_ref) < 1e-2
    grads_ref, loss_ref = om.backward(acts_ref, y_ref, t.astype(np.float64), weights,
                                      quantize=True)
    assert abs(float(loss.item()) - loss_ref) <= 2e-2 * loss_ref
    for layer, (gw, gb) in enumerate(net._views(net.grads.cpu().double())):
        assert _rel(gw.numpy().reshape(grads_ref[layer][0].shape), grads_ref[layer][0]) < 2e-2
        assert _rel(gb.numpy(), grads_ref[layer][1]) < 2e-2
    # the column sums of any width
    dz = torch.randn(m, 13, device="cuda").bfloat16()
    out = torch.empty(11, device="cuda")
    learned.check(learned._bind().pg_mlp_colsum(dz.data_ptr(), m, 11, 13, out.data_ptr(),
                                                net._stream()), "colsum")
    want = dz[:, :11].double().sum(0)
    assert bool(((out.double() - want).abs() <= m * 2.0**-24 * dz[:, :11].double().abs().sum(0) +
                 1e-7).all())
