"""Training inputs that are views off a 16-byte boundary, with and without
columns left out: the outputs and gradients are those of an aligned tensor
of the same values, to the bit (the loss is an atomic sum: 1e-6). And the
loss-gradient kernel that callers of the C interface have (training forms it
in its backward pass): against its formula, within a BF16 rounding."""

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 33, 300])
@pytest.mark.parametrize("first,cols", [(0, None), (2, 70), (1, 66)])
def test_views(m, first, cols):
    from picca_gb300 import learned
    stride = learned.FEATURE_STRIDE
    cols = cols or stride
    gen = torch.Generator(device="cuda").manual_seed(m)
    store = torch.randn(m * stride + 8, device="cuda", generator=gen).bfloat16()
    # rows of the layout's stride, from an odd element on
    view = store[3:3 + m * stride].view(m, stride)[:, first:first + cols]
    whole = torch.zeros(m, stride, device="cuda", dtype=torch.bfloat16)
    whole[:, :cols] = view
    target = torch.randn(2 * m + 1, device="cuda", generator=gen)[1:].view(m, 2)
    out = []
    for x, t in ((view, target), (whole, target.clone())):
        net = learned.WarmStartMLP(seed=3)
        y, acts = net.forward(x, keep=True)
        loss = net.backward(acts, y, t)
        out.append((y, net.grads.clone(), loss))
        assert torch.equal(net.forward(x), y)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert abs(float(out[0][2] - out[1][2])) <= 1e-6 * float(out[1][2])


@pytest.mark.parametrize("m,n", [(1, 1), (7, 3), (255, 2), (4096, 2), (1001, 5)])
def test_loss_gradient(m, n):
    from picca_gb300 import learned
    gen = torch.Generator(device="cuda").manual_seed(n)
    y, t = (torch.randn(m, n, device="cuda", generator=gen) for _ in range(2))
    dy = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    loss = torch.zeros(1, device="cuda")
    learned.check(learned._bind().pg_mlp_mse_grad(y.data_ptr(), t.data_ptr(), m, n, dy.data_ptr(),
                                                  loss.data_ptr(), None), "mse grad")
    torch.cuda.synchronize()
    d = (y - t).double()
    want = 2 * d / m
    assert bool(((dy.double() - want).abs() <= 2.0**-8 * want.abs()).all())
    assert abs(float(loss) - float((d * d).sum() / m)) <= 1e-5 * float((d * d).sum() / m)
