"""The fused training kernels against the numpy oracle and autograd: batches
below, at and past a 128-row tile, part-filled batches, one and many splits."""

import pytest

torch = pytest.importorskip("torch")
np = pytest.importorskip("numpy")

from geometricvofext_gb300 import mlp  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,split", [(64, 64, 1), (128, 128, 1), (192, 256, 8), (1024, 1024, 2), (8256, 8320, 8)])
def test_gradients_match_oracle(n, batch, split):
    from oracle import mlp_oracle as MO

    rng = np.random.default_rng(n)
    W, b = mlp.init_params(7)
    W = W + rng.normal(0, 0.02, W.shape).astype(np.float32)
    W[-1, mlp.N_OUT:] = 0.0
    b = rng.normal(0, 0.1, b.shape).astype(np.float32)
    Xh = MO.bf16(rng.normal(0, 1, (n, 128)))
    X = torch.tensor(Xh, device="cuda").to(torch.bfloat16)
    dY = torch.zeros((n, 128), device="cuda")
    dY[:, :4] = torch.tensor(rng.normal(0, 1e-2, (n, 4)), dtype=torch.float32, device="cuda")
    tr = mlp.Trainer(W, b, batch)
    for _ in range(2):  # gradients are overwritten, not added to
        Y = tr.forward(X)[:n].clone()
        gW, gb = tr.backward(X, dY, split_k=split)
    torch.cuda.synchronize()
    assert int(tr.err.item()) == 0
    Yo, Zs, Hs = MO.forward(W, b, Xh)
    gWo, gbo = MO.backward(W, b, Xh, Zs, Hs, dY.cpu().numpy())
    # BF16 rounding points as the oracle's; the hardware tanh is within 2^-10
    Yg = Y.cpu().numpy()
    assert np.linalg.norm(Yg[:, :4] - Yo[:, :4]) <= 1e-2 * np.linalg.norm(Yo[:, :4])
    for l in range(mlp.N_LAYERS):
        for a, o in ((gW[l].cpu().numpy(), gWo[l]), (gb[l].cpu().numpy(), gbo[l])):
            assert np.linalg.norm(a - o) <= 2e-2 * np.linalg.norm(o) + 1e-9, l


@pytest.mark.parametrize("n", [1, 7, 8, 1000])
def test_loss_and_gradient_match_autograd(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    X = torch.randn((n, 128), generator=g, device="cuda").to(torch.bfloat16)
    Y = 0.5 * torch.randn((n, 128), generator=g, device="cuda")
    T = torch.randn((n, 4), generator=g, device="cuda")
    T[:, :3] /= T[:, :3].norm(dim=1, keepdim=True)
    Y[0, :3] = -X[0, 124:127].float()  # a zero normal: below the clamp
    loss, dY = mlp.loss_and_grad(Y, T, X)
    y = Y[:, :4].double().requires_grad_(True)
    v = X[:, 124:127].double() + y[:, :3]
    # (clamp's gradient and the norm's at zero as autograd has them in FP64)
    nn = v / torch.clamp(v.norm(dim=1, keepdim=True), min=1e-6)
    L = (1.0 - (nn * T[:, :3].double()).sum(1)).mean() + mlp.D_WEIGHT * ((y[:, 3] - T[:, 3].double()) ** 2).mean()
    (ref,) = torch.autograd.grad(L, y)
    L = float(L.detach())
    assert abs(loss - L) <= 1e-5 * max(1.0, abs(L))
    assert torch.all(dY[:, 4:] == 0)
    torch.testing.assert_close(dY[:, :4].double(), ref, rtol=1e-4, atol=1e-6 * float(ref.abs().max()))
