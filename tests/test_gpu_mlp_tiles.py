"""The surrogate's fused passes at the sizes where their tiling changes: 4, 2 and 1 operand rows
per sample (by the number of 128-sample tiles over all heads), one to eight slices of the
weight gradients, one tile and many, and inputs at any float alignment."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(n, 6, generator=g, device="cuda"),
            torch.randn(n, 4, generator=g, device="cuda"))


# (heads, batch): 1, 6, 48, 80 and 160 tiles on 148 SMs; 2, 2, 8, 4 and 8 slices
@pytest.mark.parametrize("heads,batch", [(1, 128), (6, 128), (6, 1024), (16, 640), (20, 1024)])
def test_gradients_match_fp64_oracle(heads, batch):
    """The bounds of the network's gradient test: FP32 against FP64 accumulation of the same
    bf16 operands, and rare one-ulp bf16 flips (2e-3 of each tensor's norm)."""
    import mlp_oracle
    import sph_surrogate

    net = sph_surrogate.MLP(heads=heads, max_batch=batch, seed=heads)
    x, y = _batch(batch, 4)
    loss, g = net.gradients(x, y)
    P = net.get_params()
    for h in {0, heads - 1}:
        ref_loss, ref_g = mlp_oracle.loss_and_grads(P[h], x.cpu().numpy(), y.cpu().numpy())
        assert abs(loss[h] - ref_loss) <= 1e-4 * ref_loss
        for name, (a, b) in mlp_oracle.OFFS.items():
            num = np.linalg.norm(g[h, a:b] - ref_g[a:b])
            assert num <= 2e-3 * np.linalg.norm(ref_g[a:b]), (h, name)
    net.close()


@pytest.mark.parametrize("heads,n", [(1, 1), (1, 128), (3, 1500), (5, 6000), (4, 20011)])
def test_predictions_do_not_depend_on_the_tiling(heads, n):
    """Points predicted together and 128 at a time: the hidden layers are the same bits, the
    output sums 256 FP32 terms in another order (1e-6 of the output scale, some 16 ulps)."""
    import sph_surrogate

    net = sph_surrogate.MLP(heads=heads, max_batch=128, seed=2)
    x, _ = _batch(n, 6)
    whole = net.predict(x)
    scale = whole.abs().max()
    for a in sorted({0, n // 2 // 128 * 128, (n - 1) // 128 * 128}):
        part = net.predict(x[a:a + 128].contiguous())
        assert (whole[:, a:a + 128] - part).abs().max() <= 1e-6 * scale
    net.close()


def test_inputs_at_any_float_alignment():
    import sph_surrogate

    x, y = _batch(257, 8)
    flat = torch.zeros(257 * 6 + 1, device="cuda")
    flat[1:] = x.reshape(-1)
    odd = flat[1:].view(257, 6)[1:]  # a view 28 bytes past an aligned address
    out = []
    for xs in (x[1:].clone(), odd):
        net = sph_surrogate.MLP(heads=2, max_batch=256, seed=3)
        net.train_step(xs, y[1:], 1e-3)
        out.append((net.get_params(), net.predict(xs).cpu().numpy()))
        net.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
