"""A point's prediction does not depend on how many others are predicted with it, to the bit: the
passes take 4, 2 or 1 operand rows per sample by the number of points, and sum the outputs over the
256 neurons in the same tree each time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [1, 5])
def test_predictions_of_a_point_are_the_same_bits_in_any_batch(heads):
    import sph_surrogate

    net = sph_surrogate.MLP(heads=heads, max_batch=128, seed=5)
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(19900, 6, generator=g, device="cuda")  # 156 tiles a head: one row per sample
    whole = net.predict(x)
    # one head: 1, 30 (four rows a sample), 40, 70 (two), 80 tiles; five heads: 5 to 400
    for n in (1, 100, 128, 30 * 128, 40 * 128 - 5, 70 * 128, 80 * 128):
        assert torch.equal(net.predict(x[:n].contiguous()), whole[:, :n]), n
    net.close()
