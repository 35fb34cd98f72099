"""The preconditioner's module without a GPU."""
import torch


def test_network_without_layers_returns_its_first_input_channel():
    from efwi.cnn import Preconditioner
    feats = torch.randn(3, 2, 4, 5)
    out = Preconditioner(layers=0)(feats)
    assert torch.equal(out, feats[0].to(torch.bfloat16))
