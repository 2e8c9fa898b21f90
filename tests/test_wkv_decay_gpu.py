"""The decays of the wkv mixer (csrc/wkv.cu) against 64 bits, at the edges of the kernel's blocks of 16 tokens, 128 channels and 32 ranks.

Bound: a sum of `rank` terms of at most 1 in float32 is off by at most rank * 2^-24 * sum |w|; twice through exp of numbers of order one
that stays below 1e-5 for these sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 16, 17, 50])
@pytest.mark.parametrize("channels,rank", [(1, 1), (127, 32), (129, 33), (256, 70), (384, 64)])
def test_decay(tokens, channels, rank):
    from iitj_llm_coopt_b200 import kernels
    K = kernels.load()
    g = torch.Generator(device="cuda").manual_seed(tokens + channels)
    low, w2 = torch.randn((tokens, rank), generator=g, device="cuda"), torch.randn((channels, rank), generator=g, device="cuda") * 0.2
    w0 = torch.randn(channels, generator=g, device="cuda") - 1.0
    out = torch.full((tokens + 1, channels), 7.0, device="cuda")
    K.wkv_decay(low, w2, w0, out[:tokens])
    want = torch.exp(-torch.exp(torch.tanh(low.double()) @ w2.double().t() + w0.double()))
    assert (out[:tokens] - want).abs().max().item() < 1e-5 and (out[tokens] == 7.0).all()
