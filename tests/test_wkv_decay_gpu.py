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


def test_a_rank_that_one_block_could_not_hold():
    """12300 numbers a channel.  A running sum of about one is rounded 12300 times by at most 2^-24 of itself, up or down at random: about
    111 * 6e-8 = 7e-6, and 5e-5 is beyond the luck of 2210 sums; through both exponentials it grows by less than one."""
    from iitj_llm_coopt_b200 import kernels
    K = kernels.load()
    g = torch.Generator(device="cuda").manual_seed(5)
    low, w2 = torch.randn((17, 12300), generator=g, device="cuda"), torch.randn((130, 12300), generator=g, device="cuda") * 0.01
    w0, out = torch.randn(130, generator=g, device="cuda") - 1.0, torch.empty(17, 130, device="cuda")
    K.wkv_decay(low, w2, w0, out)
    want = torch.exp(-torch.exp(torch.tanh(low.double()) @ w2.double().t() + w0.double()))
    assert (out - want).abs().max().item() < 5e-5


# tokens that the kernel of few takes, on both sides of the limits of its rule, against the same rows among many: the same bits
@pytest.mark.parametrize("tokens,channels,rank", [(1, 1, 4), (5, 63, 8), (5, 65, 64), (18, 3072, 64), (19, 3072, 64), (9, 4096, 128), (10, 4096, 128), (32, 512, 32),
                                                  (33, 512, 32), (2, 64, 8192), (3, 130, 100), (3, 130, 50)])
def test_few_tokens_give_the_bits_of_many(tokens, channels, rank):
    from iitj_llm_coopt_b200 import kernels
    K = kernels.load()
    g = torch.Generator(device="cuda").manual_seed(channels + rank)
    low, w2 = torch.randn((tokens, rank), generator=g, device="cuda"), torch.randn((channels, rank), generator=g, device="cuda") * 0.2
    w0 = torch.randn(channels, generator=g, device="cuda") - 1.0
    few, many = torch.full((tokens + 1, channels), 7.0, device="cuda"), torch.empty(tokens + 40, channels, device="cuda")
    K.wkv_decay(low, w2, w0, few[:tokens])
    K.wkv_decay(torch.cat([low, torch.zeros(40, rank, device="cuda")]), w2, w0, many)
    assert torch.equal(few[:tokens], many[:tokens]) and (few[tokens] == 7.0).all()
