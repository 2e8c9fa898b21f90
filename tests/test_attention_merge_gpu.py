"""Prefill attention whose keys are shared out over 2 to 16 blocks a tile, and the kernel that adds their results (csrc/attention_tcgen05.cu;
a split has about 2048 keys, so many splits need long contexts): the three register budgets of 4, 8 and 16 splits, tiles with fewer splits
than the launch provides, tiles without any, rows past a tile's end.

Bound, 2-norm of the difference over that of the result: probabilities and results are each rounded to 8 bits (2^-9 of themselves), which
adds up to less than 2^-7.  Values grow along the context, so that a split that is lost or wrongly weighted moves the result by more than
a sixteenth."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def long_case(heads, kv_heads, head_dim, lens, qlens, page=16):
    g = torch.Generator(device="cuda").manual_seed(heads + head_dim)
    need = [-(-n // page) for n in lens]
    order = 1 + torch.randperm(sum(need), generator=g, device="cuda")             # page 0 pads the block tables
    table = torch.zeros(len(lens), max(need), dtype=torch.int32, device="cuda")
    cache = torch.zeros((sum(need) + 1, 2, kv_heads, page, head_dim), dtype=torch.bfloat16, device="cuda")
    q = torch.randn((sum(qlens), heads + 2 * kv_heads, head_dim), generator=g, device="cuda").bfloat16()
    want, at, row = [], 0, 0
    for b, (n, m) in enumerate(zip(lens, qlens)):
        pages = order[at:at + need[b]]
        at += need[b]
        table[b, :need[b]] = pages
        k, v = (torch.randn((n, kv_heads, head_dim), generator=g, device="cuda") for _ in range(2))
        k, v = (k * 1.5).bfloat16(), (v + 4.0 * torch.arange(n, device="cuda").view(n, 1, 1) / n).bfloat16()
        for x, plane in ((k, 0), (v, 1)):
            full = torch.zeros((need[b] * page, kv_heads, head_dim), dtype=torch.bfloat16, device="cuda")
            full[:n] = x
            cache[pages, plane] = full.view(need[b], page, kv_heads, head_dim).transpose(1, 2)
        kk, vv = (x.double().repeat_interleave(heads // kv_heads, 1) for x in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[row:row + m, :heads].double(), kk) * head_dim ** -0.5
        late = torch.arange(n, device="cuda").view(1, n) > torch.arange(n - m, n, device="cuda").view(m, 1)
        want.append(torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(late, float("-inf")), -1), vv).reshape(m, -1))
        row += m
    request = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(qlens)).int().cuda()
    positions = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, qlens)]).int().cuda()
    meta = SimpleNamespace(block_table=table, token_request=request, positions=positions, query_lens=list(qlens), seq_lens_host=list(lens))
    return q.view(q.shape[0], -1), cache, meta, torch.cat(want)


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(2, 1, 64), (3, 3, 128)])
def test_two_to_sixteen_splits(heads, kv_heads, head_dim):
    from iitj_llm_coopt_b200 import kernels
    K = kernels.load()
    lens, qlens = [32300, 18500, 9700, 3900, 700], [70, 129, 33, 128, 5]          # 16, 9, 5, 2 splits at most, and none
    q, cache, meta, want = long_case(heads, kv_heads, head_dim, lens, qlens)
    before = K.attention_splits
    try:
        for splits in (1, 2, 4, 5, 8, 9, 15, 16):
            K.attention_splits = splits
            out = torch.full((q.shape[0] + 1, heads * head_dim), 7.0, dtype=torch.bfloat16, device="cuda")
            K.attention(q, cache, meta, out[:-1], heads, kv_heads, head_dim)
            assert ((out[:-1] - want).norm() / want.norm()).item() < 2 ** -7, splits
            assert (out[-1] == 7.0).all()
    finally:
        K.attention_splits = before
    assert K.attention_status() == 0
