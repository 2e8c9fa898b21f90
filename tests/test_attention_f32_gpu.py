"""float32 attention of prompt tiles and of single decoded tokens (csrc/attention_f32.cu): bit for bit what the general kernel
(csrc/attention_generic.cu, itself compared with the plain restatement in test_kernels_gpu.py) gives for the same tokens."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from iitj_llm_coopt_b200 import kernels
    return kernels.load()


def case(heads, kv_heads, head_dim, page, lens, qlens, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    need = [-(-n // page) for n in lens]
    perm = iter(torch.randperm(sum(need) + 3, generator=g).tolist())
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    cache = torch.full((sum(need) + 3, 2, kv_heads, page, head_dim), float("nan"))          # slots that nothing wrote
    for b, n in enumerate(lens):
        for j in range(need[b]):
            table[b, j] = p = next(perm)
            rows = min(page, n - j * page)
            cache[p, :, :, :rows] = torch.randn((2, kv_heads, rows, head_dim), generator=g) * scale
    q = torch.randn((sum(qlens), (heads + 2 * kv_heads) * head_dim), generator=g) * scale
    request = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(qlens)).int()
    positions = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, qlens)]).int()
    return q.cuda(), cache.cuda(), SimpleNamespace(block_table=table.cuda(), token_request=request.cuda(), positions=positions.cuda(),
                                                   query_lens=list(qlens), seq_lens_host=list(lens))


def general(K, q, cache, meta, heads, kv_heads, head_dim, window, scale):
    out = torch.empty(q.shape[0], heads * head_dim, device="cuda")
    K._call("llm_attention_generic", q.data_ptr(), q.shape[1], cache.data_ptr(), meta.block_table.data_ptr(), meta.block_table.shape[1],
            meta.token_request.data_ptr(), meta.positions.data_ptr(), out.data_ptr(), out.shape[1], 0, q.shape[0], heads, kv_heads,
            head_dim, cache.shape[3], window, scale, K._stream())
    return out


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("heads,kv_heads,page,window", [(4, 1, 16, 0), (3, 3, 8, 0), (6, 2, 7, 45), (2, 1, 16, 1), (2, 2, 64, 200)])
def test_same_numbers_as_the_general_kernel(K, head_dim, heads, kv_heads, page, window):
    # whole prompts and portions around the tile of 64 queries and the tile of 32 keys; single tokens around it and around a span of 1024
    lens = [1, 2, 63, 65, 130, 333, 1100, 31, 32, 33, 1023, 1024, 1025, 2100, 700]
    qlens = [1, 2, 63, 65, 70, 64, 37, 1, 1, 1, 1, 1, 1, 1, 1]
    for scale in (1.0, 6.0):                                    # the larger one: probabilities that underflow
        q, cache, meta = case(heads, kv_heads, head_dim, page, lens, qlens, 5, scale)
        out = torch.full((q.shape[0], heads * head_dim), 7.0, device="cuda")
        assert K._attention_f32_takes(q, cache, meta, out, heads, kv_heads, head_dim)
        K.attention(q, cache, meta, out, heads, kv_heads, head_dim, window=window, scale=0.17)
        want = general(K, q, cache, meta, heads, kv_heads, head_dim, window, 0.17)
        assert want.isfinite().all() and torch.equal(out, want)


def test_values_that_are_not_finite_stay_with_the_queries_that_see_them(K):
    q, cache, meta = case(2, 1, 64, 16, [100, 90], [100, 1], 6)
    page = meta.block_table[0, 3].item()
    cache[page, 1, 0, 5, 7] = float("inf")                      # position 53 of request 0
    cache[page, 1, 0, 6, 8] = float("nan")                      # position 54
    out = torch.empty(101, 128, device="cuda")
    K.attention(q, cache, meta, out, 2, 1, 64)
    want = general(K, q, cache, meta, 2, 1, 64, 0, 0.125)
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.nan_to_num(), want.nan_to_num())
    assert out[:53].isfinite().all() and not out[53:100].isfinite().all() and out[100].isfinite().all()
