"""float32 products on the tensor cores (csrc/gemm_f32_tc.cu) against the same product in 64 bits.

Bound: every factor is held exactly in three bfloat16 pieces; left out are piece products of at most 2^-23 of a product, and
a chunk of 128 k is added up by the tensor cores in eight steps that cut off (at most 2^-23 of the running sum each), which
shrinks a chunk by less than 8 * 2^-23 / 2 = 4.8e-7 of itself in the mean.  In the 2-norm of a result with random signs that and
the rounded sum over at most 160 chunks stay below 1e-6."""
import pytest
import torch

import test_attention_f32_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from iitj_llm_coopt_b200 import kernels
    return kernels.load()


def product(x, w, swiglu=False):
    y = x.double() @ w.double().t()
    if swiglu:
        n = w.shape[0] // 2
        y = torch.nn.functional.silu(y[:, :n]) * y[:, n:]
    return y


def rnd(shape, seed, scale=1.0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale


# token counts at the edges of the two kernels and of the tiles; k at one piece, at the edges of boxes (32), steps (64), chunks (128) and
# segments (256), with every kind of cluster (2 .. 8 blocks) and beyond eight chunks a block
@pytest.mark.parametrize("tokens", [1, 16, 17, 80, 81, 333])
@pytest.mark.parametrize("n,k", [(1, 4), (130, 36), (128, 64), (129, 132), (64, 256), (200, 264), (300, 1028), (130, 1792), (257, 4104), (64, 20000)])
def test_product(K, tokens, n, k):
    for swiglu in (False, True):
        x, w = rnd((tokens, k), 1), rnd(((2 if swiglu else 1) * n, k), 2, k ** -0.5)
        out = torch.full((tokens + 1, n), 7.0, device="cuda")
        K.linear(x, w, out[:tokens], swiglu=swiglu)
        want = product(x, w, swiglu)
        assert ((out[:tokens] - want).norm() / want.norm()).item() < 1e-6
        assert (out[tokens] == 7.0).all() and K.gemm_status() == 0
        row = torch.empty(1, n, device="cuda")                   # a row by itself: the same number, bit for bit
        K.linear(x[tokens // 2:tokens // 2 + 1].contiguous(), w, row, swiglu=swiglu)
        assert torch.equal(row[0], out[tokens // 2])


# more blocks than the GPU holds at a time, so that loads land late and in any order: every kind of block, with and without clusters
@pytest.mark.parametrize("tokens,n,k", [(5, 40000, 2048), (16, 9000, 8192), (200, 20000, 1024), (32, 6000, 4096)])
def test_many_blocks(K, tokens, n, k):
    x, w = rnd((tokens, k), 1), rnd((n, k), 2, k ** -0.5)
    out = torch.empty(tokens, n, device="cuda")
    K.linear(x, w, out)
    want = product(x, w)
    assert ((out - want).norm() / want.norm()).item() < 1e-6 and K.gemm_status() == 0


# few tokens: one block and two to an SM, clusters of one to eight blocks, one wave and several; a row has the same bits in every cut
@pytest.mark.parametrize("n,k", [(14000, 1500), (9000, 3000), (18944, 3584), (5120, 3072), (2560, 2560), (1536, 1536), (8192, 2048), (768, 768), (20000, 2048)])
def test_cuts_of_few_tokens(K, n, k):
    x, w = rnd((16, k), 1), rnd((n, k), 2, k ** -0.5)
    want, first = product(x, w), None
    for tokens in (16, 12, 8, 4, 1):
        out = torch.full((tokens + 1, n), 7.0, device="cuda")
        K.linear(x[:tokens].contiguous(), w, out[:tokens])
        assert ((out[:tokens] - want[:tokens]).norm() / want[:tokens].norm()).item() < 1e-6 and K.gemm_status() == 0
        first = out[:16] if first is None else first
        assert torch.equal(out[:tokens], first[:tokens]) and (out[tokens] == 7.0).all()


def test_infinities_and_nans_go_where_they_would(K):
    x, w = rnd((40, 300), 3), rnd((70, 300), 4)
    x[3, 5], x[4, 299], x[5, 0] = float("inf"), float("nan"), -float("inf")
    w[7, 5] = float("inf")
    w[8, :] = 0.0
    x[6, 11] = 3.4e38                                            # rounds to infinity in eight bits; stays finite here
    w[:, 11] = w[:, 11].abs().clamp(1e-3, 0.9)
    want = (x.double() @ w.double().t()).float()
    for rows in (slice(0, 40), slice(0, 9)):
        out = torch.empty(40, 70, device="cuda")[rows]
        K.linear(x[rows].contiguous(), w, out)
        assert torch.equal(out.isnan(), want[rows].isnan()) and torch.equal(out.isposinf(), want[rows].isposinf())
        assert torch.equal(out.isneginf(), want[rows].isneginf())
        ok = want[rows].isfinite()
        assert ((out - want[rows])[ok].abs() <= 1e-5 * want[rows][ok].abs() + 1e-4).all()


@pytest.mark.parametrize("tokens", [8, 40])
def test_nans_stay_nans_whatever_their_payload(K, tokens):
    x, w = rnd((tokens, 300), 3), rnd((70, 300), 4)
    bits = torch.tensor([0x7f800001, 0x7fc00000, -0x7fffff, 0x7f80ffff, -1], dtype=torch.int64).int().cuda()     # low, high, negative, all low bits
    for i, at in enumerate((0, 33, 131, 255, 299)):
        x.view(torch.int32)[i, at] = bits[i]
        w.view(torch.int32)[7 * i, at] = bits[4 - i]
    w[69, 100], x[6, 7] = float("inf"), float("inf")             # infinities beside them stay infinite
    want = (x.double() @ w.double().t()).float()
    out = torch.empty(tokens, 70, device="cuda")
    K.linear(x, w, out)
    assert want.isnan().any() and want.isinf().any()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isposinf(), want.isposinf()) and torch.equal(out.isneginf(), want.isneginf())
    ok = want.isfinite()
    assert ((out - want)[ok].abs() <= 1e-5 * want[ok].abs() + 1e-4).all()


def test_rows_that_start_off_a_boundary_take_the_other_kernel(K):
    base = rnd((5 * 64 + 1,), 5)
    x, w = base[1:].view(5, 64), rnd((30, 64), 6)
    assert not K.lib.llm_gemm_f32_tc_supported(64, x.data_ptr(), w.data_ptr()) and not K.lib.llm_gemm_f32_tc_supported(66, w.data_ptr(), w.data_ptr())
    out = torch.empty(5, 30, device="cuda")
    K.linear(x, w, out)
    assert ((out - product(x, w)).norm() / product(x, w).norm()).item() < 1e-6


def test_on_two_streams_at_once(K):
    streams = [torch.cuda.Stream() for _ in range(2)]
    xs, ws = [rnd((100, 512), 7 + i) for i in range(2)], [rnd((700, 512), 9 + i) for i in range(2)]
    want = [product(x, w) for x, w in zip(xs, ws)]
    torch.cuda.synchronize()
    outs = [[torch.empty(100, 700, device="cuda") for _ in range(20)] for _ in range(2)]
    torch.cuda.synchronize()
    for j in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                K.linear(xs[i], ws[i], outs[i][j])
    torch.cuda.synchronize()
    for i in range(2):
        for o in outs[i]:
            assert ((o - want[i]).norm() / want[i].norm()).item() < 1e-6


# against 64 bits no further off than the chain of fused multiply-adds that takes the other rows, for random signs and (the tensor cores cut
# sums off instead of rounding them) for factors of one sign; from K = 256 on the chain loses more with every number
@pytest.mark.parametrize("k", [4, 8, 16, 32, 48, 64, 68, 96, 128, 132, 160, 192, 256, 2048])
@pytest.mark.parametrize("one_sign", [False, True])
def test_no_further_off_than_a_chain(K, k, one_sign):
    x, w = rnd((96, k), 1), rnd((512, k), 2)
    if one_sign:
        x, w = x.abs(), w.abs()
    want, out, chain = product(x, w), torch.empty(96, 512, device="cuda"), torch.empty(96, 512, device="cuda")
    K.linear(x, w, out)
    K._call("llm_gemm_f32", x.data_ptr(), w.data_ptr(), chain.data_ptr(), 96, 512, k, k, k, 512, 0, K._stream())
    assert (out - want).norm().item() <= (chain - want).norm().item()


# sums whose large pieces cancel: what is left are the small products, and not one of them is missing.  All pieces' sums of these factors are
# held exactly, and 24 roundings of numbers below one (chunks and segments) are off by 24 * 2^-25 = 7e-7; sixteen low pieces, as one
# instruction adds them, are worth 1e-5.
@pytest.mark.parametrize("tokens", [5, 60, 100])
def test_small_products_are_all_there(K, tokens):
    k, n = 2048, 300
    sign = torch.ones(k, device="cuda")
    sign[1::2] = -1.0
    rest = lambda rows, seed: torch.randint(-2 ** 14, 2 ** 14, (rows, k), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * 2.0 ** -23
    for x, w in ((torch.ones(tokens, k, device="cuda"), sign * (1.0 + rest(n, 1))), (sign * (1.0 + rest(tokens, 2)), torch.ones(n, k, device="cuda"))):
        x, w, out = x.contiguous(), w.contiguous(), torch.empty(tokens, n, device="cuda")
        for _ in range(20):
            K.linear(x, w, out)
            assert (out - product(x, w)).abs().max().item() < 1e-6


# beside a kernel that keeps the SMs' load paths or the memory busy: the same bits as alone.  (A box of W that was handed back while its
# numbers were still on their way into registers was overwritten by its successor here.)
@pytest.mark.parametrize("other", ["attention", "copies"])
@pytest.mark.parametrize("tokens", [5, 300])
def test_beside_other_work(K, tokens, other):
    q, cache, meta = test_attention_f32_gpu.case(32, 8, 64, 16, [900, 800, 700, 600, 300] * 8, [1] * 40, 5)
    ctx, a, b = torch.empty(40, 2048, device="cuda"), torch.empty(1 << 27, device="cuda"), torch.empty(1 << 27, device="cuda")
    x, ws = rnd((tokens, 2048), 1), [rnd((2 * 8192, 2048), 2 + i, 2048 ** -0.5) for i in range(4)]
    first, outs = [torch.empty(tokens, 8192, device="cuda") for _ in ws], [torch.empty(tokens, 8192, device="cuda") for _ in ws]
    for w, o in zip(ws, first):
        K.linear(x, w, o, swiglu=True)
    assert ((first[0] - product(x, ws[0], True)).norm() / product(x, ws[0], True).norm()).item() < 1e-6
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(25):
        for w, o in zip(ws, outs):
            with torch.cuda.stream(side):
                if other == "copies":
                    a.copy_(b)
                else:
                    for _ in range(8):
                        K.attention(q, cache, meta, ctx, 32, 8, 64)
            K.linear(x, w, o, swiglu=True)
        torch.cuda.synchronize()
        assert all(torch.equal(o, f) for o, f in zip(outs, first)) and K.gemm_status() == 0


# the listed form against the products of each expert by itself (bit for bit) and against 64 bits: tiles of one to 64 rows, experts without
# rows, choices of experts without tensors, both kernels
@pytest.mark.parametrize("tokens,experts,top", [(1, 4, 2), (8, 5, 2), (9, 3, 2), (100, 4, 1), (150, 3, 2)])
@pytest.mark.parametrize("form", [False, "clamped", "silu", "silu_weighted"])
def test_listed_products(K, tokens, experts, top, form):
    n, k, pairs = 200, 300, tokens * top
    g = torch.Generator().manual_seed(tokens)
    chosen = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(tokens)]).int()
    chosen[chosen == 1] = experts                              # nobody at expert 1; those choices have no tensors
    weights = torch.rand((tokens, top), generator=g).cuda() + 0.5
    x, w = rnd((tokens, k), 3), rnd((experts, (2 if form else 1) * n, k), 4, k ** -0.5)
    i32 = dict(dtype=torch.int32, device="cuda")
    plan = K.moe_plan(chosen.cuda(), experts, torch.zeros(pairs, **i32), torch.empty(pairs, **i32),
                      torch.empty((K.moe_tile_bound(pairs, experts) + 1, 4), **i32), weights=weights, row_weight=torch.ones(pairs, device="cuda"))
    out = torch.full((pairs, n), 7.0, device="cuda")
    K.moe_linear(x, w, out, plan, gather=True, glu=form, limit=1.5, slope=1.7)
    place = plan["place"].view(tokens, top).cpu()
    for e in range(experts):
        at = [(t, j) for t in range(tokens) for j in range(top) if chosen[t, j] == e]
        if not at:
            continue
        rows = torch.tensor([place[t, j] for t, j in at]).cuda()
        xe = x[torch.tensor([t for t, _ in at]).cuda()].contiguous()
        y = xe.double() @ w[e].double().t()
        if form:
            gate, up = y[:, :n], y[:, n:]
            if form == "clamped":
                gate, up = gate.clamp(max=1.5), up.clamp(-1.5, 1.5)
                y = gate * torch.sigmoid(1.7 * gate) * (up + 1.0)
            else:
                s = torch.stack([weights[t, j] for t, j in at]).double().view(-1, 1) if form == "silu_weighted" else 1.0
                y = torch.nn.functional.silu(s * gate) * (s * up)
        assert ((out[rows] - y).norm() / y.norm()).item() < 1e-6
        if form in (False, "silu"):
            alone = torch.empty(len(at), n, device="cuda")
            K.linear(xe, w[e], alone, swiglu=bool(form))
            assert torch.equal(out[rows], alone)
    live = int((chosen < experts).sum())
    assert (out[live:] == 7.0).all() and K.gemm_status() == 0


def test_the_same_numbers_every_time(K):
    """A large product ten times over, bit for bit: 10^8 and more waits of whole warps."""
    x, w = rnd((2400, 2048), 1), rnd((60000, 2048), 2, 2048 ** -0.5)
    first, out = torch.empty(2400, 60000, device="cuda"), torch.empty(2400, 60000, device="cuda")
    K.linear(x, w, first)
    for _ in range(10):
        K.linear(x, w, out)
        assert torch.equal(out, first)
