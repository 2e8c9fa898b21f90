"""Whole float32 steps of the engine at the 1B layer sizes, launched kernel by kernel (no graphs) with pauses in between, so that every
kernel meets its neighbours at ever other moments: all passes give the same bits, and those of the plain implementation to 5e-5 (float32
sums behind a few layers are 1e-6 off 64 bits)."""
import time

import pytest
import torch

import plain_kobolix
import plain_llama
from iitj_llm_coopt_b200 import LLM, StepEntry, kernels
from iitj_llm_coopt_b200.config.registry import architecture_for
from iitj_llm_coopt_b200.presets import shape_config
from iitj_llm_coopt_b200.weights.random_init import random_checkpoint

pytestmark = pytest.mark.gpu


def config(shape, layers):
    cfg = shape_config(shape)
    return dict(cfg, layers=cfg["layers"][:layers]) if "layers" in cfg else dict(cfg, num_hidden_layers=layers)


def oracle(cfg, arch, spec, seed, sequences):
    """The last position's logits of every sequence."""
    w = random_checkpoint(arch, spec, seed, device="cuda")
    if "layers" in cfg:
        w = {name: t.cpu().double() for name, t in w.items()}
        return torch.stack([plain_kobolix.forward(cfg, w, toks)[-1] for toks in sequences]).cuda()
    w = {name: t.double() for name, t in w.items()}
    return torch.stack([plain_llama.forward(cfg, w, toks)[-1] for toks in sequences]).double()


# (context, new tokens) of each request: five requests decoding, a short prompt, a decode step of matrix memories and of a delta rule
@pytest.mark.parametrize("shape,layers,lengths", [("1b", 4, [(880, 1), (610, 1), (340, 1), (777, 1), (512, 1)]), ("1b", 4, [(0, 9)]),
                                                  ("kobolix-1b", 3, [(20, 1)])])
def test_passes_agree(shape, layers, lengths):
    cfg = config(shape, layers)
    arch = architecture_for(cfg)
    typed = arch.config_class.from_dict(cfg)
    spec = arch.model_spec(typed)
    g = torch.Generator().manual_seed(layers)
    tokens = [torch.randint(0, spec.vocab, (c + n,), generator=g).tolist() for c, n in lengths]
    llm = LLM(config=typed, random_seed=3, dtype="float32", page_size=16, max_num_seqs=8, num_pages=400, max_model_len=1024, seed=0,
              cuda_graphs=False)
    runner, cache, K = llm.engine.runner, llm.engine.cache, kernels.load()
    ids = [f"r{i}" for i in range(len(tokens))]
    entries = [StepEntry(r, t[c:], [n - 1]) for r, t, (c, n) in zip(ids, tokens, lengths)]

    def one_pass():
        for r, t, (c, _) in zip(ids, tokens, lengths):       # (states of matrix memories cannot be cut back: stored anew)
            if not cache.has(r):
                cache.admit(r)
                if c:
                    runner.step([StepEntry(r, t[:c], [])])
        out = runner.step(entries).clone()
        for r, (c, _) in zip(ids, lengths):
            if c and shape == "1b":
                cache.truncate(r, c)
            else:
                cache.release(r)
        return out

    first = one_pass()
    want = oracle(cfg, arch, spec, 3, tokens)
    assert ((first - want).norm() / want.norm()).item() < 5e-5
    differ = torch.zeros((), device="cuda")
    for pause in (0.0, 0.005, 0.001):
        for _ in range(100):
            differ += (one_pass() != first).any()
            if pause:
                torch.cuda.synchronize()
                time.sleep(pause)
    was = K.set_pdl(False)
    for _ in range(20):
        differ += (one_pass() != first).any()
    K.set_pdl(was)
    assert differ.item() == 0 and K.gemm_status() == 0
