"""What a float32 step takes beside its workspace: the bfloat16 pieces of the rows of every product (csrc/gemm_f32_tc.cu), 6 bytes a number,
allocated and given back by each product."""
import pytest
import torch

from iitj_llm_coopt_b200 import LLM, StepEntry
from iitj_llm_coopt_b200.config.registry import architecture_for
from iitj_llm_coopt_b200.engine.llm import workspace_bytes_estimate
from iitj_llm_coopt_b200.presets import shape_config


def spec_of(shape):
    cfg = shape_config(shape)
    arch = architecture_for(cfg)
    return arch.model_spec(arch.config_class.from_dict(cfg))


# the longest row of a product: the inner width, or with routed experts the chosen rows of the wider of inner width and stream
@pytest.mark.parametrize("shape,longest", [("1b", 8192), ("8b", 14336), ("kobolix-1b", 2 * 4096), ("lifusun-1b", 8192)])
def test_the_estimate_counts_the_pieces(shape, longest):
    spec = spec_of(shape)
    per_token = {size: (workspace_bytes_estimate(spec, 2048, 8, size) - workspace_bytes_estimate(spec, 1024, 8, size)) / 1024 for size in (2, 4)}
    rest = 2 * per_token[2] - 2 * 4 * spec.width          # (the stream is float32 in both types)
    assert per_token[4] - rest >= 2 * 6 * longest


@pytest.mark.gpu
def test_captured_prompt_steps_share_the_pieces():
    cfg = dict(shape_config("1b"), num_hidden_layers=2)
    typed = architecture_for(cfg).config_class.from_dict(cfg)
    llm = LLM(config=typed, random_seed=1, dtype="float32", page_size=16, max_num_seqs=8, num_pages=200, max_model_len=1024, seed=0)
    runner, cache = llm.engine.runner, llm.engine.cache
    assert runner.use_graphs
    seen, results = [], {}
    for n in (640, 632, 624, 616, 608, 600):
        tokens = torch.randint(0, 1000, (n,), generator=torch.Generator().manual_seed(n)).tolist()
        for i in range(7):
            cache.admit("r")
            logits = runner.step([StepEntry("r", tokens, [n - 1])])
            results.setdefault(n, logits.clone())
            assert torch.equal(logits, results[n])        # eager, while it is captured, and replayed
            cache.release("r")
        torch.cuda.synchronize()
        seen.append(torch.cuda.memory_reserved())
    assert runner.graph_captures == 6
    assert seen[-1] - seen[0] < 6 * 600 * 8192            # less than one more set of pieces, and not five
