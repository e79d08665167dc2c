"""Prompts of llama models: all tokens at once against one decode step per token and the oracle."""

import pytest
import torch

from megakernels_b200.demos.latency.scheduler import LatencyScheduleOptions, covers_model
from megakernels_b200.llama import LlamaConfig
from oracle.llama_ref import TorchReferenceModel, assert_logits_parity
from tests.gpu_utils import interpreter, make_pair, rel_err
from tests.oracle_utils import build_model, build_schedule, seeded_tokens

CONFIGS = {
    "1b": lambda **kw: LlamaConfig.llama_3_2_1b(**{"num_hidden_layers": 2, "vocab_size": 4096, **kw}),
    "8b": lambda **kw: LlamaConfig.llama_3_1_8b(**{"num_hidden_layers": 2, "vocab_size": 4096, **kw}),
    "70b": lambda **kw: LlamaConfig.llama_3_1_70b(**{"num_hidden_layers": 1, "vocab_size": 4096, **kw}),
}


def test_only_whole_schedules_count_as_the_model():
    model = build_model(CONFIGS["1b"](), 64)
    for options in (None, LatencyScheduleOptions(num_attention_partitions=3, coalesce_o_proj=True, merge_in_last_partial=True)):
        schedule = build_schedule(model, options)
        instructions = schedule.get_linear_instructions()
        assert covers_model(schedule.globs, instructions)
        for dropped in (0, len(instructions) // 2, -1):
            rest = [x for i, x in enumerate(instructions) if i != dropped % len(instructions)]
            kind = type(instructions[dropped]).__name__
            assert covers_model(schedule.globs, rest) == (kind in ("PartialAttention", "AttentionReduction")), kind
    for kw in (dict(layer_limit=1), dict(stop_after_op="oproj")):
        schedule = build_schedule(model, **kw)
        assert not covers_model(schedule.globs, schedule.get_linear_instructions())


# portions of 1 (a lone last token), rows of a 128-row tile and their remainders, keys over several tiles
@pytest.mark.gpu
@pytest.mark.parametrize("shape,count,portion", [
    ("1b", 2, 2048), ("1b", 4, 2048), ("1b", 128, 2048), ("1b", 129, 128), ("1b", 300, 2048), ("8b", 61, 2048), ("8b", 257, 100), ("70b", 130, 2048),
])
def test_prompt_equals_a_step_per_token(shape, count, portion):
    """Caches and logits within the decode path's own distance from the oracle (2e-2, two layers);
    nothing beyond the prompt is written."""
    from megakernels_b200.generators import MK_Generator

    cpu_model, _, model, schedule = make_pair(CONFIGS[shape](), count + 9, 0, poison=True)
    globs = schedule.globs
    ids = torch.tensor(seeded_tokens(globs.vocab_size, count, seed=4))
    gen = MK_Generator(model, interpreter(), schedule)
    gen.prompt_portion = portion
    assert gen._takes_prompts(count)
    before = [c.clone() for c in model.stacked_kv_cache]
    for pos in range(count):
        last = gen.run(ids[pos].view(1, 1).cuda(), pos)
    want = [c.clone() for c in model.stacked_kv_cache] + [globs.logits.clone(), last.clone()]
    for c, b in zip(model.stacked_kv_cache, before):
        c.copy_(b)
    token = gen.prefill(ids.cuda())
    gen.check()
    assert torch.equal(token, torch.argmax(globs.logits).view(1)) and torch.equal(globs.argmax_out.long(), token)
    for c, w, b in zip(model.stacked_kv_cache, want, before):
        assert rel_err(c[:, 0, :count], w[:, 0, :count]) <= 2e-2
        assert torch.equal(c[:, 0, count:], b[:, 0, count:])
    assert rel_err(globs.logits, want[2]) <= 2e-2
    if shape == "1b":
        ref = TorchReferenceModel(cpu_model)
        for pos, tok in enumerate(ids.tolist()):
            logits = ref.decode_token(tok, pos)
        assert_logits_parity(globs.logits, logits, "after the prompt")
    # decoding goes on from the prompt's cache
    step = gen.run(token.view(1, 1), count)
    gen.check()
    assert int(step) == int(torch.argmax(globs.logits))


@pytest.mark.gpu
def test_calls_that_stay_a_step_per_token():
    from megakernels_b200.generators import MK_Generator

    _, _, model, schedule = make_pair(CONFIGS["1b"](), 40, 0)
    gen = MK_Generator(model, interpreter(), schedule)
    assert gen._takes_prompts(40) and not gen._takes_prompts(41) and not gen._takes_prompts(1)
    with pytest.raises(Exception, match="41|40"):  # as a step beyond the cache
        gen.prefill(torch.zeros(41, dtype=torch.long, device="cuda"))

    class Own(MK_Generator):
        def run(self, input_ids, pos_id):
            return super().run(input_ids, pos_id)

    assert not Own(model, interpreter(), schedule)._takes_prompts(8)
    gen.enable_cuda_graph(warmup_pos=3)
    ids = torch.tensor(seeded_tokens(4096, 12)).cuda()
    token = gen.prefill(ids)
    replayed = gen.run(ids[-1:].view(1, 1), 11)  # the last token again: the same logits from the captured step
    assert int(replayed) == int(torch.argmax(schedule.globs.logits)) == int(token)
    gen.replace_with_noops()
    assert not gen._takes_prompts(12)
