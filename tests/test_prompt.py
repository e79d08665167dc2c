"""Prompts of llama models: all tokens at once against one decode step per token and the oracle."""

import ctypes

import pytest
import torch

from megakernels_b200.demos.latency.mk import interpret_with_mk
from megakernels_b200.demos.latency.scheduler import LatencyScheduleOptions, covers_model
from megakernels_b200.llama import LlamaConfig
from megakernels_b200.scheduler import assign_to_sms, tensorize_instructions
from megakernels_b200.native import mk_llama
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
    for options in (None, LatencyScheduleOptions(num_attention_partitions=3, coalesce_o_proj=True, merge_in_last_partial=True),
                    LatencyScheduleOptions(num_attention_partitions=2)):
        schedule = build_schedule(model, options)
        instructions = schedule.get_linear_instructions()
        assert covers_model(schedule.globs, instructions)
        tensorize_instructions(schedule.globs, assign_to_sms("rr", schedule=schedule))
        assert covers_model(schedule.globs, schedule.globs.instructions)
        of_kind = {type(x): i for i, x in enumerate(instructions)}  # the last one of each
        assert len(of_kind) == 6 + (not schedule.globs.skip_attn_reduction and not schedule.globs.merge_in_last_partial)
        for kind, at in [*of_kind.items(), (None, 0), (None, len(instructions) // 2)]:
            rest = instructions[:at] + instructions[at + 1 :]
            assert not covers_model(schedule.globs, rest), kind
            # one twice, also in another's place: as many blocks as before
            assert not covers_model(schedule.globs, instructions + [instructions[at]]), kind
            other = next(i for i, x in enumerate(instructions) if type(x) is type(instructions[at]) and i != at)
            assert not covers_model(schedule.globs, rest + [instructions[other]]), kind
        edited = schedule.globs.instructions.clone()
        sm, place = (edited[:, :, 0] == 2).nonzero()[0].tolist()
        edited[sm, place] = 0  # a no-op where attention was
        assert not covers_model(schedule.globs, edited)
    for kw in (dict(layer_limit=1), dict(stop_after_op="oproj")):
        schedule = build_schedule(model, **kw)
        assert not covers_model(schedule.globs, schedule.get_linear_instructions())


# portions of 1 (a lone last token), rows of a 128-row tile and their remainders, keys over several tiles; short last
# portions over 512 keys and more, whose tiles a cluster shares
@pytest.mark.gpu
@pytest.mark.parametrize("shape,count,portion", [
    ("1b", 2, 2048), ("1b", 4, 2048), ("1b", 128, 2048), ("1b", 129, 128), ("1b", 300, 2048), ("8b", 61, 2048), ("8b", 257, 100), ("70b", 130, 2048),
    ("1b", 620, 560), ("1b", 700, 100), ("1b", 561, 560), ("8b", 641, 100), ("70b", 530, 520),
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


def own_weight_model(seed):
    """One layer at the 1B widths in which head j's attention leaves ``p_j sum |v_j| - h_j`` in element j of the residual
    stream and then in logit j, exact but for the attention's own rounding: other positions' values and the
    feed-forward are zero, ``h_j`` (the last token's embedding) takes off nearly all of it."""
    model = build_model(CONFIGS["1b"](num_hidden_layers=1), 700, device="cuda")
    globs = build_schedule(model).globs
    tensorize_instructions(globs, assign_to_sms("rr", instructions=[], sm_count=globs.sm_count()))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    draw = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")  # noqa: E731
    H, D, Hq, Hkv = 2048, 64, 32, 8
    for name in ("qkv_proj_weights", "o_proj_weights", "down_proj_weights"):
        getattr(globs, name).zero_()
    for w in (globs.attn_ln_weights, globs.mlp_ln_weights, globs.lm_head_norm_weights):
        w.fill_(1.0)
    wk = draw(Hkv, D, H) * (2.0 * (H / 2)) ** -0.5
    wk[:, :, :Hq] = 0
    gain = torch.tensor([0.125, 0.25, 0.09, 0.19], device="cuda")  # own scores of about -8 gain: never a row's maximum
    wq = -(gain.view(1, 4, 1, 1) * wk.view(Hkv, 1, D, H)).reshape(Hq * D, H)
    wv = draw(Hkv * D, H) * 3e-4  # (so that h_j hardly counts in the row's norm)
    wv[:, : H // 2] = 0  # only the last token's embedding lies there
    globs.qkv_proj_weights[0] = torch.cat([wq, wk.view(-1, H), wv])
    globs.lm_head_weights.zero_()
    globs.lm_head_weights[:Hq, :Hq].fill_diagonal_(1.0)
    return model, globs, draw


@pytest.mark.gpu
@pytest.mark.parametrize("count,cached", [(2, 0), (3, 0), (130, 0), (2, 640), (40, 600)])
def test_own_key_keeps_its_32_bit_weight(count, cached):
    """A query's softmax weight of its own position is 32-bit, as in the step per token.  Rounding it to bf16 (up to 2^-8,
    0.4 of that in the mean square) would move all entries of a head alike; the attention output's own rounding to bf16,
    of that size too, moves each by itself, and the mean over 64 entries weighted by |v| (as good as 41 equal
    ones) moves by 0.4 2^-8 / 6.4."""
    model, globs, draw = own_weight_model(seed=count + cached)
    H, D, Hq, Hkv = 2048, 64, 32, 8
    for c in model.stacked_kv_cache:
        c.zero_()
    hidden = torch.zeros(count, H, device="cuda", dtype=torch.bfloat16)
    hidden[:-1, Hq : H // 2] = draw(count - 1, H // 2 - Hq).bfloat16()
    hidden[-1, H // 2 :] = draw(H // 2).bfloat16()
    at = cached + torch.arange(count, device="cuda")
    cos, sin = globs.rope_cos[at].double(), globs.rope_sin[at].double()
    rounded = lambda x: x.to(torch.bfloat16).double()  # noqa: E731
    w = globs.qkv_proj_weights[0].double()
    for _ in range(3):  # (h_j changes the row's norm a little)
        x = hidden.double()
        act = rounded(x / (x.pow(2).mean(-1, keepdim=True) + globs.rms_norm_eps).sqrt())
        q, k, v = (act @ w.T).split([Hq * D, Hkv * D, Hkv * D], dim=-1)
        turned = []
        for y, heads in ((q, Hq), (k, Hkv)):
            y = y.view(count, heads, D // 2, 2)
            c, s = cos.view(count, 1, D // 2, 2), sin.view(count, 1, D // 2, 2)
            turned.append(rounded(torch.stack([y[..., 0] * c[..., 0] - y[..., 1] * s[..., 0],
                                               y[..., 1] * c[..., 1] + y[..., 0] * s[..., 1]], -1)).view(count, heads, D))
        q, k, v = turned[0][-1], turned[1].repeat_interleave(Hq // Hkv, 1), rounded(v[-1]).view(Hkv, D).repeat_interleave(Hq // Hkv, 0)
        score = torch.cat([torch.zeros(Hq, cached, device="cuda", dtype=torch.float64), torch.einsum("hd,thd->ht", q, k) * globs.attn_scale], 1)
        p = torch.softmax(score, -1)[:, -1]
        assert (score[:, -1] < score.amax(-1)).all()
        signs = v.sign()
        globs.o_proj_weights[0, :Hq] = torch.block_diag(*signs.float().unsqueeze(1)).bfloat16()
        whole = p * (signs * v).sum(-1)
        hidden[-1, :Hq] = -whole.bfloat16()
    x = hidden[-1].double()
    x[:Hq] += whole
    logits_scale = 1 / (x.pow(2).mean() + globs.rms_norm_eps).sqrt()
    interpreter().module.sync_status(interpreter().prompt(globs, hidden, cached, True))
    error = (globs.logits[:Hq].double().view(-1) / logits_scale - x[:Hq]) / whole
    assert float(error.pow(2).mean().sqrt()) < 2 * 0.4 * 2.0**-8 / 6.4, error


@pytest.mark.gpu
@pytest.mark.parametrize("shape,count,portion", [("1b", 2, 2048), ("8b", 61, 2048), ("1b", 300, 128), ("1b", 400, 2048)])
def test_residual_stream_of_the_last_token(shape, count, portion):
    """As after a step: embedding plus the exact sum, in steps of 2^-32, of what the layers added (fp32 sums would
    have lost the low bits of the smaller terms)."""
    from megakernels_b200.generators import MK_Generator

    _, _, model, schedule = make_pair(CONFIGS[shape](), count, 0)
    globs = schedule.globs
    ids = torch.tensor(seeded_tokens(globs.vocab_size, count, seed=6)).cuda()
    gen = MK_Generator(model, interpreter(), schedule)
    gen.prompt_portion = portion
    for pos in range(count):
        gen.run(ids[pos].view(1, 1), pos)
    gen.check()
    want, hidden = globs.residual_stream(), globs.hidden_states.clone()
    globs.residual_acc.fill_(1 << 40)
    gen.prefill(ids)
    gen.check()
    assert torch.equal(globs.hidden_states, hidden)
    assert rel_err(globs.residual_stream(), want) <= 2e-2
    sums = globs.residual_acc.double() * 2.0**-32
    assert (sums.float().double() != sums).float().mean() > 0.25


@pytest.mark.gpu
def test_edited_or_replaced_instructions_run_as_steps():
    from megakernels_b200.generators import MK_Generator

    _, _, model, schedule = make_pair(CONFIGS["1b"](), 40, 0)
    globs = schedule.globs
    gen = MK_Generator(model, interpreter(), schedule)
    assert gen._takes_prompts(8)
    whole, globs.instructions = globs.instructions, globs.instructions.clone()
    assert not gen._takes_prompts(8)
    globs.instructions = whole
    assert gen._takes_prompts(8)
    globs.instructions[globs.instructions[:, :, 0] == 2] = 0
    assert not gen._takes_prompts(8)
    assert not MK_Generator(model, interpreter(), schedule)._takes_prompts(8)


@pytest.mark.gpu
@pytest.mark.parametrize("as_handle", [False, True])
def test_prompt_on_another_stream_keeps_its_workspace(as_handle):
    """The launches wait on a busy stream; what the current stream allocates and fills meanwhile is other memory."""
    from megakernels_b200.generators import MK_Generator

    count = 200
    _, _, model, schedule = make_pair(CONFIGS["1b"](), count, 0)
    globs = schedule.globs
    MK_Generator(model, interpreter(), schedule)
    module = interpreter().module
    embed = model.model.embed_tokens.embed_tokens.weight
    ids = torch.tensor(seeded_tokens(globs.vocab_size, count, seed=7)).cuda()
    globs.pos_id = count - 1

    def prompt(hidden, stream):
        return interpret_with_mk(globs, lambda *args, **kw: module.mk_llama_prompt(
            *args, hidden=hidden, pos0=0, want_logits=True, **{**kw, "stream": stream}))

    module.sync_status(prompt(embed[ids], None))
    want = globs.logits.clone()
    globs.logits.zero_()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)  # some 50 ms
    call = prompt(embed[ids], side.cuda_stream if as_handle else side)
    assert not side.query()
    junk = [torch.full((1 << k,), 255, dtype=torch.uint8, device="cuda") for k in range(16, 25) for _ in range(4)]  # every size up to 16 MB
    torch.cuda.current_stream().synchronize()
    module.sync_status(call, stream=side)
    assert torch.equal(globs.logits, want)
    del junk


def test_prompts_record_no_timings():
    lib = mk_llama.load_library()
    g, p = mk_llama.MkbGlobals(), mk_llama.MkbPrompt(struct_bytes=ctypes.sizeof(mk_llama.MkbPrompt))
    g.flags = mk_llama.MKB_FLAG_RECORD_TIMINGS
    assert lib.mkb_prompt(ctypes.byref(g), ctypes.byref(p), None) == 5  # MKB_ERR_UNSUPPORTED
    assert "timings" in lib.mkb_last_error().decode()


@pytest.mark.gpu
def test_prompt_honours_the_wait_limit():
    """A tile whose inner dimension takes longer than the limit: the epilogue's wait for it gives up and the status says so."""
    model = build_model(CONFIGS["1b"](num_hidden_layers=1), 2048, device="cuda")
    globs = build_schedule(model).globs
    tensorize_instructions(globs, assign_to_sms("rr", instructions=[], sm_count=globs.sm_count()))
    wide = 200 * 2048  # 6,400 steps of at least 0.26 us (the tensor cores' rate) where the feed-forward comes back
    up = torch.zeros(1, wide, 2048, device="cuda", dtype=torch.bfloat16)
    globs.up_proj_weights = globs.gate_proj_weights = up
    globs.down_proj_weights = up.view(1, 2048, wide)
    globs.silu_out = torch.zeros(wide, device="cuda", dtype=torch.bfloat16)
    globs.barriers = torch.zeros(1, globs.barriers.shape[1], 256, device="cuda", dtype=torch.int32)
    hidden = torch.randn(2048, 2048, device="cuda").bfloat16()
    module, globs.pos_id = interpreter().module, 2047

    def prompt(**kw):
        call = interpret_with_mk(globs, lambda *args, **rest: module.mk_llama_prompt(
            *args, hidden=hidden, pos0=0, want_logits=True, **rest, **kw))
        return module.sync_status(call)

    prompt()
    with pytest.raises(RuntimeError, match="TIMEOUT"):
        prompt(wait_timeout_ms=1)
    prompt()  # the device and the status record are as before


@pytest.mark.gpu
def test_prompt_takes_what_steps_take():
    """Whole numbers of any type into a captured step's generator, embeddings kept in another type than the kernel's."""
    from megakernels_b200.generators import MK_Generator

    _, _, model, schedule = make_pair(CONFIGS["1b"](), 40, 0)
    gen = MK_Generator(model, interpreter(), schedule)
    ids = torch.tensor(seeded_tokens(4096, 12))
    want = gen.prefill(ids.cuda())
    embed = model.model.embed_tokens.embed_tokens
    embed.weight = embed.weight.float()
    assert torch.equal(gen.prefill(ids.cuda()), want)
    gen.enable_cuda_graph(warmup_pos=3)
    assert gen._takes_prompts(12)
    assert torch.equal(gen.prefill(ids.to(torch.int16)), want)
    gen.check()


@pytest.mark.gpu
@pytest.mark.parametrize("fits", [0, 1])
def test_prompt_without_memory_for_a_portion_goes_by_steps(fits, monkeypatch):
    from megakernels_b200.generators import MK_Generator

    _, _, model, schedule = make_pair(CONFIGS["1b"](), 40, 0)
    gen = MK_Generator(model, interpreter(), schedule)
    gen.prompt_portion = 16
    ids = torch.tensor(seeded_tokens(4096, 40)).cuda()
    want = [gen.prefill(ids).clone(), schedule.globs.logits.clone()]
    calls, prompt = [], interpreter().prompt

    def short(*args):
        calls.append(args)
        if len(calls) > fits:
            raise torch.OutOfMemoryError("no room")
        return prompt(*args)

    monkeypatch.setattr(interpreter(), "prompt", short)
    assert torch.equal(gen.prefill(ids), want[0])
    gen.check()
    assert len(calls) == fits + 1 and schedule.globs.pos_id == 39
    assert rel_err(schedule.globs.logits, want[1]) <= 2e-2


@pytest.mark.gpu
def test_prompt_under_capture():
    """Captured into a graph, a prompt's launches (which may begin early) give the same bits on replay with other tokens."""
    from megakernels_b200.generators import MK_Generator

    _, _, model, schedule = make_pair(CONFIGS["1b"](), 300, 0)
    globs = schedule.globs
    gen = MK_Generator(model, interpreter(), schedule)
    first, second = (torch.tensor(seeded_tokens(globs.vocab_size, 300, seed=s)).cuda() for s in (8, 9))
    want = [gen.prefill(second).clone(), globs.logits.clone(), *(c.clone() for c in model.stacked_kv_cache)]
    ids = first.clone()
    gen.prefill(ids)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        token = gen.prefill(ids)
    ids.copy_(second)
    graph.replay()
    gen.check()
    for got, w in zip([token, globs.logits, *model.stacked_kv_cache], want):
        assert torch.equal(got, w)
