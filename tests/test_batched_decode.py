"""Batched decode: B independent sequences per launch, ragged lengths.

The reference has no kernel for this (its latency kernel decodes one sequence; its batched
instruction set needs batches that are multiples of 128, demos/throughput/instructions.py:30-31;
its torch path shares one length across the batch, llama.py:121-130), so the oracle is B
independent single-sequence runs of the pinned torch restatement on the same weights.
"""

import pytest
import torch

from megakernels_b200.demos.latency.instructions import (
    AttentionReduction,
    BatchAttention,
    PartialAttention,
    RMS_Norm,
)
from megakernels_b200.demos.latency.scheduler import LatencyScheduleBuilder, LatencyScheduleOptions
from megakernels_b200.llama import LlamaConfig, LlamaForCausalLM
from megakernels_b200.model_types import ExtraModelConfig
from megakernels_b200.scheduler import assign_to_sms, serialize_and_pad, tensorize_instructions
from megakernels_b200.utils import set_sm_count_override


def batched_schedule(cfg, batch, parts, max_len, device="cpu", draw_on="zeros"):
    extra = ExtraModelConfig(interleave_rope=True, max_len_override=max_len, max_batch_size=batch)
    model = LlamaForCausalLM.from_random(cfg, extra, device=device, seed=0, draw_on=draw_on)
    opts = LatencyScheduleOptions(num_attention_partitions=parts, coalesce_o_proj=True, batch_size=batch)
    schedule = LatencyScheduleBuilder(opts).build(model)
    tensorize_instructions(schedule.globs, assign_to_sms("rr", schedule=schedule))
    return model, schedule


def test_single_sequence_words_are_unchanged_by_the_batch_fields():
    """A sequence index of 0 lands in the zero padding: the padded words equal the reference's."""
    assert serialize_and_pad(PartialAttention(3, 5, 4, 2))[:7] == [2, 3, 5, 4, 2, 0, 0]
    assert serialize_and_pad(PartialAttention(3, 5, 4, 2, 6))[:7] == [2, 3, 5, 4, 2, 6, 0]
    words = serialize_and_pad(AttentionReduction(1, 8, 3, True, [0, 1, 2], None, 5))
    assert words[:11] == [3, 1, 8, 3, 1, 3, 0, 1, 2, 0, 5]
    assert serialize_and_pad(RMS_Norm(7, 1, 3))[:5] == [9, 7, 1, 3, 0]


@pytest.mark.parametrize("batch", [2, 8, 16])
def test_schedule_by_shares(batch):
    """What ``merge_in_last_partial`` schedules for a batch: every SM's share of every layer once, between its QKV and o-proj, no instruction per
    head; the words."""
    assert serialize_and_pad(BatchAttention(3, 17, 148))[:5] == [10, 3, 17, 148, 0]
    set_sm_count_override(148)
    extra = ExtraModelConfig(interleave_rope=True, max_len_override=64, max_batch_size=batch)
    cfg = LlamaConfig.llama_3_1_8b(num_hidden_layers=2, vocab_size=4096)
    model = LlamaForCausalLM.from_random(cfg, extra, device="cpu", seed=0, draw_on="zeros")
    opts = LatencyScheduleOptions(num_attention_partitions=1, coalesce_o_proj=True, batch_size=batch, merge_in_last_partial=True)
    schedule = LatencyScheduleBuilder(opts).build(model)
    ins = schedule.get_linear_instructions()
    assert not any(isinstance(i, (PartialAttention, AttentionReduction)) for i in ins)
    for layer in range(2):
        mine = [n for n, i in enumerate(ins) if isinstance(i, BatchAttention) and i.layer_idx == layer]
        assert [(ins[n].rank, ins[n].num_ranks) for n in mine] == [(r, 148) for r in range(148)]
        kind = lambda name: [n for n, i in enumerate(ins) if type(i).__name__ == name and i.layer_idx == layer]  # noqa: E731
        assert max(kind("LayerNorm_QKV_MatVecRopeAppend")) < min(mine) and max(mine) < min(kind("O_ProjResidual"))
    for mode in ("rr", "zz"):
        queues = assign_to_sms(mode, schedule=schedule)
        assert sorted((i.layer_idx, i.rank) for q in queues for i in q if isinstance(i, BatchAttention)) == [(m, r) for m in range(2) for r in range(148)]


def test_more_than_eight_sequences_schedule_blocks_of_128_rows():
    """The tcgen05 build multiplies blocks of 128 weight rows: block indices, counts and barrier
    thresholds of the schedule follow."""
    set_sm_count_override(148)
    cfg = LlamaConfig.llama_3_1_8b(num_hidden_layers=1, vocab_size=4096)
    _, schedule = batched_schedule(cfg, 16, 1, 64)
    g = schedule.globs
    assert (g.qkv_block_size, g.o_proj_block_size, g.up_gate_proj_block_size, g.down_proj_block_size,
            g.lm_head_block_size) == (128,) * 5
    th = g.barrier_thresholds()
    assert th["attn_waits_qkv_per_head"] == 1 and th["downproj_waits_upgate"] == 2048 // 128
    assert th["qkv_waits_downproj"] == (4096 // 128) * 7 and th["upgate_waits_oproj"] == (4096 // 128) * 2
    ins = schedule.get_linear_instructions()
    qkv = sorted(b for i in ins if type(i).__name__ == "LayerNorm_QKV_MatVecRopeAppend" for b in i.block_indices())
    assert qkv == list(range((32 + 16) * 128 // 128))
    up = sorted(b for i in ins if type(i).__name__ == "LayerNormDoubleMatVecSiLU" for b in i.block_idxs)
    assert up == list(range(14336 // 128))
    assert g.barriers.shape[2] >= 16 * 32


@pytest.mark.parametrize("batch,parts", [(4, 1), (8, 3)])
def test_batched_schedule_covers_every_sequence(batch, parts):
    set_sm_count_override(148)
    cfg = LlamaConfig.llama_3_1_8b(num_hidden_layers=2, vocab_size=4096)
    _, schedule = batched_schedule(cfg, batch, parts, 64)
    g = schedule.globs
    ins = schedule.get_linear_instructions()
    assert g.batch_size == batch and g.hidden_states.shape == (batch, cfg.hidden_size)
    assert g.residual_acc.shape == (batch, cfg.hidden_size) and g.normed_states.shape == (batch, cfg.hidden_size)
    assert g.barriers.shape[2] >= batch * cfg.num_attention_heads
    for layer in range(2):
        attn = {(i.batch_idx, i.kv_head_idx, i.partial_idx) for i in ins if isinstance(i, PartialAttention) and i.layer_idx == layer}
        assert attn == {(b, kv, p) for b in range(batch) for kv in range(cfg.num_key_value_heads) for p in range(parts)}
        reds = {(i.batch_idx, i.head_start_idx) for i in ins if isinstance(i, AttentionReduction) and i.layer_idx == layer}
        want = {(b, h) for b in range(batch) for h in range(0, cfg.num_attention_heads, 4)} if parts > 1 else set()
        assert reds == want
        norms = {(i.which, i.batch_idx) for i in ins if isinstance(i, RMS_Norm) and i.layer_idx == layer}
        assert norms >= {(w, b) for w in (0, 1) for b in range(batch)}
    assert sum(isinstance(i, RMS_Norm) and i.which == 2 for i in ins) == batch
    assert g.upgate_instructions_per_layer == 0
    # topological order: a sequence's attention follows the layer's QKV and precedes its o-proj
    order = [type(i).__name__ for i in ins if getattr(i, "layer_idx", None) == 0]
    assert order.index("PartialAttention") > order.index("LayerNorm_QKV_MatVecRopeAppend")
    assert order.index("O_ProjResidual") > len(order) - 1 - order[::-1].index("PartialAttention")


@pytest.mark.gpu
@pytest.mark.parametrize(
    "shape,batch,parts,merge",
    # up to 8 sequences: mma.sync with the sequences as B-operand columns; more: tcgen05 GEMMs
    # (128-row blocks, head_dim 128 only), incl. a batch that is not a multiple of the MMA's N step;
    # merge: no reduction instructions, the last partial of a (sequence, KV head) merges the rows
    [("8b", 4, 3, False), ("8b", 8, 1, False), ("1b", 5, 2, False), ("1b", 2, 4, False), ("8b", 16, 1, False),
     ("8b", 40, 2, False), ("8b", 64, 1, False), ("8b", 4, 3, True), ("1b", 5, 2, True), ("8b", 40, 2, True)],
)
def test_batched_decode_matches_independent_sequences(shape, batch, parts, merge):
    from megakernels_b200.generators import MK_Generator
    from oracle.llama_ref import TorchReferenceModel, assert_logits_parity
    from tests.gpu_utils import interpreter

    dev = "cuda:0"
    cfg = (LlamaConfig.llama_3_1_8b if shape == "8b" else LlamaConfig.llama_3_2_1b)(num_hidden_layers=2, vocab_size=4096)
    lens = torch.randint(5, 300, (batch,), generator=torch.Generator().manual_seed(4)).tolist()
    max_len = max(lens) + 8
    extra = ExtraModelConfig(interleave_rope=True, max_len_override=max_len, max_batch_size=batch)
    model = LlamaForCausalLM.from_random(cfg, extra, device=dev, seed=0, draw_on="device")
    gen = torch.Generator(device=dev).manual_seed(2)
    for c in model.stacked_kv_cache:  # N(0,1) prefix per sequence, poison beyond it
        c.copy_((torch.randn(c.shape, generator=gen, device=dev) * 100).to(c.dtype))
        for b, n in enumerate(lens):
            c[:, b, :n] = torch.randn(c[:, b, :n].shape, generator=gen, device=dev).to(c.dtype)
    # one copy of the weights on the host, one KV cache per sequence swapped in for its run
    ref = TorchReferenceModel(model, kv_len=max_len)
    caches = [tuple(c[:, b : b + 1].cpu().clone() for c in model.stacked_kv_cache) for b in range(batch)]
    opts = LatencyScheduleOptions(num_attention_partitions=parts, coalesce_o_proj=True, batch_size=batch,
                                  merge_in_last_partial=merge)
    schedule = LatencyScheduleBuilder(opts).build(model)
    tensorize_instructions(schedule.globs, assign_to_sms("rr", schedule=schedule))
    g = schedule.globs
    assert any(isinstance(i, AttentionReduction) for i in schedule.get_linear_instructions()) == (parts > 1 and not merge)
    mk = MK_Generator(model, interpreter(), schedule)
    ids = torch.randint(0, cfg.vocab_size, (3, batch), generator=torch.Generator().manual_seed(3))
    for step in range(3):
        pos = [n + step for n in lens]
        out = mk.run(ids[step].view(batch, 1).to(dev), pos)
        mk.check()
        assert out.shape == (batch,)
        for b in range(batch):
            ref.k_cache, ref.v_cache = caches[b]
            # 2e-2 / 0.999 as everywhere (the bounds never go below the stated values); with so
            # many (sequence, step) samples some top-2 pairs are one bf16 step apart, and for
            # those the float32 restatement says whether the oracle itself can tell them apart
            exact = ref.decode_token_exact(int(ids[step, b]), pos[b])
            want = ref.decode_token(int(ids[step, b]), pos[b])
            assert_logits_parity(g.logits[b], want, f"step {step}, sequence {b} at position {pos[b]}", exact=exact)
            assert int(out[b]) == int(torch.argmax(g.logits[b])), f"fused argmax, sequence {b}"
            # the appended K/V row, and nothing beyond it
            assert torch.equal(g.k_cache[:, b, pos[b] + 1 :].cpu(), ref.k_cache[:, 0, pos[b] + 1 :])


@pytest.mark.gpu
@pytest.mark.parametrize(
    "heads,kv_heads,head_dim,lens",
    # around a run of 16 positions, a stage and a warp's share of it; nothing cached; one sequence that most shares work on
    # (its parts are as many as there are rows for); two heads and one per stage; both builds
    [(32, 8, 128, [0, 1, 2]), (32, 8, 128, [15, 16, 17, 63, 64, 65, 7]), (32, 8, 128, [3000, 0, 40]), (32, 8, 64, [31, 32, 33, 500, 0]),
     (32, 4, 128, [400, 129]), (16, 2, 128, [700, 33, 0]), (8, 1, 128, [1500, 100]), (32, 8, 128, [(37 * i * i) % 900 for i in range(9)]),
     (32, 8, 128, [(131 * i) % 1100 for i in range(64)]), (16, 2, 128, [(53 * i) % 300 for i in range(12)]),
     # units of two heads (two long sequences) and of one (a long one beside a short one), in runs and at their edges
     (32, 8, 128, [2600, 2500]), (32, 8, 128, [3500, 20]), (32, 8, 64, [5003, 4000]), (32, 8, 64, [9001, 0]), (16, 2, 128, [4097, 64])],
)
def test_attention_by_shares_matches_attention_by_sequence(heads, kv_heads, head_dim, lens):
    """What a layer's attention leaves, by shares and by an instruction per sequence and head.  Softmax weights are
    rounded to bf16 on either side, relative to other running maxima, and so are the results: three roundings of 2^-9."""
    from megakernels_b200.generators import MK_Generator
    from tests.gpu_utils import interpreter

    dev, batch = "cuda:0", len(lens)
    cfg = LlamaConfig.llama_3_1_8b(
        num_hidden_layers=1, vocab_size=4096, hidden_size=2048, intermediate_size=2048, num_attention_heads=heads,
        num_key_value_heads=kv_heads, head_dim=head_dim)
    extra = ExtraModelConfig(interleave_rope=True, max_len_override=max(lens) + 8, max_batch_size=batch)
    model = LlamaForCausalLM.from_random(cfg, extra, device=dev, seed=0, draw_on="device")
    gen = torch.Generator(device=dev).manual_seed(2)
    ids = torch.randint(0, cfg.vocab_size, (batch, 1), generator=torch.Generator().manual_seed(3)).to(dev)
    prefix = [torch.randn(c.shape, generator=gen, device=dev).to(c.dtype) for c in model.stacked_kv_cache]
    outs = []
    for merge in (True, False):
        for c, x in zip(model.stacked_kv_cache, prefix):
            c.copy_(x)
        opts = LatencyScheduleOptions(coalesce_o_proj=True, batch_size=batch, merge_in_last_partial=merge)
        schedule = LatencyScheduleBuilder(opts).build(model)
        kinds = {type(i).__name__ for i in schedule.get_linear_instructions()}
        assert ("BatchAttention" in kinds, "PartialAttention" in kinds) == (merge, not merge)
        tensorize_instructions(schedule.globs, assign_to_sms("rr", schedule=schedule))
        mk = MK_Generator(model, interpreter(), schedule)
        for _ in range(2):
            mk.run(ids, lens)
        mk.check()
        outs.append(schedule.globs.attn_out.float().clone())
    for b in range(batch):
        assert float((outs[0][b] - outs[1][b]).norm() / outs[1][b].norm()) < 3 * 2.0**-9, f"sequence {b} of length {lens[b]}"


@pytest.mark.parametrize("seed", range(6))
def test_shares_cover_every_stage_once(seed):
    """Whatever the positions, heads, rows of parts, SMs and shares: a unit's parts are its stages, numbered, no more than there are rows for; a
    share cuts at most two units."""
    import random

    from oracle.attention_shares import LineUp

    rng = random.Random(seed)
    for _ in range(150):
        batch, top = rng.choice([2, 2, 3, 5, 8, 9, 33, 64]), rng.choice([1, 40, 300, 4096, 20000, 131072])
        positions = [rng.choice([0, top, rng.randint(0, top), 15, 16, 17]) for _ in range(batch)]
        kv_heads, head_dim = rng.choice([1, 2, 4, 6, 8, 8, 12]), rng.choice([64, 128])
        rows, sms = rng.choice([24, 24, 148, 1, 2, 10]), rng.choice([148, 148, 132, 8])
        ranks = rng.choice([sms, sms, sms // 2, sms + 5, 1])
        line, seen = LineUp.of(positions, kv_heads, head_dim, rows, sms), {}
        for rank in range(ranks):
            pieces = line.pieces(rank, ranks)
            assert sum(p.parts > 1 for p in pieces) <= 2
            for p in pieces:
                assert p.parts <= max(1, min(24, rows)) and (p.last > p.first or p.stages == 0)
                seen.setdefault((p.seq, p.head), []).append(p)
        assert len(seen) == batch * kv_heads // line.heads
        for parts in seen.values():
            parts.sort(key=lambda p: p.part)
            assert [p.part for p in parts] == list(range(len(parts))) and {p.parts for p in parts} == {len(parts)}
            assert parts[0].first == 0 and parts[-1].last == parts[0].stages
            assert all(a.last == b.first for a, b in zip(parts, parts[1:]))


@pytest.mark.parametrize("positions", [[4096, 4096], [16384, 16384], [16384, 40], [16384, 40, 40], [4096] * 3, [9000, 300, 300, 300], [2000] * 8])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_shares_of_few_sequences_reach_the_sms(positions, head_dim):
    """Units of four heads of two equal sequences fall into 92 shares, of a long one beside short ones into 46: then units are smaller.
    At least 85 % of 148 SMs hold cached positions (with few stages per SM some shares are a unit's own cost)."""
    from oracle.attention_shares import LineUp

    line = LineUp.of(positions, 8, head_dim, 24, 148)
    work = [sum(p.last - p.first for p in line.pieces(r, 148)) for r in range(148)]
    assert sum(w > 0 for w in work) >= 0.85 * 148 or max(work) <= 8
    assert max(work) <= 1.35 * sum(work) / 148 + 12


@pytest.mark.parametrize("heads,kv_heads,head_dim,positions", [(8, 2, 64, [0, 40, 700]), (8, 1, 128, [300, 17]), (32, 8, 128, [150, 0])])
def test_attention_by_shares_is_attention(heads, kv_heads, head_dim, positions):
    """The parts of all shares, merged by their sums of exponentials, against softmax attention in 64 bits."""
    from oracle.attention_shares import attend

    gen = torch.Generator().manual_seed(1)
    q, T = torch.randn(len(positions), heads, head_dim, generator=gen), max(positions) + 1
    k, v = (torch.randn(len(positions), T, kv_heads, head_dim, generator=gen) for _ in range(2))
    got = attend(q, k, v, positions, head_dim**-0.5, 24, 148, 148)
    for b, p in enumerate(positions):
        for h in range(heads):
            kv = h * kv_heads // heads
            score = k[b, : p + 1, kv].double() @ q[b, h].double() * head_dim**-0.5
            assert torch.allclose(got[b, h], torch.softmax(score, 0) @ v[b, : p + 1, kv].double(), rtol=1e-12, atol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,head_dim,lens,parts", [
    (32, 8, 64, [31, 500, 0, 64, 200], 2), (32, 8, 128, [17, 900, 128, 300], 3), (16, 2, 128, [700, 33], 5), (32, 8, 128, [(37 * i) % 300 for i in range(40)], 2)])
def test_last_partial_of_a_batch_merges(heads, kv_heads, head_dim, lens, parts):
    """Instructions per sequence and head whose last part to arrive merges (what a caller of the C interface may still schedule with
    skip_attn_reduction = 2) leave what reduction instructions leave: both merge in 32 bits and round to bf16 once."""
    from megakernels_b200.generators import MK_Generator
    from tests.gpu_utils import interpreter

    dev, batch = "cuda:0", len(lens)
    cfg = LlamaConfig.llama_3_1_8b(
        num_hidden_layers=1, vocab_size=4096, hidden_size=2048, intermediate_size=2048, num_attention_heads=heads,
        num_key_value_heads=kv_heads, head_dim=head_dim)
    extra = ExtraModelConfig(interleave_rope=True, max_len_override=max(lens) + 8, max_batch_size=batch)
    model = LlamaForCausalLM.from_random(cfg, extra, device=dev, seed=0, draw_on="device")
    gen = torch.Generator(device=dev).manual_seed(2)
    ids = torch.randint(0, cfg.vocab_size, (batch, 1), generator=torch.Generator().manual_seed(3)).to(dev)
    prefix = [torch.randn(c.shape, generator=gen, device=dev).to(c.dtype) for c in model.stacked_kv_cache]
    outs = []
    for merge in (True, False):
        for c, x in zip(model.stacked_kv_cache, prefix):
            c.copy_(x)
        opts = LatencyScheduleOptions(num_attention_partitions=parts, coalesce_o_proj=True, batch_size=batch)
        schedule = LatencyScheduleBuilder(opts).build(model)
        queues = assign_to_sms("rr", schedule=schedule)
        assert any(isinstance(i, AttentionReduction) for q in queues for i in q)
        if merge:
            queues = [[i for i in q if not isinstance(i, AttentionReduction)] for q in queues]
            schedule.globs.merge_in_last_partial = True
        tensorize_instructions(schedule.globs, queues)
        mk = MK_Generator(model, interpreter(), schedule)
        for _ in range(2):
            mk.run(ids, lens)
        mk.check()
        outs.append(schedule.globs.attn_out.float().clone())
    for b in range(batch):
        assert float((outs[0][b] - outs[1][b]).norm() / outs[1][b].norm()) < 2 * 2.0**-9, f"sequence {b} of length {lens[b]}"
