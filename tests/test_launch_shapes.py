"""Decisions that are made on the host before a kernel is launched: how the streaming product cuts its
blocks, which tile size the experts get.  No GPU and no compiled library is needed for these."""
import pytest


def test_streaming_blocks_stay_inside_a_block_of_sixteen_warps():
    from fieldrun_b200.csrc import ops
    for tiles in (1, 8, 57, 220, 4000):
        for features, inner in ((8192, 3072), (3072, 6144), (1536, 3072), (3072, 1536), (48, 64), (16, 32)):
            for tile_rows in (8, 16, 32):
                for paired in (False, True):
                    shape = ops.stream_shape(tiles, features, inner, tile_rows, paired)
                    assert shape["groups"] in (1, 2, 4) and shape["splits"] >= 1
                    assert shape["splits"] * shape["groups"] * (tile_rows // 8) <= 16
                    # a part of the inner size is a multiple of 128, so at most inner / 128 parts have work
                    assert shape["splits"] <= max(1, inner // 128)


def test_streaming_blocks_cut_the_inner_size_more_when_there_are_few_tiles():
    from fieldrun_b200.csrc import ops
    one_layer = ops.stream_shape(1, 3072, 6144, 8)["splits"]          # a dense layer: one "expert"
    many = ops.stream_shape(220, 3072, 1536, 8)["splits"]
    assert one_layer > many >= 2


@pytest.mark.parametrize("assignments,decode,tensor_cores,expected", [
    (8, True, False, 8), (64, True, False, 8), (512, True, False, 8), (1024, True, False, 8), (1536, True, True, 32),
    (64, False, False, 8), (256, False, False, 8), (512, False, True, 32), (3000, False, True, 32), (10000, False, True, 64),
    (131072, False, True, 256)])
def test_experts_get_tiles_by_the_rows_an_expert_sees(assignments, decode, tensor_cores, expected):
    """256 experts: decode steps stream with tiles of 8 rows up to 4 rows per expert on average, prompts up to 1
    (their tokens crowd on fewer experts); beyond, tcgen05 with tiles of 32 rows and more."""
    import torch
    from fieldrun_b200.config import PartSpec
    from fieldrun_b200.parts import build_part
    spec = PartSpec("routed_experts", {"hidden_size": 128, "num_experts": 256, "top_k": 8, "expert_width": 128,
                                       "scoring": "sigmoid", "renormalize": True, "routed_scale": 1.0, "use_bias": True},
                    {"router": "r", "bias": "b", "w1": "e.{e}.w1", "w3": "e.{e}.w3", "w2": "e.{e}.w2"})
    part = build_part("feed_forward", spec, torch.bfloat16)
    assert part.on_tensor_cores(assignments, decode) == tensor_cores
    assert part.tile_rows(assignments, decode) == expected


def test_float32_products_of_operands_that_do_not_fit_are_left_to_the_library():
    """The kernels take their sizes from the weight: rows of another length, a result of another shape or type and operands in
    pieces must not reach them (the library refuses the first two, and takes the last)."""
    import torch
    from fieldrun_b200.parts.linear import float32_kernels_read
    rows, weight = torch.zeros(6, 96), torch.zeros(32, 96)
    assert float32_kernels_read(rows, weight, None) and float32_kernels_read(rows, weight, torch.zeros(6, 32))
    for other_rows, other_weight, out in ((torch.zeros(6, 64), weight, None), (rows, torch.zeros(32, 128), None), (rows[0], weight, None),
                                          (rows, weight, torch.zeros(5, 32)), (rows, weight, torch.zeros(6, 31)), (rows, weight, torch.zeros(6 * 32)),
                                          (rows, weight, torch.zeros(6, 32, dtype=torch.float64)), (rows, weight, torch.zeros(32, 6).t()),
                                          (torch.zeros(96, 6).t(), weight, None), (rows, torch.zeros(96, 32).t(), None), (rows[:0], weight, None),
                                          (torch.zeros(6 * 96 + 1)[1:].view(6, 96), weight, None)):
        assert not float32_kernels_read(other_rows, other_weight, out)


def test_float32_rows_are_checked_against_the_weights_before_a_launch():
    import torch
    from fieldrun_b200.csrc import ops
    lists, tile = (torch.zeros(1, dtype=torch.int32),) * 4, 1
    for x, out in ((torch.zeros(2, 8), torch.zeros(2, 16)), (torch.zeros(2, 12), torch.zeros(2, 8)), (torch.zeros(3, 12), torch.zeros(2, 16))):
        with pytest.raises(ops.KernelError, match="with rows"):
            ops.rows_f32(torch.zeros(1, 16, 12), x, None, *lists, tile, out, paired=False)
        with pytest.raises(ops.KernelError, match="with rows"):
            ops.dense_rows_f32(torch.zeros(16, 12), x, out)


def test_only_a_parts_product_may_read_its_weight_early(monkeypatch):
    """A product of any other weight, which may be the result of the kernel before it, waits for that one."""
    import inspect

    import torch
    from fieldrun_b200.csrc import ops
    from fieldrun_b200.parts import linear as products
    calls = []
    monkeypatch.setattr(ops, "_call", lambda name, *args: calls.append(args))
    monkeypatch.setattr(ops, "_ptr", lambda t: 0)
    weight, x, out = torch.zeros(16, 12), torch.zeros(2, 12), torch.zeros(2, 16)
    ops.dense_rows_f32(weight, x, out)
    ops.dense_rows_f32(weight, x, out, weights_final=True)
    assert [c[-1] for c in calls] == [0, 1]
    parameters = inspect.signature(products.linear).parameters
    assert parameters["weight_final"].default is False and products.part_linear.keywords == {"weight_final": True}


@pytest.mark.parametrize("hidden,heads,dim,experts,width,vocab,expected", [
    (3072, 48, 128, 256, 1536, 200064, {"attention32", "products32"}),       # MiniMax-M2's layer
    (96, 8, 12, 8, 48, 384, {"attention32", "products32"}),                  # small: attention in tiles; experts on the tensor cores
    (100, 4, 10, 4, 36, 384, set()),                                         # sizes that neither kernel takes
    (96, 8, 12, 8, 36, 384, {"attention32"}),                                # dense products too small at any step's rows
    (1024, 4, 130, 4, 36, 2000, {"products32"}),                             # heads beyond both attention kernels, a large head matrix
])
def test_a_float32_model_asks_for_the_kernels_its_sizes_use(hidden, heads, dim, experts, width, vocab, expected):
    import torch
    from fieldrun_b200.api import build_model
    from fieldrun_b200.config.registry import architecture_for
    config = dict(architectures=["MiniMaxM2ForCausalLM"], model_type="minimax_m2", num_hidden_layers=1, hidden_size=hidden,
                  num_attention_heads=heads, num_key_value_heads=2, head_dim=dim, rotary_dim=2, rope_theta=1e6, use_qk_norm=False,
                  num_local_experts=experts, num_experts_per_tok=2, intermediate_size=width, vocab_size=vocab, rms_norm_eps=1e-5,
                  tie_word_embeddings=False)
    arch = architecture_for(config, "config")
    model = build_model(arch, arch.config_from_dict(config, "config"), torch.float32)
    assert set(model.kernel_groups()) == {"common", "streams", "experts"} | expected


@pytest.mark.parametrize("rows,features,inner,pays", [
    (9, 200064, 3072, False), (32, 200064, 3072, False), (48, 200064, 3072, True), (32, 32768, 4096, False), (48, 32768, 4096, True),
    (64, 8192, 3072, False), (96, 8192, 3072, True), (3704, 8192, 3072, True), (128, 3072, 6144, False), (256, 3072, 6144, True),
    (256, 2048, 2048, False), (512, 2048, 2048, True), (1024, 1024, 1024, False), (2048, 1024, 1024, True), (2048, 256, 3072, False)])
def test_float32_products_are_split_where_that_was_measured_to_be_faster(rows, features, inner, pays):
    import torch
    from fieldrun_b200.parts.linear import split_products_pay
    assert split_products_pay(rows, torch.empty(features, inner, device="meta")) == pays


def test_float32_attention_leaves_steps_beyond_its_grid_to_the_general_kernel():
    from fieldrun_b200.csrc import ops
    assert ops.attention_f32_tiles_take(128, 128, 32767) and not ops.attention_f32_tiles_take(128, 128, 32768)
    assert ops.attention_f32_token_takes(128, 128, 65535) and not ops.attention_f32_token_takes(128, 128, 65536)


@pytest.mark.parametrize("kind,heads,dim,vdim,lengths,chunks", [
    ("gated_linear_attention", 16, 128, 128, [63] * 16, False), ("gated_linear_attention", 16, 128, 128, [64], True),
    ("gated_linear_attention", 16, 128, 128, [65] * 16, False), ("gated_linear_attention", 16, 128, 128, [130] * 16, True),
    ("gated_linear_attention", 64, 64, 64, [128] + [5] * 63, False), ("gated_linear_attention", 64, 64, 64, [65] * 16, True),
    ("scalar_decay_state_space", 64, 128, 64, [128], False), ("scalar_decay_state_space", 64, 128, 64, [256], True),
    ("scalar_decay_state_space", 64, 128, 64, [130] * 16, False), ("scalar_decay_state_space", 64, 128, 64, [256] * 16, True),
    ("scalar_decay_state_space", 64, 128, 64, [256] + [2] * 31, False), ("scalar_decay_state_space", 64, 128, 64, [1024] + [16] * 31, True),
    ("scalar_decay_state_space", 16, 64, 64, [128] * 64, False), ("scalar_decay_state_space", 16, 64, 64, [1024] * 4, True),
    ("gated_delta_rule", 16, 128, 128, [64], False), ("gated_delta_rule", 16, 128, 128, [128], True),
    ("gated_delta_rule", 16, 64, 64, [130] * 16, False), ("gated_delta_rule", 64, 64, 64, [65] * 16, False),
    ("gated_delta_rule", 64, 128, 64, [256] + [2] * 31, False), ("gated_delta_rule", 16, 128, 128, [64] * 64, True)])
def test_recurrences_run_in_chunks_where_that_was_measured_to_be_faster(kind, heads, dim, vdim, lengths, chunks, monkeypatch):
    from types import SimpleNamespace
    import torch
    from fieldrun_b200.csrc import ops
    from fieldrun_b200.engine.context import StepContext
    from test_recurrent_chunks_gpu import mixer_spec
    from fieldrun_b200.parts import build_part
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    part = build_part("mixer", mixer_spec(kind, heads, dim, vdim), torch.bfloat16)
    ctx = SimpleNamespace(seq_q_lens=lengths, num_seqs=len(lengths), num_tokens=sum(lengths), max_q_len=max(lengths), is_decode=False, device=None)
    ctx.chunk_count = lambda size: StepContext.chunk_count(ctx, size)
    assert part.chunks_pay(ctx) == chunks
