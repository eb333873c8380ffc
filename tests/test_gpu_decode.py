"""Parity of the CUDA decode path (through the C ABI) against the CPU oracle."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from community_kv_b200 import native, ops
from community_kv_b200.batched import BatchedDecodeRuntime
from community_kv_b200.cache import StaticCacheLayer
from community_kv_b200.config import CommunityKVConfig, GraphAggregation
from community_kv_b200.runtime import DecodeRuntime, convert_prefill_tensors
from community_kv_b200.state import DecodeLayerWorkspace
from community_kv_b200.synthetic import make_layer, make_query
from tests.helpers import OracleLayer, assert_state_equal, assert_step_equal, fp16_ulp_distance

pytestmark = pytest.mark.gpu
SCALE = 128 ** -0.5


def _cover(converted):
    capacity = converted.mutable.community_capacity
    return [min(capacity, c + converted.decode_capacity) for c in converted.initial_community_counts]


def _run_sequence(layer, config, steps, *, seed, integer=False, splits=None, defer_update=False,
                  exact_scores=False, max_communities=0):

    device = torch.device("cuda", 0)
    runtime = DecodeRuntime(config, splits=splits, defer_update=defer_update, max_communities=max_communities)
    state = runtime.prepare_layer(0, **layer.to(device).prepare_kwargs())
    twin = OracleLayer(
        state.converted.csr,
        state.converted.mutable,
        state.converted.current_position,
        token_budget=state.workspace.selection.token_budget,
        num_sink=config.num_sink,
        cover=_cover(state.converted),
        max_communities=max_communities,
    )
    key = layer.key.to(device)[None]
    value = layer.value.to(device)[None]
    for step in range(steps):
        query = make_query(seed=seed + step, query_heads=layer.query_heads, integer_valued=integer)
        out = runtime.decode(
            layer_idx=0,
            query=query.to(device)[None, :, None, :],
            key=key,
            value=value,
            softmax_scale=SCALE,
        )
        assert out.shape == (1, 1, layer.query_heads, 128)
        runtime.synchronize_updates()
        where = f"step {step}"
        if exact_scores:  # the device scores themselves, bit for bit, where the scan covers them
            cover = torch.as_tensor(twin.cover)[:, None]
            covered = torch.arange(twin.scores.shape[1])[None, :] < cover
            want_scores = twin.exact_scores(query)
            got_scores = state.workspace.selection.scores.cpu()
            assert torch.equal(got_scores.view(torch.int16)[covered], want_scores.view(torch.int16)[covered]), where
        want = twin.step(query=query, key=layer.key, value=layer.value, softmax_scale=SCALE, lam=config.lam,
                         device_scores=state.workspace.selection.scores, assignment=config.online_assignment)
        assert_step_equal(
            selection=state.workspace.selection,
            attention=state.workspace.attention,
            update=state.workspace.update,
            result=want,
            where=where,
        )
        assert_state_equal(state.converted.mutable, twin.state, where)
        assert torch.equal(state.converted.current_position.cpu(), twin.current), where
    runtime.assert_no_overflow()
    return state, twin


@pytest.mark.parametrize(
    "aggregation", [GraphAggregation.QUERY_GROUP, GraphAggregation.PER_QUERY_HEAD, GraphAggregation.LAYER_WISE]
)
def test_single_layer_config0_parity(aggregation):
    """Single-layer configuration: ctx 8192, 32/8 heads, 64 planted clusters, budget 1024."""

    layer = make_layer(seed=0, seq_len=8192, communities=64, max_decode_tokens=8, aggregation=aggregation)
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation=aggregation)
    _run_sequence(layer, config, steps=4, seed=100)


def test_unfused_kernels_give_the_same_result(monkeypatch):
    """The four stand-alone kernels and the single cluster launch are the same path."""

    monkeypatch.setenv("CKV_UNFUSED", "1")
    layer = make_layer(seed=0, seq_len=8192, communities=64, max_decode_tokens=8, aggregation="query_group")
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=4, seed=100)


@pytest.mark.parametrize("kv_heads,splits,expected,kernels", [(2, None, 32, 4), (3, 11, 11, 1), (1, 9, 9, 1)])
def test_more_than_eight_splits(kv_heads, splits, expected, kernels):
    """A budget above 4096 on few heads: the default number of splits, and a cluster of more than eight CTAs."""

    layer = make_layer(seed=51, seq_len=12007, communities=301, kv_heads=kv_heads, max_decode_tokens=6,
                       zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=8192, num_sink=10, lam=0.5, aggregation="query_group")
    state, twin = _run_sequence(layer, config, steps=4, seed=5100, splits=splits)
    assert state.workspace.attention.splits == expected
    assert native.library().ckv_decode_layer_kernels(ctypes.byref(state.args)) == kernels


@pytest.mark.parametrize(
    "batch,kv_heads,group,splits,communities,kernels",
    [
        (1, 2, 4, None, 20000, 1),  # the default of 32 splits over sixteen CTAs
        (1, 1, 1, 17, 20000, 1),    # nine CTAs, two splits but for one
        (1, 2, 8, 31, 20000, 1),    # sixteen CTAs, two splits but for one
        (1, 2, 4, 32, 300, 4),      # few communities: four kernels
        (1, 20, 2, 16, 300, 1),     # 320 of 444 CTA slots
        (1, 21, 2, 16, 300, 4),     # 336: no room for the next launch
        (1, 2, 16, 16, 300, 4),     # two blocks of query heads
        (3, 4, 4, 13, 300, 1),      # a batch
        (3, 9, 4, None, 300, 4),    # 27 units: sixteen splits, all the slots
    ],
)
def test_splits_alone_decide_the_bits(monkeypatch, batch, kv_heads, group, splits, communities, kernels):
    """However many CTAs share the splits, output and state are those of the four stand-alone kernels."""

    device = torch.device("cuda", 0)
    config = CommunityKVConfig(token_budget=8192, num_sink=10, lam=0.5, aggregation="query_group")
    length = 40000 if communities > 1000 else 9001
    layers = [make_layer(seed=70 + b, seq_len=length, communities=communities, kv_heads=kv_heads, group_size=group,
                         max_decode_tokens=6) for b in range(batch)]
    key = torch.stack([layer.key for layer in layers]).to(device)
    value = torch.stack([layer.value for layer in layers]).to(device)

    def run(unfused):
        monkeypatch.setenv("CKV_UNFUSED", unfused)
        runtime = BatchedDecodeRuntime(config, splits=splits)
        state = runtime.prepare_layer(0, [convert_prefill_tensors(**layer.to(device).prepare_kwargs()) for layer in layers])
        outputs = []
        for step in range(4):
            query = torch.stack([make_query(seed=80 + 10 * step + b, query_heads=kv_heads * group) for b in range(batch)])
            outputs.append(runtime.decode(layer_idx=0, query=query.to(device), key=key, value=value,
                                          softmax_scale=SCALE).clone())
        ws = state.workspace.attention
        launched = native.library().ckv_decode_layer_kernels(ctypes.byref(state.args))
        return launched, [*outputs, ws.lse, ws.topk_scores, ws.topk_positions, *state.mutable.tensors()]

    four, want = run("1")
    launched, got = run("0")
    assert (four, launched) == (4, kernels)
    for first, second in zip(got, want):
        assert torch.equal(first.contiguous().view(torch.uint8), second.contiguous().view(torch.uint8))


@pytest.mark.parametrize("unfused", [False, True])
def test_fixed_order_scores_are_bit_exact(monkeypatch, unfused):
    """``CKV_TENSOR_SCORES=0``: the CUDA-core scoring path sums in the fixed order the CPU restatement
    reproduces, so the fp16 scores themselves (and with them everything else) match bit for bit."""

    monkeypatch.setenv("CKV_TENSOR_SCORES", "0")
    assert not ops.tensor_scores_enabled()
    if unfused:
        monkeypatch.setenv("CKV_UNFUSED", "1")
    layer = make_layer(seed=13, seq_len=16384, communities=700, max_decode_tokens=8, zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=6, seed=1300)
    layer = make_layer(seed=0, seq_len=8192, communities=64, max_decode_tokens=8, aggregation="per_query_head")
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="per_query_head")
    _run_sequence(layer, config, steps=3, seed=100)


@pytest.mark.parametrize("unfused", [False, True])
def test_tensor_core_scores(monkeypatch, unfused):
    """Scoring on the tensor cores (single cluster launch and the stand-alone kernels): scores within one
    fp16 unit in the last place of the fixed-order ones, the rest of the step exact given those scores."""

    monkeypatch.setenv("CKV_TENSOR_SCORES", "1")
    assert ops.tensor_scores_enabled()
    if unfused:
        monkeypatch.setenv("CKV_UNFUSED", "1")
    layer = make_layer(seed=11, seq_len=16384, communities=700, max_decode_tokens=8, zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=6, seed=1100)
    layer = make_layer(seed=12, kv_heads=2, group_size=8, seq_len=4096, communities=100, max_decode_tokens=4)
    config = CommunityKVConfig(token_budget=512, num_sink=4, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=3, seed=1200, splits=3)


@pytest.mark.parametrize("aggregation", [GraphAggregation.QUERY_GROUP, GraphAggregation.LAYER_WISE])
def test_deferred_update_gives_the_same_result(aggregation):
    """Attention on the caller's stream, online assignment on a second stream: same step, same state."""

    layer = make_layer(seed=21, seq_len=8192, communities=200, max_decode_tokens=10, aggregation=aggregation,
                       zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation=aggregation)
    _run_sequence(layer, config, steps=8, seed=2100, defer_update=True)


@pytest.mark.parametrize(
    "aggregation,defer", [(GraphAggregation.QUERY_GROUP, False), (GraphAggregation.QUERY_GROUP, True),
                          (GraphAggregation.PER_QUERY_HEAD, False), (GraphAggregation.LAYER_WISE, False)]
)
def test_nearest_centroid_assignment_variant(aggregation, defer):
    """Not in the reference: every decoded token joins the community whose centroid is nearest to its key
    (largest inner product, first maximum).  State and outputs against the CPU restatement, bit for bit;
    the variant never opens a community, and its choices differ from the modularity rule's."""

    layer = make_layer(seed=23, seq_len=8192, communities=96, max_decode_tokens=12, aggregation=aggregation,
                       zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation=aggregation,
                               online_assignment="nearest_centroid")
    before = layer.to(torch.device("cuda", 0)).prepare_kwargs()["num_communities"].clone()
    state, twin = _run_sequence(layer, config, steps=10, seed=2300, defer_update=defer)
    counts = state.converted.mutable.community_counts
    assert int(counts.max()) == int(before.max()) and int(counts.min()) == int(before.min())
    with pytest.raises(ValueError):
        CommunityKVConfig(online_assignment="nearest")


@pytest.mark.parametrize("communities", [255, 257, 1301])
def test_nearest_centroid_over_many_communities(communities):
    """Around one row per lane group of the cluster (256 rows), and more rows than are in flight at once."""

    layer = make_layer(seed=communities, seq_len=8192, communities=communities, kv_heads=2, max_decode_tokens=6)
    config = CommunityKVConfig(token_budget=512, num_sink=10, lam=0.5, aggregation="query_group",
                               online_assignment="nearest_centroid")
    _run_sequence(layer, config, steps=4, seed=2400)


@pytest.mark.parametrize("aggregation", [GraphAggregation.QUERY_GROUP, GraphAggregation.LAYER_WISE])
def test_fp32_centroid_table(aggregation):
    """Not the reference's layout: the centroid table in fp32.  The scores (fixed-order sum of products
    rounded one by one), everything downstream and the unquantised running mean against the CPU
    restatement, bit for bit; the call runs the four stand-alone kernels."""

    layer = make_layer(seed=29, seq_len=8192, communities=80, max_decode_tokens=10, aggregation=aggregation)
    table = layer.assembled.centroids.float()
    generator = torch.Generator().manual_seed(291)
    layer.assembled.centroids = table * 1.0009765625 + 1e-3 * torch.randn(table.shape, generator=generator)
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation=aggregation,
                               centroid_dtype="fp32")
    with pytest.raises(TypeError, match="FP8"):  # the reference's layout unless asked otherwise
        convert_prefill_tensors(**layer.prepare_kwargs())
    state, twin = _run_sequence(layer, config, steps=8, seed=2900, exact_scores=True)
    assert state.converted.mutable.centroids.dtype == torch.float32
    assert native.library().ckv_decode_layer_kernels(ctypes.byref(state.args)) >= 4


def test_single_layer_configuration_as_worded():
    """The single-layer configuration to the letter: ctx 8192, 32 / 8 heads, 64 planted clusters, the
    centroids the per-community mean keys in fp32, the eight best communities per KV head, budget 1024.
    Scores, selection, attention output, neighbour candidates and the online update against the CPU
    restatement (scores and state bit for bit)."""

    layer = make_layer(seed=0, seq_len=8192, communities=64, max_decode_tokens=8, aggregation="query_group")
    assembled = layer.assembled
    heads, capacity, _ = assembled.centroids.shape
    labels = assembled.token_communities[:, : layer.prefill_seq_len].long()  # [graphs, S]
    means = torch.zeros((heads, capacity, 128), dtype=torch.float32)
    for head in range(heads):
        graph, kv = int(assembled.retrieval_to_graph[head]), int(assembled.retrieval_to_kv[head])
        keep = torch.arange(layer.prefill_seq_len) >= 10  # the ten sink positions are not members
        means[head].index_add_(0, labels[graph][keep], layer.key[kv, : layer.prefill_seq_len][keep].float())
        sizes = assembled.community_sizes[head].clamp(min=1).float()
        means[head] /= sizes[:, None]
    assembled.centroids = means
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="query_group",
                               centroid_dtype="fp32")
    state, _ = _run_sequence(layer, config, steps=4, seed=100, exact_scores=True, max_communities=8)
    assert int(state.workspace.selection.descriptor_counts.max()) <= 8


def test_many_small_communities_and_delta_chains():
    """Mean community size ~16 (the tuned regime): many descriptors, decode deltas get re-selected."""

    layer = make_layer(seed=1, kv_heads=2, seq_len=4096, communities=256, max_decode_tokens=24)
    config = CommunityKVConfig(token_budget=512, num_sink=4, lam=0.5, aggregation="query_group")
    state, twin = _run_sequence(layer, config, steps=24, seed=200, splits=4)
    assert int(state.converted.mutable.deltas.community_sizes.sum()) == 24 * 2


def test_integer_fixture_is_exact_end_to_end():
    """Small-integer operands: every fp32 sum is exact, so even the bf16 output must match closely."""

    layer = make_layer(seed=2, kv_heads=2, seq_len=2048, communities=32, max_decode_tokens=6, integer_valued=True)
    config = CommunityKVConfig(token_budget=256, num_sink=2, lam=0.25, aggregation="query_group")
    _run_sequence(layer, config, steps=6, seed=300, integer=True, splits=2)


@pytest.mark.parametrize("group_size,kv_heads", [(1, 4), (2, 4), (5, 2), (8, 2), (12, 1), (16, 1)])
def test_group_sizes(group_size, kv_heads):
    layer = make_layer(seed=3 + group_size, kv_heads=kv_heads, group_size=group_size, seq_len=2048,
                       communities=48, max_decode_tokens=4)
    config = CommunityKVConfig(token_budget=256, num_sink=3, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=2, seed=400 + group_size, splits=1)


def test_zipf_communities_full_context_unit():
    """One (sequence, layer) of the batched long-context configuration: ctx 131072, 4096 Zipf communities, budget 2048."""

    layer = make_layer(seed=5, seq_len=131072, communities=4096, max_decode_tokens=4, zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=2048, num_sink=10, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=2, seed=500)


def test_config3_layer_with_online_assignment():
    """One layer of the whole-model configuration: ctx 32768, 512 Zipf(1.1) communities per KV head,
    budget 2048, every decoded token assigned online (eight steps)."""

    layer = make_layer(seed=7, seq_len=32768, communities=512, max_decode_tokens=12, zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=2048, num_sink=10, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=8, seed=700)


def test_batched_sequences_match_per_sequence_oracle():
    device = torch.device("cuda", 0)
    config = CommunityKVConfig(token_budget=512, num_sink=10, lam=0.5, aggregation="query_group")
    layers = [
        make_layer(seed=10 + b, kv_heads=4, seq_len=4096, communities=96 + 16 * b, max_decode_tokens=6,
                   zipf_exponent=1.1 if b % 2 else None)
        for b in range(3)
    ]
    runtime = BatchedDecodeRuntime(config, splits=2)
    converted = [convert_prefill_tensors(**layer.to(device).prepare_kwargs()) for layer in layers]
    state = runtime.prepare_layer(0, converted)
    twins = []
    for b in range(3):
        csr, mutable, current = state.sequence_view(b)
        twins.append(
            OracleLayer(csr, mutable, current, token_budget=state.token_budget, num_sink=config.num_sink,
                        cover=state.workspace.selection.score_cover[b].cpu().tolist())
        )
    key = torch.stack([layer.key for layer in layers]).to(device)
    value = torch.stack([layer.value for layer in layers]).to(device)
    for step in range(5):
        queries = torch.stack([make_query(seed=600 + 10 * step + b, query_heads=16) for b in range(3)])
        out = runtime.decode(layer_idx=0, query=queries.to(device), key=key, value=value, softmax_scale=SCALE)
        assert out.shape == (3, 16, 128)
        for b in range(3):
            want = twins[b].step(query=queries[b], key=layers[b].key, value=layers[b].value,
                                 softmax_scale=SCALE, lam=config.lam,
                                 device_scores=state.workspace.selection.scores[b])
            ws = state.workspace
            view = lambda obj, names: type("V", (), {n: getattr(obj, n)[b] for n in names})
            assert_step_equal(
                selection=view(ws.selection, ["scores", "descriptor_counts", "communities", "cumulative_ends",
                                               "tile_descriptors", "positions"]),
                attention=view(ws.attention, ["output", "lse", "topk_positions", "topk_scores"]),
                update=view(ws.update, ["assigned_communities", "overflow"]),
                result=want,
                where=f"step {step} seq {b}",
            )
            _, mutable, current = state.sequence_view(b)
            assert_state_equal(mutable, twins[b].state, f"step {step} seq {b}")
            assert torch.equal(current.cpu(), twins[b].current)
    runtime.assert_no_overflow()


def test_standalone_entry_points_and_skip_update():
    """score -> select -> attention as three separate C-ABI calls, without the online update."""

    device = torch.device("cuda", 0)
    layer = make_layer(seed=20, kv_heads=2, seq_len=2048, communities=40, max_decode_tokens=4)
    config = CommunityKVConfig(token_budget=256, num_sink=5, lam=0.5, aggregation="query_group")
    converted = convert_prefill_tensors(**layer.to(device).prepare_kwargs())
    ws = DecodeLayerWorkspace.allocate(
        retrieval_head_count=2, graph_count=2, group_size=4, community_capacity=converted.mutable.community_capacity,
        token_budget=256, num_sink=5, dtype=torch.bfloat16, device=device, splits=2,
    )
    sinks = torch.arange(5, dtype=torch.int32, device=device)
    twin = OracleLayer(converted.csr, converted.mutable, converted.current_position, token_budget=256,
                       num_sink=5, cover=None)
    query = make_query(seed=21, query_heads=8)
    mutable = converted.mutable
    ops.score_centroids(query=query.to(device), centroids=mutable.centroids,
                        community_sizes=mutable.community_sizes, community_counts=mutable.community_counts,
                        workspace=ws.selection)
    segments = ops.select_weighted_descriptors_auto(
        community_sizes=mutable.community_sizes, community_counts=mutable.community_counts,
        workspace=ws.selection, csr=converted.csr, state=mutable, sink_positions=sinks,
        current_position=converted.current_position)
    ws.selection.positions.fill_(-7)  # the attention entry point must resolve positions itself
    ops.segmented_attention(
        query=query.to(device), key=layer.key.to(device), value=layer.value.to(device), csr=converted.csr,
        deltas=mutable.deltas, segments=segments, sink_positions=sinks,
        current_position=converted.current_position, softmax_scale=SCALE, workspace=ws.attention,
        update_state=mutable, update_workspace=None, update_lam=0.5, positions=ws.selection.positions)
    want = twin.step(query=query, key=layer.key, value=layer.value, softmax_scale=SCALE, lam=0.5, update=False,
                     device_scores=ws.selection.scores)
    assert_step_equal(selection=ws.selection, attention=ws.attention, update=ws.update, result=want,
                      check_update=False)
    assert_state_equal(mutable, twin.state, "skip-update leaves the state untouched")
    assert int(converted.current_position[0]) == 2048


def test_topk_communities_mode_and_underfill():
    """Extension (top-k communities under a token budget): at most k communities; unfilled slots are masked."""

    device = torch.device("cuda", 0)
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="query_group")
    layer = make_layer(seed=30, kv_heads=4, seq_len=8192, communities=64, max_decode_tokens=4)
    converted = [convert_prefill_tensors(**layer.to(device).prepare_kwargs())]
    runtime = BatchedDecodeRuntime(config)
    state = runtime.prepare_layer(0, converted, max_communities=5)
    csr, mutable, current = state.sequence_view(0)
    twin = OracleLayer(csr, mutable, current, token_budget=1024, num_sink=10,
                       cover=state.workspace.selection.score_cover[0].cpu().tolist(), max_communities=5)
    key = layer.key.to(device)[None]
    value = layer.value.to(device)[None]
    for step in range(3):
        query = make_query(seed=700 + step, query_heads=16)
        runtime.decode(layer_idx=0, query=query.to(device)[None], key=key, value=value, softmax_scale=SCALE)
        want = twin.step(query=query, key=layer.key, value=layer.value, softmax_scale=SCALE, lam=0.5,
                         device_scores=state.workspace.selection.scores[0])
        ws = state.workspace
        view = lambda obj, names: type("V", (), {n: getattr(obj, n)[0] for n in names})
        assert int(ws.selection.descriptor_counts.max()) <= 5
        assert int((ws.selection.positions == -1).sum()) > 0  # 5 of 64 clusters cannot fill 1013 slots
        assert_step_equal(
            selection=view(ws.selection, ["scores", "descriptor_counts", "communities", "cumulative_ends",
                                           "tile_descriptors", "positions"]),
            attention=view(ws.attention, ["output", "lse", "topk_positions", "topk_scores"]),
            update=view(ws.update, ["assigned_communities", "overflow"]),
            result=want, where=f"step {step}")
        assert_state_equal(state.sequence_view(0)[1], twin.state, f"step {step}")


def test_overflow_flags_stop_the_cursor():
    """Exhaust the decode-delta pools on purpose: flags are raised, the cursor stops, nothing faults."""

    layer = make_layer(seed=40, kv_heads=1, seq_len=1024, communities=16, max_decode_tokens=2)
    config = CommunityKVConfig(token_budget=128, num_sink=2, lam=0.5, aggregation="query_group")
    device = torch.device("cuda", 0)
    runtime = DecodeRuntime(config, splits=1)
    state = runtime.prepare_layer(0, **layer.to(device).prepare_kwargs())
    twin = OracleLayer(state.converted.csr, state.converted.mutable, state.converted.current_position,
                       token_budget=128, num_sink=2, cover=_cover(state.converted))
    key, value = layer.key.to(device)[None], layer.value.to(device)[None]
    for step in range(4):
        query = make_query(seed=800 + step, query_heads=4)
        runtime.decode(layer_idx=0, query=query.to(device)[None, :, None, :], key=key, value=value,
                       softmax_scale=SCALE)
        want = twin.step(query=query, key=layer.key, value=layer.value, softmax_scale=SCALE, lam=0.5,
                         device_scores=state.workspace.selection.scores)
        assert torch.equal(state.workspace.update.overflow.cpu(), want.overflow), step
        assert_state_equal(state.converted.mutable, twin.state, f"step {step}")
        assert torch.equal(state.converted.current_position.cpu(), twin.current)
    with pytest.raises(RuntimeError, match="overflow"):
        runtime.assert_no_overflow()


def test_full_cache_masks_the_cursor_row():
    """Once the cache is full the cursor equals its capacity: the update reports it (overflow bit 8) and
    the attention treats that slot as masked instead of reading one row past the head's slice."""

    device = torch.device("cuda", 0)
    layer = make_layer(seed=41, kv_heads=2, seq_len=1024, communities=16, max_decode_tokens=3).to(device)
    config = CommunityKVConfig(token_budget=128, num_sink=2, lam=0.5, aggregation="query_group")
    runtime = DecodeRuntime(config, splits=2)
    state = runtime.prepare_layer(0, **layer.prepare_kwargs())
    rows = 1024 + 2  # a cache that ends two rows after the prompt
    key = layer.key[:, :rows].contiguous()[None]
    value = layer.value[:, :rows].contiguous()[None]
    # poison what lies right behind the last head's slice: it must never be read
    for step in range(4):
        query = make_query(seed=810 + step, query_heads=8).to(device)
        out = runtime.decode(layer_idx=0, query=query[None, :, None, :], key=key, value=value, softmax_scale=SCALE)
        assert torch.isfinite(out.float()).all(), step
        flags = state.workspace.update.overflow.cpu()
        cursor = state.converted.current_position.cpu()
        if step < 2:
            assert int(flags.max()) == 0 and int(cursor.min()) == 1024 + step + 1
        else:
            assert bool(((flags & 8) == 8).all()) and int(cursor.max()) == rows
            # every slot of the budget is a cached row or masked, never the row at the capacity
            assert int(state.workspace.selection.positions.max()) <= rows
    with pytest.raises(RuntimeError, match="overflow"):
        runtime.assert_no_overflow()


def test_shape_errors_are_reported_before_launch():
    device = torch.device("cuda", 0)
    layer = make_layer(seed=50, kv_heads=1, seq_len=1024, communities=16, max_decode_tokens=2)
    config = CommunityKVConfig(token_budget=128, num_sink=2)
    runtime = DecodeRuntime(config)
    runtime.prepare_layer(0, **layer.to(device).prepare_kwargs())
    with pytest.raises(ValueError, match="query shape"):
        runtime.decode(layer_idx=0, query=torch.zeros((1, 4, 2, 128), device=device, dtype=torch.bfloat16),
                       key=layer.key.to(device)[None], value=layer.value.to(device)[None], softmax_scale=SCALE)
    with pytest.raises(RuntimeError, match="not prepared"):
        runtime.decode(layer_idx=3, query=torch.zeros((1, 4, 1, 128), device=device, dtype=torch.bfloat16),
                       key=layer.key.to(device)[None], value=layer.value.to(device)[None], softmax_scale=SCALE)


def test_append_kv_rows():
    """ckv_append_kv: one row per (sequence, head) into both caches, scalar and per-unit index."""

    device = torch.device("cuda", 0)
    torch.manual_seed(5)
    key = torch.randn((3, 2, 40, 128), device=device).to(torch.bfloat16)
    value = torch.randn_like(key)
    new_key = torch.randn((3, 2, 128), device=device).to(torch.bfloat16)
    new_value = torch.randn_like(new_key)
    want_key, want_value = key.clone(), value.clone()
    want_key[:, :, 17] = new_key
    want_value[:, :, 17] = new_value
    ops.append_kv(key, value, new_key, new_value, 17)
    assert torch.equal(key, want_key) and torch.equal(value, want_value)
    rows = torch.tensor([0, 39, -1, 5, 5, 12], dtype=torch.int32, device=device)
    for unit, row in enumerate(rows.tolist()):
        if row >= 0:
            want_key.view(6, 40, 128)[unit, row] = new_key.view(6, 128)[unit]
            want_value.view(6, 40, 128)[unit, row] = new_value.view(6, 128)[unit]
    ops.append_kv(key, value, new_key, new_value, rows)
    assert torch.equal(key, want_key) and torch.equal(value, want_value)
    with pytest.raises(ValueError):
        ops.append_kv(key, value, new_key, new_value, 40)


@pytest.mark.parametrize("units", [1, 4, 5, 33, 70])
def test_append_kv_moves_the_cursor(units):
    """One launch writes the rows and moves the cursor on: four warps, a warp per unit, several units per warp."""

    device = torch.device("cuda", 0)
    torch.manual_seed(units)
    key = torch.randn((units, 9, 128), device=device).to(torch.bfloat16)
    value = torch.randn_like(key)
    want_key, want_value = key.clone(), value.clone()
    cursor = torch.tensor([5], dtype=torch.int32, device=device)
    for row in (5, 6, 7):
        new_key = torch.randn((units, 128), device=device).to(torch.bfloat16)
        new_value = torch.randn_like(new_key)
        want_key[:, row], want_value[:, row] = new_key, new_value
        ops.append_kv(key, value, new_key, new_value, cursor, advance=True)
    assert int(cursor) == 8
    assert torch.equal(key, want_key) and torch.equal(value, want_value)
    with pytest.raises(ValueError):
        ops.append_kv(key, value, new_key, new_value, 3, advance=True)
    with pytest.raises(ValueError):
        ops.append_kv(key[:4], value[:4], new_key[:4], new_value[:4], cursor.repeat(4), advance=True)


@pytest.mark.parametrize("units", [128, 129, 700])
def test_append_kv_moves_the_cursor_behind_many_rows(units):
    """On both sides of the line between one CTA for rows and cursor, and two launches; also replayed from a graph."""

    device = torch.device("cuda", 0)
    torch.manual_seed(units)
    key = torch.randn((units, 9, 128), device=device).to(torch.bfloat16)
    value = torch.randn_like(key)
    new = [torch.randn((units, 128), device=device).to(torch.bfloat16) for _ in range(2)]
    want = [key.clone(), value.clone()]
    cursor = torch.tensor([5], dtype=torch.int32, device=device)
    ops.append_kv(key, value, *new, cursor, advance=True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.append_kv(key, value, *new, cursor, advance=True)
    for row in (5, 6, 7):
        if row > 5:
            for tensor in new:
                tensor.copy_(torch.randn_like(tensor))
            graph.replay()
        want[0][:, row], want[1][:, row] = new
    assert int(cursor) == 8
    assert torch.equal(key, want[0]) and torch.equal(value, want[1])


def test_append_kv_of_many_rows_uses_the_chip():
    """A cursor that moves does not leave 4096 rows to one CTA (25 times as long as over the chip)."""

    device = torch.device("cuda", 0)
    key = torch.zeros((4096, 130, 128), dtype=torch.bfloat16, device=device)
    value = torch.zeros_like(key)
    new = [torch.ones((4096, 128), dtype=torch.bfloat16, device=device) for _ in range(2)]
    cursor = torch.zeros(1, dtype=torch.int32, device=device)

    def microseconds(advance):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            cursor.zero_()
            for _ in range(100):
                ops.append_kv(key, value, *new, cursor, advance=advance)
        spans = []
        for _ in range(5):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            begin.record()
            graph.replay()
            end.record()
            end.synchronize()
            spans.append(begin.elapsed_time(end) * 10)
        return min(spans)

    ops.append_kv(key, value, *new, cursor)
    assert microseconds(True) < 4 * microseconds(False) + 5


def test_the_cache_appends_under_capture():
    """The device phase of the plug-in's cache needs no host: a captured append writes another row at every replay."""

    device = torch.device("cuda", 0)
    layer = StaticCacheLayer(max_cache_len=12)
    prompt = torch.randn((1, 6, 4, 128), device=device).to(torch.bfloat16)
    row_key, row_value = (torch.randn((1, 6, 1, 128), device=device).to(torch.bfloat16) for _ in range(2))
    with torch.inference_mode():
        layer.update(prompt, prompt)
        layer.enable_device_updates()
        layer.update(row_key, row_value)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            layer.update(row_key, row_value)
        want_key, want_value = layer.keys.clone(), layer.values.clone()
        for row in (5, 6, 7):
            row_key.copy_(torch.randn_like(row_key))
            row_value.copy_(torch.randn_like(row_value))
            graph.replay()
            want_key[:, :, row], want_value[:, :, row] = row_key[:, :, 0], row_value[:, :, 0]
        layer.sync_valid_length()
    assert layer.valid_length == 8
    assert torch.equal(layer.keys, want_key) and torch.equal(layer.values, want_value)


@pytest.mark.parametrize("units", [1, 3, 40])
def test_append_kv_past_the_last_row(units):
    """A row that only the device knows and that lies outside the cache writes nothing: not into the next head's rows,
    not behind the last head's.  The caches lie inside larger buffers that must stay as they were."""

    device = torch.device("cuda", 0)
    rows = 9
    torch.manual_seed(units)
    buffers = [torch.randn((units + 2, rows, 128), device=device).to(torch.bfloat16) for _ in range(2)]
    key, value = (buffer[1:-1] for buffer in buffers)
    want = [buffer.clone() for buffer in buffers]
    new = [torch.randn((units, 128), device=device).to(torch.bfloat16) for _ in range(2)]
    cursor = torch.tensor([rows - 1], dtype=torch.int32, device=device)
    for _ in range(3):
        ops.append_kv(key, value, *new, cursor, advance=True)
    for buffer, row in zip(want, new):
        buffer[1:-1, rows - 1] = row
    assert int(cursor) == rows + 2
    assert all(torch.equal(buffer, expected) for buffer, expected in zip(buffers, want))
    for outside in (rows, rows + 1, -1):
        ops.append_kv(key, value, *new, torch.full((1,), outside, dtype=torch.int32, device=device))
        ops.append_kv(key, value, *new, torch.full((units,), outside, dtype=torch.int32, device=device))
    assert all(torch.equal(buffer, expected) for buffer, expected in zip(buffers, want))


@pytest.mark.parametrize("kv_heads,group,fp32,deferred", [(2, 4, False, False), (5, 2, False, True), (9, 1, False, False),
                                                          (6, 2, True, False)])
def test_shared_graph_in_two_launches(monkeypatch, kv_heads, group, fp32, deferred):
    """One graph for all heads: the cluster launch and the update behind it (or beside the next step) leave the
    bits of the four stand-alone kernels, the followers' tables included (four of them at a time, and remainders)."""

    device = torch.device("cuda", 0)
    config = CommunityKVConfig(token_budget=512, num_sink=10, lam=0.5, aggregation="layer_wise",
                               centroid_dtype="fp32" if fp32 else "e4m3")
    layer = make_layer(seed=90 + kv_heads, seq_len=3001, communities=60, kv_heads=kv_heads, group_size=group,
                       max_decode_tokens=8, aggregation="layer_wise")
    if fp32:
        layer.assembled.centroids = layer.assembled.centroids.float()
    layer = layer.to(device)
    key, value = layer.key[None], layer.value[None]

    def run(unfused):
        monkeypatch.setenv("CKV_UNFUSED", unfused)
        runtime = DecodeRuntime(config, defer_update=deferred)
        state = runtime.prepare_layer(0, **{k: v.clone() if isinstance(v, torch.Tensor) else v
                                            for k, v in layer.prepare_kwargs().items()})
        outputs = []
        for step in range(6):
            query = make_query(seed=900 + step, query_heads=kv_heads * group).to(device)
            outputs.append(runtime.decode(layer_idx=0, query=query.view(1, kv_heads * group, 1, 128), key=key,
                                          value=value, softmax_scale=SCALE).clone())
        runtime.assert_no_overflow()
        launched = native.library().ckv_decode_layer_kernels(ctypes.byref(state.args))
        ws = state.workspace.attention
        return launched, [*outputs, ws.lse, ws.topk_scores, ws.topk_positions, *state.converted.mutable.tensors()]

    four, want = run("1")
    launched, got = run("0")
    assert (four, launched) == (4, 4 if fp32 else 2)
    for first, second in zip(got, want):
        assert torch.equal(first.contiguous().view(torch.uint8), second.contiguous().view(torch.uint8))


@pytest.mark.parametrize("kv_heads,fp32", [(20, False), (21, True), (45, False), (70, False)])
def test_followers_of_a_shared_graph_match_the_oracle(kv_heads, fp32):
    """Heads that share one graph, four to a warp: full warps, a remainder, the most warps and more heads than those
    take at once.  The followers' centroids, sizes and counts are the oracle's."""

    layer = make_layer(seed=30 + kv_heads, kv_heads=kv_heads, group_size=1, seq_len=1031, communities=24,
                       max_decode_tokens=5, aggregation="layer_wise")
    if fp32:
        layer.assembled.centroids = layer.assembled.centroids.float()
    config = CommunityKVConfig(token_budget=256, num_sink=3, lam=0.5, aggregation="layer_wise",
                               centroid_dtype="fp32" if fp32 else "e4m3")
    _run_sequence(layer, config, steps=4, seed=3000 + kv_heads)


@pytest.mark.parametrize("kv_heads,splits,kernels", [(3, 11, 2), (1, 9, 1), (2, None, 4)])
def test_shared_graph_with_more_than_eight_splits(kv_heads, splits, kernels):
    """One graph for all heads in a cluster of more than eight CTAs, and in the four kernels, against the oracle."""

    layer = make_layer(seed=53, seq_len=12007, communities=301, kv_heads=kv_heads, max_decode_tokens=6,
                       aggregation="layer_wise", zipf_exponent=1.1)
    config = CommunityKVConfig(token_budget=8192, num_sink=10, lam=0.5, aggregation="layer_wise")
    state, _ = _run_sequence(layer, config, steps=4, seed=5300, splits=splits)
    assert native.library().ckv_decode_layer_kernels(ctypes.byref(state.args)) == kernels


@pytest.mark.parametrize("kv_heads,kernels", [(12, 2), (13, 4)])
def test_shared_graph_on_both_sides_of_the_line(kv_heads, kernels):
    """96 CTAs of the cluster launch are the most that take two launches."""

    layer = make_layer(seed=57, kv_heads=kv_heads, group_size=1, seq_len=2053, communities=40, max_decode_tokens=5,
                       aggregation="layer_wise")
    config = CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="layer_wise")
    state, _ = _run_sequence(layer, config, steps=3, seed=5700, splits=8)
    assert native.library().ckv_decode_layer_kernels(ctypes.byref(state.args)) == kernels


@pytest.mark.parametrize("batch,kv_heads,deferred", [(3, 5, False), (3, 5, True), (2, 23, False)])
def test_shared_graphs_in_a_batch(batch, kv_heads, deferred):
    """Every sequence has a graph of its own that all its heads share: leaders and followers of each are the oracle's."""

    device = torch.device("cuda", 0)
    config = CommunityKVConfig(token_budget=256, num_sink=3, lam=0.5, aggregation="layer_wise")
    layers = [make_layer(seed=110 + b, kv_heads=kv_heads, group_size=2, seq_len=1500, communities=30 + 7 * b,
                         max_decode_tokens=6, aggregation="layer_wise") for b in range(batch)]
    runtime = BatchedDecodeRuntime(config, splits=2, defer_update=deferred)
    state = runtime.prepare_layer(0, [convert_prefill_tensors(**layer.to(device).prepare_kwargs()) for layer in layers])
    twins = []
    for b in range(batch):
        twins.append(OracleLayer(*state.sequence_view(b), token_budget=256, num_sink=3,
                                 cover=state.workspace.selection.score_cover[b].cpu().tolist()))
    key = torch.stack([layer.key for layer in layers]).to(device)
    value = torch.stack([layer.value for layer in layers]).to(device)
    for step in range(4):
        queries = torch.stack([make_query(seed=1200 + 10 * step + b, query_heads=2 * kv_heads) for b in range(batch)])
        runtime.decode(layer_idx=0, query=queries.to(device), key=key, value=value, softmax_scale=SCALE)
        torch.cuda.synchronize()
        for b in range(batch):
            twins[b].step(query=queries[b], key=layers[b].key, value=layers[b].value, softmax_scale=SCALE, lam=config.lam,
                          device_scores=state.workspace.selection.scores[b])
            _, mutable, current = state.sequence_view(b)
            assert_state_equal(mutable, twins[b].state, f"step {step} seq {b}")
            assert torch.equal(current.cpu(), twins[b].current)
    runtime.assert_no_overflow()


def test_overflow_leaves_the_followers_alone():
    """Beyond the room for decoded tokens a shared graph reports it, and its followers' tables stay as they are."""

    layer = make_layer(seed=43, kv_heads=3, seq_len=1024, communities=16, max_decode_tokens=2, aggregation="layer_wise")
    config = CommunityKVConfig(token_budget=128, num_sink=2, lam=0.5, aggregation="layer_wise")
    device = torch.device("cuda", 0)
    runtime = DecodeRuntime(config, splits=1)
    state = runtime.prepare_layer(0, **layer.to(device).prepare_kwargs())
    twin = OracleLayer(state.converted.csr, state.converted.mutable, state.converted.current_position,
                       token_budget=128, num_sink=2, cover=_cover(state.converted))
    key, value = layer.key.to(device)[None], layer.value.to(device)[None]
    flags = []
    for step in range(5):
        before = [tensor.clone() for tensor in (state.converted.mutable.centroids.view(torch.uint8),
                                                state.converted.mutable.community_sizes,
                                                state.converted.mutable.community_counts)]
        query = make_query(seed=820 + step, query_heads=layer.query_heads)
        runtime.decode(layer_idx=0, query=query.to(device)[None, :, None, :], key=key, value=value, softmax_scale=SCALE)
        want = twin.step(query=query, key=layer.key, value=layer.value, softmax_scale=SCALE, lam=0.5,
                         device_scores=state.workspace.selection.scores)
        assert torch.equal(state.workspace.update.overflow.cpu(), want.overflow), step
        assert_state_equal(state.converted.mutable, twin.state, f"step {step}")
        flags.append(int(state.workspace.update.overflow.max()))
        if flags[-1]:
            after = (state.converted.mutable.centroids.view(torch.uint8), state.converted.mutable.community_sizes,
                     state.converted.mutable.community_counts)
            assert all(torch.equal(x[1:], y[1:]) for x, y in zip(before, after))
    assert flags[0] == 0 and flags[-1] != 0


def test_many_followers_cost_an_update_little():
    """The followers of a shared graph are updated side by side: 63 of them (head after head 45 us) do not triple
    the update's time of three."""

    device = torch.device("cuda", 0)
    config = CommunityKVConfig(token_budget=256, num_sink=3, lam=0.5, aggregation="layer_wise")

    def microseconds(kv_heads):
        layer = make_layer(seed=70, kv_heads=kv_heads, group_size=1, seq_len=1031, communities=24,
                           max_decode_tokens=340, aggregation="layer_wise").to(device)
        runtime = DecodeRuntime(config)
        state = runtime.prepare_layer(0, **layer.prepare_kwargs())
        query = make_query(seed=71, query_heads=kv_heads).to(device)
        runtime.decode(layer_idx=0, query=query.view(1, kv_heads, 1, 128), key=layer.key[None], value=layer.value[None],
                       softmax_scale=SCALE)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(50):
                native.call("ckv_online_update", state.args, native.current_stream(device))
        spans = []
        for _ in range(6):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            begin.record()
            graph.replay()
            end.record()
            end.synchronize()
            spans.append(begin.elapsed_time(end) * 20)
        runtime.assert_no_overflow()
        return min(spans)

    assert microseconds(64) < 3 * microseconds(4)


@pytest.mark.parametrize("communities", [5, 32, 33, 992, 1025])
def test_selection_over_few_communities(monkeypatch, communities):
    """The stand-alone selection keeps a histogram per warp that has a community: one, some and all of the 32 warps."""

    monkeypatch.setenv("CKV_UNFUSED", "1")
    layer = make_layer(seed=60 + communities, seq_len=8192, communities=communities, kv_heads=2, max_decode_tokens=6)
    config = CommunityKVConfig(token_budget=512, num_sink=10, lam=0.5, aggregation="query_group")
    _run_sequence(layer, config, steps=3, seed=6100)


def test_fp32_layers_back_to_back():
    """The kernels of a layer with an fp32 table do not stand in the way of the layer before it: back to back it takes
    about what it takes with a small kernel in between (let go early, an eighth longer)."""

    device = torch.device("cuda", 0)
    layer = make_layer(seed=7, seq_len=8192, communities=64, max_decode_tokens=1000)
    layer.assembled.centroids = layer.assembled.centroids.float()
    layer = layer.to(device)
    runtime = DecodeRuntime(CommunityKVConfig(token_budget=1024, num_sink=10, lam=0.5, aggregation="query_group",
                                              centroid_dtype="fp32"))
    runtime.prepare_layer(0, **layer.prepare_kwargs())
    query = make_query(seed=900, query_heads=layer.query_heads).to(device)[None, :, None, :]
    cache = torch.zeros((2, 8, 16, 128), dtype=torch.bfloat16, device=device)
    row = torch.ones((8, 128), dtype=torch.bfloat16, device=device)

    def microseconds(apart):
        def step():
            if apart:
                ops.append_kv(cache[0], cache[1], row, row, 3)
            runtime.decode(layer_idx=0, query=query, key=layer.key[None], value=layer.value[None], softmax_scale=SCALE)

        step()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(40):
                step()
        spans = []
        for _ in range(6):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            begin.record()
            graph.replay()
            end.record()
            end.synchronize()
            spans.append(begin.elapsed_time(end) * 25)
        return min(spans)

    apart = microseconds(True)
    assert microseconds(False) < 1.08 * apart
    runtime.assert_no_overflow()


def test_full_size_batch_one_launch_equals_four_kernels():
    """The batched long-context configuration as far as one layer goes (8 sequences x 8 KV heads at ctx 131072,
    1024-4096 Zipf communities, budget 2048): the single cluster launch and the four
    stand-alone kernels, fed the same inputs for three steps, leave bit-identical
    workspaces and graph state (one unit of this size is checked against the CPU oracle
    by ``test_zipf_communities_full_context_unit``)."""

    from dataclasses import fields

    from community_kv_b200 import native
    from community_kv_b200.workload import build_decode_workload

    device = torch.device("cuda", 0)

    def build():
        return build_decode_workload(
            layers=1, batch=8, kv_heads=8, group_size=4, seq_len=131072, communities=(1024, 4096),
            token_budget=2048, num_sink=10, max_decode_tokens=8, device=device, seed=3, zipf_exponent=1.1)

    fused, plain = build(), build()
    generator = torch.Generator(device=device).manual_seed(1)
    stream = native.current_stream(device)

    def tensors(obj):
        found = {}
        for item in fields(obj):
            value = getattr(obj, item.name)
            if isinstance(value, torch.Tensor):
                found[item.name] = value
            elif hasattr(value, "__dataclass_fields__"):
                found.update({f"{item.name}.{k}": v for k, v in tensors(value).items()})
        return found

    for step in range(3):
        query = torch.randn((8, 32, 128), generator=generator, device=device).to(torch.bfloat16)
        for work, flag in ((fused, 0), (plain, native.FLAG_UNFUSED)):
            args = work.runtime.pack(0, query=query, key=work.key[0], value=work.value[0], softmax_scale=SCALE)
            args.flags = (args.flags & ~native.FLAG_UNFUSED) | flag
            assert native.library().ckv_decode_layer_kernels(args) == (4 if flag else 1)
            native.call("ckv_decode_layer", args, stream)
        torch.cuda.synchronize()
        left, right = fused.state(0), plain.state(0)
        for name, a in {**tensors(left.workspace), **tensors(left.mutable)}.items():
            b = {**tensors(right.workspace), **tensors(right.mutable)}[name]
            if name.endswith(("partials", "partial_topk_packed", "score_cover")) or not a.numel():
                continue
            same = torch.equal(a.view(torch.uint8) if a.dtype == torch.float8_e4m3fn else a, b.view(torch.uint8) if b.dtype == torch.float8_e4m3fn else b)
            if not same and a.is_floating_point():  # NaN-free by construction; compare bits
                same = torch.equal(a.contiguous().view(torch.int16 if a.element_size() == 2 else torch.int32),
                                   b.contiguous().view(torch.int16 if b.element_size() == 2 else torch.int32))
            assert same, f"step {step}: {name} differs between the two paths"
        assert torch.equal(left.current_position, right.current_position)
    fused.runtime.assert_no_overflow()
