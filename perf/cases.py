"""What a user of this package has it do, as timed cases.

Six kinds of work, all through the public entry points:

* ``token``      one decoded token of one sequence through a few layers: the new row goes into the cache,
                 the layer scores, selects, attends and assigns.  ``plugin`` cases go through the attention
                 plug-in and its static cache, as a Hugging Face ``generate`` does; the others hold a
                 ``DecodeRuntime`` and their own cache.
* ``batch``      the same step for several sequences at once (``BatchedDecodeRuntime``).
* ``prompt``     one layer's prefill through the plug-in: attention and the eight neighbours of every row.
* ``attention``, ``edges``   one layer's prefill by the direct calls: attention alone, and attention with
                 the exact neighbours per KV head.
* ``partition``  what lies between a layer's prefill and its first decoded token, the partition itself
                 excepted: adjacency, modularity weights, decode state, installation in the runtime.

A decode state has room for ``DECODE_TOKENS`` tokens.  A pass decodes the next one; when the room is used
up, the next pass begins the same request anew from a copy of the state as it was after the prompt.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from community_kv_b200 import (
    CommunityKVAttention,
    CommunityKVConfig,
    CommunityKVRuntime,
    DecodeRuntime,
    PartitionConfig,
)
from community_kv_b200.assembly import assemble_layer, build_adjacency, init_modularity_state, reshape_by_aggregation
from community_kv_b200.batched import BatchedDecodeRuntime
from community_kv_b200.cache import StaticCache
from community_kv_b200.ops import append_kv
from community_kv_b200.prefill import prefill_attention, prefill_attention_edges
from community_kv_b200.runtime import convert_prefill_tensors
from community_kv_b200.synthetic import SyntheticPartitionedLayer

HEAD_DIM = 128
SCALE = HEAD_DIM**-0.5
NUM_SINK = 10
KAPPA = 8
LAM = 0.5
DECODE_TOKENS = 128  # tokens generated per request
QUERY_RING = 16  # different tokens a state cycles through

_TOKEN = dict(
    kind="token", plugin=True, layers=6, ctx=32768, kv_heads=8, group=4, communities=512, zipf=True, budget=2048,
    aggregation="query_group", centroids="e4m3", assignment="modularity", top=0, deferred=False,
)
_BATCH = dict(
    kind="batch", layers=3, batch=8, ctx=131072, kv_heads=8, group=4, communities_low=1024, communities_high=4096,
    budget=2048, deferred=True,
)


def listed():
    return [
        # the smallest decode step: one layer of a short context, fp32 mean-key centroids, the eight best
        # communities of every head
        dict(_TOKEN, name="token_8k_top8_fp32", plugin=False, layers=1, ctx=8192, communities=64, zipf=False,
             budget=1024, centroids="fp32", top=8),
        # the package's default settings in a model: a graph per query head, budget 4096, communities of 16 tokens
        dict(_TOKEN, name="token_32k_default", communities=2048, zipf=False, budget=4096, aggregation="per_query_head"),
        # a model whose query groups share a graph, few large communities of very unequal sizes
        dict(_TOKEN, name="token_32k_grouped"),
        # one graph for the whole layer, wide query groups, a length that divides nothing
        dict(_TOKEN, name="token_20k_layer_wise", layers=4, ctx=20011, kv_heads=4, group=8, communities=997, zipf=False,
             budget=1024, aggregation="layer_wise"),
        # the token joins its nearest centroid; the graph update runs beside the next layer
        dict(_TOKEN, name="token_50k_nearest", plugin=False, layers=4, ctx=50021, communities=1500,
             assignment="nearest_centroid", deferred=True),
        # the longest context one GPU decodes: a million tokens, planted clusters, budget 8192
        dict(_TOKEN, name="token_1m", plugin=False, layers=1, ctx=1048576, communities=16384, zipf=False, budget=8192),
        # a serving step: eight sequences of 128K tokens
        dict(_BATCH, name="batch8_128k"),
        # a serving step of few, shorter sequences
        dict(_BATCH, name="batch3_10k", layers=4, batch=3, ctx=10007, group=2, communities_low=100,
             communities_high=700, budget=1024, deferred=False),
        # a short question
        dict(name="prompt_517", kind="prompt", batch=1, length=517, kv_heads=8, group=4),
        # a long document
        dict(name="prompt_16k", kind="prompt", batch=1, length=16384, kv_heads=8, group=4),
        # exact neighbours for a graph per KV head
        dict(name="edges_6k", kind="edges", batch=1, length=6001, kv_heads=8, group=4, edges=16),
        # a layer of an 8K prompt with a graph per query head
        dict(name="partition_8k", kind="partition", ctx=8192, kv_heads=8, group=4, communities=512,
             aggregation="per_query_head"),
    ]


def _spread(rng, low, high):
    """A whole number between ``low`` and ``high``, spread over its logarithm."""

    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["token"] * 4 + ["batch"] * 2 + ["prompt"] * 2 + ["attention", "edges", "partition", "partition"])
    heads = rng.choice([(8, 4), (8, 4), (4, 8), (8, 2), (2, 8), (4, 4), (8, 1)])
    if kind == "token":
        ctx = _spread(rng, 4096, 1048576)
        plugin = ctx <= 131072 and rng.random() < 0.5
        zipf = rng.random() < 0.5
        aggregation = rng.choice(["per_query_head", "per_query_head", "query_group", "query_group", "layer_wise"])
        plain = plugin or rng.random() < 0.5
        return dict(
            _TOKEN, plugin=plugin, layers=rng.randint(2, 4) if ctx <= 131072 else 1, ctx=ctx, kv_heads=heads[0],
            group=heads[1], zipf=zipf,
            communities=_spread(rng, 64, min(4096, ctx // 8) if zipf else min(16384, ctx // 16)),
            budget=rng.choice([b for b in (512, 1024, 2048, 4096, 8192) if b <= ctx // 4]), aggregation=aggregation,
            centroids="e4m3" if plain else rng.choice(["e4m3", "fp32"]), top=0 if plain else rng.choice([0, 8, 64]),
            assignment="modularity" if plain else rng.choice(["modularity", "nearest_centroid"]),
            deferred=not plugin and rng.random() < 0.5,
        )
    if kind == "batch":
        ctx = _spread(rng, 4096, 131072)
        low = _spread(rng, 64, min(1024, ctx // 16))
        return dict(
            _BATCH, layers=rng.randint(2, 3), batch=rng.randint(2, 8), ctx=ctx, kv_heads=heads[0], group=heads[1],
            communities_low=low, communities_high=4 * low, budget=rng.choice([512, 1024, 2048]),
            deferred=rng.random() < 0.5,
        )
    if kind == "partition":
        return dict(
            kind=kind, ctx=_spread(rng, 1024, 8192), kv_heads=heads[0], group=heads[1],
            communities=_spread(rng, 32, 512),
            aggregation=rng.choice(["per_query_head", "query_group", "layer_wise"]),
        )
    case = dict(kind=kind, batch=1 if kind == "prompt" else rng.randint(1, 2),
                length=_spread(rng, 64, 16384 if kind == "prompt" else 8192), kv_heads=heads[0], group=heads[1])
    if kind == "edges":
        case["edges"] = rng.choice([8, 16])
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(generator, *shape):
    return torch.randn(shape, generator=generator, device="cuda", dtype=torch.bfloat16)


def _cluster_rows(generator, heads, tokens, clusters):
    """Cluster of every token ``[heads, tokens]``, none empty; keys ``[heads, tokens, 128]``: centre plus noise."""

    cluster = torch.randint(0, clusters, (heads, tokens), generator=generator, device="cuda")
    cluster[:, NUM_SINK + torch.arange(clusters, device="cuda") * (tokens - NUM_SINK) // clusters] = torch.arange(
        clusters, device="cuda")
    centres = _normal(generator, heads, clusters, HEAD_DIM)
    key = torch.empty((heads, tokens, HEAD_DIM), dtype=torch.bfloat16, device="cuda")
    for head in range(heads):
        key[head] = (centres[head][cluster[head]] + 0.3 * _normal(generator, tokens, HEAD_DIM)) * SCALE
    return cluster, key


def _zipf_labels(generator, counts, tokens):
    """Random communities with sizes proportional to ``rank ** -1.1``, ``counts[i]`` of them in row i, none empty."""

    widest = max(counts)
    share = torch.arange(1, widest + 1, device="cuda", dtype=torch.float32).pow(-1.1).repeat(len(counts), 1)
    number = torch.tensor(counts, device="cuda").view(-1, 1)
    share *= torch.arange(widest, device="cuda") < number
    edge = (share / share.sum(1, keepdim=True)).cumsum(1)
    draw_at = torch.rand((len(counts), tokens), generator=generator, device="cuda")
    rank = torch.searchsorted(edge, draw_at).minimum(number - 1)
    order = torch.rand((len(counts), widest), generator=generator, device="cuda")
    order = order.masked_fill(torch.arange(widest, device="cuda") >= number, 2.0).argsort(1)  # live ids first
    labels = order.gather(1, rank)
    for row, count in enumerate(counts):
        live = torch.arange(count, device="cuda")
        labels[row, NUM_SINK + live * (tokens - NUM_SINK) // count] = live
    return labels


def _graph_labels(generator, per_kv, case):
    """Labels ``[graphs, ctx]`` int32 from the KV heads' labels; the query heads of a group differ in a tenth."""

    if case["aggregation"] == "layer_wise":
        labels = per_kv[:1].clone()
    elif case["aggregation"] == "query_group":
        labels = per_kv.clone()
    else:
        labels = per_kv.repeat_interleave(case["group"], 0)
        other = torch.randint(0, labels.shape[1], labels.shape, generator=generator, device="cuda")
        moved = torch.rand(labels.shape, generator=generator, device="cuda") < 0.1
        labels = torch.where(moved, labels.gather(1, other), labels)
        count = case["communities"]
        first = NUM_SINK + torch.arange(count, device="cuda") * (labels.shape[1] - NUM_SINK) // count
        labels[:, first] = per_kv.repeat_interleave(case["group"], 0)[:, first]
    # the sink positions are no members: they carry labels of their own
    labels[:, :NUM_SINK] = labels.amax(1, keepdim=True) + 1 + torch.arange(NUM_SINK, device="cuda")
    return labels.to(torch.int32)


def _mean_keys(labels, key, assembled):
    """fp32 centroids ``[retrieval heads, capacity, 128]``: the mean key of every community."""

    heads, capacity, _ = assembled.centroids.shape
    rows = labels[assembled.retrieval_to_graph.long(), NUM_SINK:].long()
    total = torch.zeros((heads, capacity, HEAD_DIM), device="cuda")
    for head in range(heads):
        total[head].index_add_(0, rows[head], key[int(assembled.retrieval_to_kv[head]), NUM_SINK:].float())
    return total / assembled.community_sizes.clamp(min=1).unsqueeze(-1)


def _layer_tensors(assembled, case, ctx):
    return dict(
        member_offsets=assembled.member_offsets, member_positions=assembled.member_positions,
        num_communities=assembled.num_communities, centroids=assembled.centroids,
        community_sizes=assembled.community_sizes, community_weight=assembled.community_weight,
        total_weight=assembled.total_weight, token_communities=assembled.token_communities,
        retrieval_to_graph=assembled.retrieval_to_graph, retrieval_to_kv=assembled.retrieval_to_kv,
        prefill_seq_len=ctx, max_decode_tokens=DECODE_TOKENS,
        group_size=case["kv_heads"] * case["group"] // assembled.retrieval_to_graph.numel(),
        aggregation=case.get("aggregation", "query_group"), query_heads=case["kv_heads"] * case["group"],
        kv_heads=case["kv_heads"],
    )


def _rings(generator, layers, lead, query_heads, key):
    """``QUERY_RING`` tokens: queries of one topic (their correlation is 0.64), keys like the cached ones."""

    topic = torch.randn((layers, *lead, query_heads, HEAD_DIM), generator=generator, device="cuda")
    query = 0.8 * topic + 0.6 * torch.randn((QUERY_RING, *topic.shape), generator=generator, device="cuda")
    old = torch.stack([k[..., 100 : 100 + QUERY_RING, :] for k in key])  # [layers, *lead, Hkv, ring, 128]
    fresh_key = old.movedim(-2, 0) + 0.1 * SCALE * _normal(generator, QUERY_RING, *old.shape[:-2], HEAD_DIM)
    fresh_value = SCALE * _normal(generator, *fresh_key.shape)
    return query.to(torch.bfloat16), fresh_key.contiguous(), fresh_value


def _decode_state(layers, extra=()):
    """Every tensor a decode step changes, and a copy of it as it is now."""

    live = []
    for layer in layers:
        mutable = getattr(layer, "mutable", None) or layer.converted.mutable
        position = layer.current_position if hasattr(layer, "current_position") else layer.converted.current_position
        live += [t for t in mutable.tensors()
                 if t is not mutable.retrieval_to_graph and t is not mutable.retrieval_to_kv] + [position]
    live += list(extra)
    # one-byte views where copying a type is a matter of its bytes
    live = [t.view(torch.uint8) if t.dtype == torch.float8_e4m3fn else t for t in live]
    return live, [t.clone() for t in live]


def _decode_outputs(layer):
    mutable = getattr(layer, "mutable", None) or layer.converted.mutable
    attention = layer.workspace.attention
    centroids = mutable.centroids
    return [
        attention.output, attention.lse, attention.topk_scores, attention.topk_positions,
        layer.workspace.update.assigned_communities, mutable.community_sizes, mutable.community_weight,
        mutable.token_communities, mutable.deltas.positions,
        centroids.view(torch.uint8) if centroids.dtype == torch.float8_e4m3fn else centroids,
    ]


def _prepare_token(case, seed):
    generator = _generator(seed)
    ctx, kv_heads, group = case["ctx"], case["kv_heads"], case["group"]
    rows = ctx + DECODE_TOKENS
    keys, values, tensors = [], [], []
    for _ in range(case["layers"]):
        if case["zipf"]:
            per_kv = _zipf_labels(generator, [case["communities"]] * kv_heads, ctx)
            key = SCALE * _normal(generator, kv_heads, ctx, HEAD_DIM)
        else:
            per_kv, key = _cluster_rows(generator, kv_heads, ctx, case["communities"])
        labels = _graph_labels(generator, per_kv, case)
        assembled = assemble_layer(labels, key, aggregation=case["aggregation"], query_heads=kv_heads * group,
                                   num_sink=NUM_SINK, max_decode_tokens=DECODE_TOKENS)
        if case["centroids"] == "fp32":
            assembled.centroids = _mean_keys(labels, key, assembled)
        tensors.append(_layer_tensors(assembled, case, ctx))
        keys.append(key[None])
        values.append(SCALE * _normal(generator, 1, kv_heads, ctx, HEAD_DIM))
    query, fresh_key, fresh_value = _rings(generator, case["layers"], (1,), kv_heads * group, keys)
    config = CommunityKVConfig(token_budget=case["budget"], num_sink=NUM_SINK, lam=LAM, aggregation=case["aggregation"],
                               online_assignment=case["assignment"], centroid_dtype=case["centroids"])
    s = SimpleNamespace(step=0, layers=range(case["layers"]), ctx=ctx)
    s.tokens = [[(query[r, i].unsqueeze(-2), fresh_key[r, i].unsqueeze(-2), fresh_value[r, i].unsqueeze(-2))
                 for i in s.layers] for r in range(QUERY_RING)]
    if case["plugin"]:
        def partitioned(layer_idx, **_):
            t = tensors[layer_idx]
            return SyntheticPartitionedLayer(
                layer_idx=layer_idx, community_counts=t["num_communities"],
                **{k: v for k, v in t.items() if k not in ("num_communities", "max_decode_tokens", "group_size")})

        runtime = CommunityKVRuntime(config=config, partition=PartitionConfig(), num_layers=case["layers"],
                                     max_decode_tokens=DECODE_TOKENS, partitioner=partitioned)
        runtime.start_request()
        s.cache = StaticCache(num_hidden_layers=case["layers"], max_cache_len=rows)
        for i in s.layers:
            s.cache.update(keys[i], values[i], i)
            runtime.submit_prefill_layer(layer_idx=i, topk_indices=None, topk_scores=None, keys=keys[i][0],
                                         completion_event=None)
        runtime.finish_prefill()
        s.cache.enable_device_updates()
        s.attention = CommunityKVAttention(runtime)
        s.modules = [SimpleNamespace(layer_idx=i) for i in s.layers]
        s.runtime = runtime.decode_runtime
        cursors = [s.cache.layer(i).cumulative_length for i in s.layers]
    else:
        s.runtime = DecodeRuntime(config, defer_update=case["deferred"], max_communities=case["top"])
        for i in s.layers:
            s.runtime.prepare_layer(i, **tensors[i])
        room = torch.zeros((1, kv_heads, DECODE_TOKENS, HEAD_DIM), dtype=torch.bfloat16, device="cuda")
        s.keys = [torch.cat((k, room), 2) for k in keys]
        s.values = [torch.cat((v, room), 2) for v in values]
        cursors = []
    prepared = [s.runtime.layers[i] for i in s.layers]
    s.live, s.saved = _decode_state(prepared, cursors)
    s.outputs = [_decode_outputs(layer) for layer in prepared]
    return s


def _prepare_batch(case, seed):
    generator = _generator(seed)
    ctx, kv_heads, group, batch = case["ctx"], case["kv_heads"], case["group"], case["batch"]
    host = torch.Generator().manual_seed(seed)
    config = CommunityKVConfig(token_budget=case["budget"], num_sink=NUM_SINK, lam=LAM, aggregation="query_group")
    s = SimpleNamespace(step=0, layers=range(case["layers"]), ctx=ctx, keys=[], values=[])
    s.runtime = BatchedDecodeRuntime(config, defer_update=case["deferred"])
    for i in s.layers:
        key = SCALE * _normal(generator, batch, kv_heads, ctx + DECODE_TOKENS, HEAD_DIM)
        value = SCALE * _normal(generator, *key.shape)
        sequences = []
        for b in range(batch):
            counts = torch.randint(case["communities_low"], case["communities_high"] + 1, (kv_heads,), generator=host)
            counts[b % kv_heads] = case["communities_high"]  # the widest head sets the capacity of all
            labels = _zipf_labels(generator, counts.tolist(), ctx).to(torch.int32)
            assembled = assemble_layer(labels, key[b, :, :ctx], aggregation="query_group", query_heads=kv_heads * group,
                                       num_sink=NUM_SINK, max_decode_tokens=DECODE_TOKENS)
            sequences.append(convert_prefill_tensors(**_layer_tensors(assembled, case, ctx)))
        s.runtime.prepare_layer(i, sequences)
        s.keys.append(key)
        s.values.append(value)
    query, fresh_key, fresh_value = _rings(generator, case["layers"], (batch,), kv_heads * group, s.keys)
    s.tokens = [[(query[r, i], fresh_key[r, i], fresh_value[r, i]) for i in s.layers] for r in range(QUERY_RING)]
    prepared = [s.runtime.layers[i] for i in s.layers]
    s.live, s.saved = _decode_state(prepared)
    s.outputs = [_decode_outputs(layer) for layer in prepared]
    return s


def _prepare_prefill(case, seed):
    generator = _generator(seed)
    batch, length, kv_heads = case["batch"], case["length"], case["kv_heads"]
    _, key = _cluster_rows(generator, batch * kv_heads, length, max(1, min(256, length // 4)))
    key = key.view(batch, kv_heads, length, HEAD_DIM)
    value = SCALE * _normal(generator, *key.shape)
    query = _normal(generator, batch, length, kv_heads * case["group"], HEAD_DIM)
    s = SimpleNamespace(query=query, key=key, value=value)
    if case["kind"] == "prompt":
        s.edges = []

        def keep(*, topk_indices, topk_scores, **_):  # stands where the host's partition begins
            s.edges[:] = [topk_indices, topk_scores]

        s.runtime = CommunityKVRuntime(config=CommunityKVConfig(num_sink=NUM_SINK), partition=PartitionConfig(),
                                       num_layers=1, max_decode_tokens=DECODE_TOKENS, partitioner=keep)
        s.attention = CommunityKVAttention(s.runtime)
        s.module = SimpleNamespace(layer_idx=0)
        # the plug-in is handed [B, H, S, 128]: the query a view of the projection, K and V the cache's rows
        s.query = query.transpose(1, 2)
        room = torch.zeros((batch, kv_heads, DECODE_TOKENS, HEAD_DIM), dtype=torch.bfloat16, device="cuda")
        s.key, s.value = torch.cat((key, room), 2), torch.cat((value, room), 2)
    else:
        s.key, s.value = key.transpose(1, 2).contiguous(), value.transpose(1, 2).contiguous()
        s.count = case.get("edges", 0)
    return s


def _prepare_partition(case, seed):
    generator = _generator(seed)
    ctx, kv_heads, heads = case["ctx"], case["kv_heads"], case["kv_heads"] * case["group"]
    per_kv, key = _cluster_rows(generator, kv_heads, ctx, case["communities"])
    labels = _graph_labels(generator, per_kv, case)
    # neighbours of a row: earlier members of its cluster, a few skipped at random; the newest rows before it
    # where the cluster has too few.  Scores: falling shares of a softmax.
    first = NUM_SINK + KAPPA - 1
    rows = ctx - first
    order = per_kv.argsort(dim=1, stable=True)  # members of a cluster side by side, oldest first
    place = torch.empty_like(order).scatter_(1, order, torch.arange(ctx, device="cuda").expand(kv_heads, -1))
    begin = torch.searchsorted(per_kv.gather(1, order).contiguous(), per_kv.contiguous())
    rank = (place - begin).repeat_interleave(case["group"], 0)[:, first:]
    place = place.repeat_interleave(case["group"], 0)[:, first:]
    order = order.repeat_interleave(case["group"], 0)
    back = (1 + torch.rand((heads, rows, KAPPA), generator=generator, device="cuda").mul(1.6).long()).cumsum(-1)
    found = order.gather(1, (place.unsqueeze(-1) - back).clamp(min=0).view(heads, -1)).view(heads, rows, KAPPA)
    recent = torch.arange(first, ctx, device="cuda").view(1, -1, 1) - torch.arange(KAPPA, device="cuda")
    neighbour = torch.where((back <= rank.unsqueeze(-1)) & (found >= NUM_SINK), found, recent)
    score = torch.rand((heads, rows, KAPPA), generator=generator, device="cuda").mul(0.1)
    score = score.sort(-1, descending=True).values
    config = CommunityKVConfig(token_budget=512, num_sink=NUM_SINK, lam=LAM, aggregation=case["aggregation"])
    # where the host's partition takes the edges from: room for all that the rows can enumerate
    room = heads * rows * (KAPPA + KAPPA * (KAPPA + 1) // 2)
    edges = [torch.zeros(room, dtype=dtype, device="cuda") for dtype in (torch.int32, torch.int32, torch.float32)]
    return SimpleNamespace(case=case, config=config, key=key, labels=labels, edges=edges,
                           neighbour=neighbour.to(torch.int32).contiguous(), score=score.contiguous())


_PREPARE = {"token": _prepare_token, "batch": _prepare_batch, "partition": _prepare_partition}


def prepare(case, seed):
    state = _PREPARE.get(case["kind"], _prepare_prefill)(case, seed)
    state.kind = case["kind"]
    return state


# ---- passes ------------------------------------------------------------------------------------------------------


def _next_token(s):
    """Row of the next token in the sequence; a new request when the last one has used up its room."""

    if s.step == DECODE_TOKENS:
        s.runtime.synchronize_updates()
        torch._foreach_copy_(s.live, s.saved)
        s.step = 0
    s.step += 1
    return s.ctx + s.step - 1


def _run_token(s):
    row = _next_token(s)
    token = s.tokens[s.step % QUERY_RING]
    if hasattr(s, "attention"):
        for i in s.layers:
            query, key, value = token[i]
            keys, values = s.cache.update(key, value, i)
            s.attention.forward(s.modules[i], query, keys, values, None, SCALE)
    else:
        for i in s.layers:
            query, key, value = token[i]
            append_kv(s.keys[i], s.values[i], key.squeeze(-2), value.squeeze(-2), row)
            s.runtime.decode(layer_idx=i, query=query, key=s.keys[i], value=s.values[i], softmax_scale=SCALE)
    return s.outputs


def _run_batch(s):
    row = _next_token(s)
    token = s.tokens[s.step % QUERY_RING]
    for i in s.layers:
        query, key, value = token[i]
        append_kv(s.keys[i], s.values[i], key, value, row)
        s.runtime.decode(layer_idx=i, query=query, key=s.keys[i], value=s.values[i], softmax_scale=SCALE)
    return s.outputs


def _run_partition(s):
    case = s.case
    ctx, heads = case["ctx"], case["kv_heads"] * case["group"]
    shaped = reshape_by_aggregation(s.neighbour, s.score, aggregation=case["aggregation"],
                                    num_kv_heads=case["kv_heads"], num_sink=NUM_SINK)
    source, destination, weight = build_adjacency(*shaped, seq_len=ctx, lam=LAM)
    for room, found in zip(s.edges, (source, destination, weight)):
        room[: found.numel()].copy_(found)
    capacity = int(s.labels.max()) + 1 + DECODE_TOKENS
    community_weight, total_weight = init_modularity_state(s.labels, source, destination, weight,
                                                           community_capacity=capacity)
    assembled = assemble_layer(s.labels, s.key, aggregation=case["aggregation"], query_heads=heads, num_sink=NUM_SINK,
                               max_decode_tokens=DECODE_TOKENS, community_weight=community_weight,
                               total_weight=total_weight)
    layer = DecodeRuntime(s.config).prepare_layer(0, **_layer_tensors(assembled, case, ctx))
    mutable, csr = layer.converted.mutable, layer.converted.csr
    return [*s.edges, csr.member_offsets, csr.member_positions, csr.community_counts,
            mutable.centroids.view(torch.uint8), mutable.community_sizes, mutable.community_weight,
            mutable.total_weight, mutable.token_communities, layer.converted.current_position]


def _run_prompt(s):
    s.runtime.start_request()
    out, _ = s.attention.forward(s.module, s.query, s.key, s.value, None, SCALE)
    return [out, *s.edges]


def _run_edges(s):
    out, lse, index, score, _ = prefill_attention_edges(
        s.query, s.key, s.value, softmax_scale=SCALE, num_sink=NUM_SINK, edges_per_row=s.count)
    return [out, lse, index, score]


def _run_attention(s):
    return list(prefill_attention(s.query, s.key, s.value, softmax_scale=SCALE))


_RUN = {"token": _run_token, "batch": _run_batch, "partition": _run_partition, "prompt": _run_prompt,
        "edges": _run_edges, "attention": _run_attention}


def run(state):
    return _RUN[state.kind](state)


# ---- what a pass cannot do without -------------------------------------------------------------------------------


def work(case):
    if case["kind"] in ("token", "batch"):
        query_heads = case["kv_heads"] * case["group"]
        if case["kind"] == "token":
            heads = max(query_heads if case["aggregation"] == "per_query_head" else 0, case["kv_heads"])
            batch, communities = 1, case["communities"]
            row = HEAD_DIM * (4 if case["centroids"] == "fp32" else 1)
            tokens = case["budget"]
            if case["top"]:
                tokens = min(tokens, NUM_SINK + 1 + case["top"] * case["ctx"] // communities)
            scans = 2 if case["assignment"] == "nearest_centroid" else 1
        else:
            heads, batch, row, scans = case["kv_heads"], case["batch"], HEAD_DIM, 1
            communities, tokens = (case["communities_low"] + case["communities_high"]) // 2, case["budget"]
        units = case["layers"] * batch * heads
        # the head's centroids and sizes, the selected K and V rows, the query group in and out
        moved = units * (communities * (row + 4) + tokens * 2 * 2 * HEAD_DIM)
        moved += case["layers"] * batch * query_heads * 2 * 2 * HEAD_DIM
        per_row = case["layers"] * batch * query_heads * 2 * HEAD_DIM
        return {"bytes": moved, "flops": per_row * (scans * communities + 2 * tokens)}
    if case["kind"] == "partition":
        ctx, heads = case["ctx"], case["kv_heads"] * case["group"]
        graphs = {"per_query_head": heads, "query_group": case["kv_heads"], "layer_wise": 1}[case["aggregation"]]
        retrieval = max(graphs, case["kv_heads"])
        rows = heads * (ctx - NUM_SINK - KAPPA + 1)
        # neighbours and scores in; of the 44 edges a row enumerates about 18 are new to its graph, about 6
        # where the query heads of a group share it
        moved = rows * (KAPPA * 8 + (18 if graphs == heads else 6) * 12)
        moved += graphs * ctx * 3 * 4 + case["kv_heads"] * ctx * 2 * HEAD_DIM  # labels in and out, members, keys
        moved += retrieval * (case["communities"] + DECODE_TOKENS) * (HEAD_DIM + 12)
        return {"bytes": moved, "flops": rows * 44 * 3 + retrieval * ctx * HEAD_DIM}
    batch, length, kv_heads = case["batch"], case["length"], case["kv_heads"]
    query_heads = kv_heads * case["group"]
    moved = batch * length * (2 * query_heads + 2 * kv_heads) * 2 * HEAD_DIM  # Q in, O out, K and V in
    moved += batch * length * {"prompt": query_heads * KAPPA * 8, "edges": kv_heads * case.get("edges", 0) * 8,
                               "attention": 0}[case["kind"]]
    return {"bytes": moved, "flops": 2 * batch * length * length * HEAD_DIM * query_heads}


def tolerance(case):
    if case["kind"] == "partition":
        # fp32 sums in another order; every whole value is exact
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "prompt":
        # bf16 attention; neighbours are ranked by a score rounded to 1/256, whose last bit is the hardware's
        return {"rel": 1e-2, "max": 0.1, "differ": 1e-2}
    # bf16 attention; selection, neighbours and graph state are exact
    return {"rel": 1e-2, "max": 0.1}
