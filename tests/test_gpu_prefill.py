"""The prefill score-graph kernel (tcgen05) against the CPU oracle, through the C ABI."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from community_kv_b200 import native
from community_kv_b200.prefill import (
    _pack,
    check_status,
    prefill_attention,
    prefill_attention_edges,
    prefill_attention_topk,
)
from oracle import prefill_oracle as oracle

pytestmark = pytest.mark.gpu
SCALE = 128 ** -0.5


def _inputs(seed, length, heads, kv_heads, clusters=16, batch=1):
    generator = torch.Generator().manual_seed(seed)
    centres = torch.randn((kv_heads, clusters, 128), generator=generator)
    labels = torch.randint(0, clusters, (batch, length, kv_heads), generator=generator)
    key = centres[torch.arange(kv_heads).view(1, 1, -1), labels] + 0.3 * torch.randn(
        (batch, length, kv_heads, 128), generator=generator
    )
    value = torch.randn((batch, length, kv_heads, 128), generator=generator)
    query = torch.randn((batch, length, heads, 128), generator=generator)
    # planted structure: queries lean towards their own cluster centre
    query = query + 0.5 * key.repeat_interleave(heads // kv_heads, dim=2)
    return (query.to(torch.bfloat16), (key / 128**0.5).to(torch.bfloat16) * 4, (value / 128**0.5).to(torch.bfloat16))


def _check_attention(out, lse, q, k, v, want_out, want_lse):
    diff = (out.float().cpu().numpy() - want_out)
    assert np.abs(diff).max() <= 2e-2, np.abs(diff).max()
    assert np.abs(diff).mean() <= 1e-3
    np.testing.assert_allclose(lse.cpu().numpy(), want_lse, atol=2e-3, rtol=0)


@pytest.mark.parametrize(
    "length,heads,kv_heads",
    [(256, 4, 1), (300, 8, 2), (640, 2, 2), (200, 8, 1), (512, 2, 1), (64, 4, 2), (1, 2, 1), (130, 4, 1), (129, 2, 2)],
)
def test_attention_output_and_lse(length, heads, kv_heads):
    q, k, v = _inputs(1, length, heads, kv_heads)
    out, lse = prefill_attention(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE)
    torch.cuda.synchronize()
    want_out, want_lse, _ = oracle.causal_attention(q[0].float().numpy(), k[0].float().numpy(), v[0].float().numpy(), SCALE)
    _check_attention(out[0], lse[0], q, k, v, want_out, want_lse)


def test_reference_topk_rule():
    length, heads, kv_heads, sinks = 640, 4, 1, 10
    q, k, v = _inputs(2, length, heads, kv_heads)
    out, lse, _, _, val, idx = prefill_attention_topk(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks)
    torch.cuda.synchronize()
    assert val.shape == (1, heads, length - sinks - 7, 8) and idx.dtype == torch.int32
    want_out, want_lse, raw = oracle.causal_attention(q[0].float().numpy(), k[0].float().numpy(), v[0].float().numpy(), SCALE)
    _check_attention(out[0], lse[0], q, k, v, want_out, want_lse)
    got_idx = idx[0].cpu().numpy()
    got_val = val[0].cpu().numpy()
    exact_rows = 0
    total_rows = 0
    for head in range(heads):
        want_val, want_idx, want_key = oracle.reference_topk(raw[head], want_lse[head], SCALE, sinks)
        keys = oracle.quantised_keys(raw[head])
        for row in range(want_idx.shape[0]):
            position = row + sinks + 7
            total_rows += 1
            mine = got_idx[head, row]
            assert mine.min() >= sinks and mine.max() <= position
            assert len(set(mine.tolist())) == 8
            if np.array_equal(mine, want_idx[row]):
                exact_rows += 1
                np.testing.assert_allclose(got_val[head, row], want_val[row], rtol=2e-2, atol=1e-9)
                continue
            # the tensor-core score may land on the other side of a quantisation step:
            # every disagreement must sit within one step of the cut
            floor_key = want_key[row].min()
            for j in set(mine.tolist()) ^ set(want_idx[row].tolist()):
                assert abs(int(keys[position, j]) - int(floor_key)) <= 1, (head, row, j)
    assert exact_rows / total_rows > 0.97, exact_rows / total_rows


@pytest.mark.parametrize(
    "length,heads,kv_heads,edges",
    [(384, 4, 1, 16), (300, 8, 2, 8), (260, 2, 2, 16), (320, 4, 2, 16), (272, 8, 1, 16), (700, 8, 2, 16)],
)
def test_exact_edges_are_bit_exact(length, heads, kv_heads, edges):
    sinks = 4
    q, k, v = _inputs(3, length, heads, kv_heads)
    out, lse, edge_idx, edge_score, flags = prefill_attention_edges(
        q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks, edges_per_row=edges
    )
    torch.cuda.synchronize()
    want_idx, want_score = oracle.exact_edges(q[0].float().numpy(), k[0].float().numpy(), SCALE, sinks, edges)
    assert np.array_equal(edge_idx[0].cpu().numpy(), want_idx)
    assert np.array_equal(edge_score[0].cpu().numpy().view(np.uint32), want_score.view(np.uint32))
    want_out, want_lse, _ = oracle.causal_attention(q[0].float().numpy(), k[0].float().numpy(), v[0].float().numpy(), SCALE)
    _check_attention(out[0], lse[0], q, k, v, want_out, want_lse)
    assert int(flags.sum()) <= flags.numel() // 20


@pytest.mark.parametrize("length,heads,kv_heads,batch", [(896, 2, 2, 2), (897, 2, 2, 2), (1100, 3, 3, 1), (1000, 8, 1, 2)])
def test_exact_edges_head_after_head(length, heads, kv_heads, batch):
    """On both sides of the line between tiles of all heads by length and one head's tiles behind another's."""

    sinks, edges = 4, 16
    q, k, v = _inputs(17, length, heads, kv_heads, batch=batch)
    _, _, edge_idx, edge_score, _ = prefill_attention_edges(
        q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks, edges_per_row=edges)
    for b in range(batch):
        want_idx, want_score = oracle.exact_edges(q[b].float().numpy(), k[b].float().numpy(), SCALE, sinks, edges)
        assert np.array_equal(edge_idx[b].cpu().numpy(), want_idx)
        assert np.array_equal(edge_score[b].cpu().numpy().view(np.uint32), want_score.view(np.uint32))


@pytest.mark.parametrize("length,heads,kv_heads,sinks", [(100, 4, 2, 4), (129, 8, 2, 0), (12, 2, 1, 3), (9, 4, 1, 4)])
def test_reference_topk_rule_short_and_ragged(length, heads, kv_heads, sinks):
    """Rows shorter than one tile, a tile of a single row, a prompt barely longer than the sinks."""

    q, k, v = _inputs(6, length, heads, kv_heads)
    out, lse, _, _, val, idx = prefill_attention_topk(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks)
    torch.cuda.synchronize()
    rows = max(0, length - sinks - 7)
    assert val.shape == (1, heads, rows, 8) and idx.shape == (1, heads, rows, 8)
    want_out, want_lse, raw = oracle.causal_attention(q[0].float().numpy(), k[0].float().numpy(), v[0].float().numpy(), SCALE)
    _check_attention(out[0], lse[0], q, k, v, want_out, want_lse)
    for head in range(heads):
        if rows == 0:
            break
        want_val, want_idx, want_key = oracle.reference_topk(raw[head], want_lse[head], SCALE, sinks)
        keys = oracle.quantised_keys(raw[head])
        got_idx = idx[0, head].cpu().numpy()
        for row in range(rows):
            position = row + sinks + 7
            mine = got_idx[row]
            assert mine.min() >= sinks and mine.max() <= position and len(set(mine.tolist())) == 8
            floor_key = want_key[row].min()
            for j in set(mine.tolist()) ^ set(want_idx[row].tolist()):
                assert abs(int(keys[position, j]) - int(floor_key)) <= 1, (head, row, j)


@pytest.mark.parametrize("length,kv_heads", [(35, 1), (462, 4), (463, 4), (700, 4)])
def test_exact_edges_of_eight_heads_per_group(length, kv_heads):
    """Four rounds of candidates per row, on both sides of the line between few rows and many (444 CTAs of four)."""

    sinks, edges = 4, 16
    q, k, v = _inputs(19, length, 8 * kv_heads, kv_heads)
    _, _, edge_idx, edge_score, _ = prefill_attention_edges(
        q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks, edges_per_row=edges)
    want_idx, want_score = oracle.exact_edges(q[0].float().numpy(), k[0].float().numpy(), SCALE, sinks, edges)
    assert np.array_equal(edge_idx[0].cpu().numpy(), want_idx)
    assert np.array_equal(edge_score[0].cpu().numpy().view(np.uint32), want_score.view(np.uint32))


def test_exact_edges_of_a_prompt_shorter_than_the_list():
    q, k, v = _inputs(7, 12, 4, 2)
    out, lse, edge_idx, edge_score, flags = prefill_attention_edges(
        q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=4, edges_per_row=16)
    torch.cuda.synchronize()
    assert edge_idx.shape == (1, 2, 0, 16) and edge_score.shape == (1, 2, 0, 16) and flags.numel() == 0
    want_out, want_lse, _ = oracle.causal_attention(q[0].float().numpy(), k[0].float().numpy(), v[0].float().numpy(), SCALE)
    _check_attention(out[0], lse[0], q, k, v, want_out, want_lse)


def test_exact_edges_rescan_path():
    """A huge slack flags every row: the brute-force re-scan must give the same exact answer."""

    length, heads, kv_heads, edges, sinks = 200, 4, 1, 16, 3
    q, k, v = _inputs(4, length, heads, kv_heads)
    _, _, edge_idx, edge_score, flags = prefill_attention_edges(
        q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks, edges_per_row=edges, exact_slack=1e9
    )
    torch.cuda.synchronize()
    want_idx, want_score = oracle.exact_edges(q[0].float().numpy(), k[0].float().numpy(), SCALE, sinks, edges)
    assert np.array_equal(edge_idx[0].cpu().numpy(), want_idx)
    assert np.array_equal(edge_score[0].cpu().numpy().view(np.uint32), want_score.view(np.uint32))


@pytest.mark.parametrize("batch,kv_heads,length,slack", [(1, 2, 700, 1e-3), (1, 2, 700, 1e9), (2, 32, 2500, 1e-3)])
def test_exact_edges_without_a_queue(batch, kv_heads, length, slack):
    """The queue of rows to scan again is optional: without it the flags lead to the same edges, with few rows, with
    all of them, and with more rows than the launch looks at in one go."""

    generator = torch.Generator(device="cuda").manual_seed(length)
    q, k = (torch.randn((batch, length, kv_heads, 128), generator=generator, device="cuda").to(torch.bfloat16)
            for _ in range(2))
    _, _, want_idx, want_score, want_flags = prefill_attention_edges(
        q, k, k, softmax_scale=SCALE, num_sink=3, edges_per_row=16, exact_slack=slack)
    rows = length - 18
    assert 0 < int(want_flags.sum()) and (slack < 1 or int(want_flags.sum()) > 0.9 * want_flags.numel())
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    args, *keep = _pack(q, k, k, softmax_scale=SCALE, num_sink=3, mode=2, edges_per_row=16, exact_slack=slack,
                        status=status)
    candidates = torch.empty((batch, kv_heads, length, 1, 17), dtype=torch.int64, device="cuda")
    edge_idx = torch.full((batch, kv_heads, rows, 16), -2, dtype=torch.int32, device="cuda")
    edge_score = torch.zeros((batch, kv_heads, rows, 16), device="cuda")
    flags = torch.empty((batch, kv_heads, rows), dtype=torch.int32, device="cuda")
    native.fill(args, candidates=candidates.data_ptr(), edge_idx=edge_idx.data_ptr(), edge_score=edge_score.data_ptr(),
                edge_flags=flags.data_ptr(), rescan_list=None)
    native.call("ckv_prefill_topk", args, native.current_stream(q.device))
    check_status(status)
    del keep  # the tensors that the launch wrote and read
    assert torch.equal(edge_idx, want_idx) and torch.equal(edge_score, want_score) and torch.equal(flags, want_flags)


def test_batch_and_validation():
    q, k, v = _inputs(5, 192, 4, 2, batch=2)
    out, lse = prefill_attention(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE)
    torch.cuda.synchronize()
    for b in range(2):
        want_out, want_lse, _ = oracle.causal_attention(q[b].float().numpy(), k[b].float().numpy(), v[b].float().numpy(), SCALE)
        _check_attention(out[b], lse[b], q, k, v, want_out, want_lse)
    # caller-owned status word: the calls queue without a host round trip, one check at the end
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    again, _ = prefill_attention(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, status=status)
    prefill_attention_topk(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=4, status=status)
    check_status(status)
    assert torch.equal(again, out)
    with pytest.raises(ValueError):
        prefill_attention(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, status=status.to(torch.int64))
    with pytest.raises(RuntimeError):
        check_status(torch.full((1,), 4, dtype=torch.int32, device="cuda"))
    with pytest.raises(TypeError):
        prefill_attention(q.cuda().float(), k.cuda(), v.cuda(), softmax_scale=SCALE)
    with pytest.raises(ValueError):
        prefill_attention(q.cuda()[:, :, :3], k.cuda(), v.cuda(), softmax_scale=SCALE)


def test_full_size_properties():
    """The prefill configuration at full size (S = 16384, 32 / 8 heads, 256 planted clusters): sampled rows
    against fp32 torch arithmetic - attention within tolerance; every edge's score is the group
    maximum of that key, edges are sorted, and nothing outside the list beats the last edge."""

    device = torch.device("cuda", 0)
    length, heads, kv_heads, sinks, edges = 16384, 32, 8, 10, 16
    generator = torch.Generator(device=device).manual_seed(9)
    centres = torch.randn((kv_heads, 256, 128), generator=generator, device=device)
    labels = torch.randint(0, 256, (length, kv_heads), generator=generator, device=device)
    key = centres[torch.arange(kv_heads, device=device), labels] + 0.3 * torch.randn(
        (length, kv_heads, 128), generator=generator, device=device)
    key = (key * SCALE).to(torch.bfloat16)[None]
    value = (torch.randn((1, length, kv_heads, 128), generator=generator, device=device) * SCALE).to(torch.bfloat16)
    query = torch.randn((1, length, heads, 128), generator=generator, device=device).to(torch.bfloat16)
    out, lse, edge_idx, edge_score, flags = prefill_attention_edges(
        query, key, value, softmax_scale=SCALE, num_sink=sinks, edges_per_row=edges)
    torch.cuda.synchronize()
    skip = sinks + edges - 1
    group = heads // kv_heads
    rows = torch.randint(skip, length, (48,), generator=generator, device=device).tolist() + [skip, length - 1]
    k32, v32 = key[0].float(), value[0].float()
    for row in rows:
        q_row = query[0, row].float()  # [heads, 128]
        scores = torch.einsum("hd,jhd->hj", q_row.view(kv_heads, group, 128).reshape(heads, 128),
                              k32[: row + 1].repeat_interleave(group, dim=1)) * SCALE
        probabilities = torch.softmax(scores, dim=-1)
        want = torch.einsum("hj,jhd->hd", probabilities, v32[: row + 1].repeat_interleave(group, dim=1))
        assert float((out[0, row].float() - want).abs().max()) <= 2e-2, row
        best = scores.view(kv_heads, group, row + 1).amax(dim=1)  # [kv, keys]
        best[:, :sinks] = float("-inf")
        got_idx = edge_idx[0, :, row - skip].long()
        got_score = edge_score[0, :, row - skip]
        assert bool((got_idx >= sinks).all()) and bool((got_idx <= row).all()), row
        assert bool((got_score[:, :-1] >= got_score[:, 1:]).all()), row
        torch.testing.assert_close(got_score, best.gather(1, got_idx), rtol=0, atol=2e-5)
        rest = best.scatter(1, got_idx, float("-inf"))
        assert bool((rest.amax(dim=1) <= got_score[:, -1] + 2e-5).all()), row
    assert int(flags.sum()) <= flags.numel() // 100


def test_full_size_reference_topk_rule():
    """The reference's top-8 rule at full size (S = 16384, 32 / 8 heads): for sampled rows the rule is
    restated in fp32 torch arithmetic - key15 = clamp(rn((q.k + 48) * 256)), four column classes keep
    their six best packed candidates, the row reports the eight largest.  The kernel's scores come from
    the tensor cores, so a disagreement is accepted only where the keys involved sit within one
    quantisation step of the cut; the reported probabilities must match exp(score * scale - lse)."""

    device = torch.device("cuda", 0)
    length, heads, kv_heads, sinks = 16384, 32, 8, 10
    generator = torch.Generator(device=device).manual_seed(11)
    centres = torch.randn((kv_heads, 256, 128), generator=generator, device=device)
    labels = torch.randint(0, 256, (length, kv_heads), generator=generator, device=device)
    key = centres[torch.arange(kv_heads, device=device), labels] + 0.3 * torch.randn(
        (length, kv_heads, 128), generator=generator, device=device)
    key = (key * SCALE).to(torch.bfloat16)[None]
    value = (torch.randn((1, length, kv_heads, 128), generator=generator, device=device) * SCALE).to(torch.bfloat16)
    query = torch.randn((1, length, heads, 128), generator=generator, device=device).to(torch.bfloat16)
    out, lse, _, _, val, idx = prefill_attention_topk(query, key, value, softmax_scale=SCALE, num_sink=sinks)
    torch.cuda.synchronize()
    skip = sinks + 7
    group = heads // kv_heads
    rows = torch.randint(skip, length, (40,), generator=generator, device=device).tolist() + [skip, 127, 128, length - 1]
    k32 = key[0].float()
    exact_rows = 0
    for row in rows:
        q_row = query[0, row].float()  # [heads, 128]
        raw = torch.einsum("hd,jhd->hj", q_row, k32[: row + 1].repeat_interleave(group, dim=1))  # [heads, keys]
        keys = torch.clamp(torch.round((raw + 48.0) * 256.0), 0, 32767).long()
        columns = torch.arange(row + 1, device=device)
        packed = (keys << 17) | columns
        packed[:, :sinks] = -1
        kept = []
        for cls in range(4):
            members = packed[:, ((columns % 8) // 2) == cls]
            kept.append(members.topk(min(6, members.shape[1]), dim=1).values)
        want = torch.cat(kept, dim=1).topk(8, dim=1).values  # [heads, 8], descending
        want_idx = want & 0x1FFFF
        got_idx = idx[0, :, row - skip].long()
        got_val = val[0, :, row - skip]
        assert bool((got_idx >= sinks).all()) and bool((got_idx <= row).all()), row
        for head in range(heads):
            mine, theirs = set(got_idx[head].tolist()), set(want_idx[head].tolist())
            assert len(mine) == 8, (row, head)
            if got_idx[head].tolist() == want_idx[head].tolist():
                exact_rows += 1
            floor_key = int(want[head, -1] >> 17)
            for j in mine ^ theirs:
                assert abs(int(keys[head, j]) - floor_key) <= 1, (row, head, j)
        # probabilities from the dequantised key of the column the kernel chose
        chosen = keys.gather(1, got_idx).float() / 256.0 - 48.0
        want_val = torch.exp(chosen * SCALE - lse[0, :, row].unsqueeze(1))
        torch.testing.assert_close(got_val, want_val, rtol=3e-2, atol=1e-9)
    assert exact_rows / (len(rows) * heads) > 0.9, exact_rows / (len(rows) * heads)


@pytest.mark.parametrize("length,heads,kv_heads,sinks", [(517, 4, 1, 10), (385, 2, 1, 0), (300, 4, 2, 70), (401, 8, 2, 150)])
def test_reference_topk_rule_with_ties(length, heads, kv_heads, sinks):
    """Whole-number scores: every product and sum is exact, so the neighbours are the oracle's without any
    allowance.  Most keys tie, so the gates in front of the insertion and the order among equal keys decide
    every row; the sinks end inside the first key block, in its upper half and in the second block."""

    generator = torch.Generator().manual_seed(length)
    q = torch.randint(-1, 2, (1, length, heads, 128), generator=generator).to(torch.bfloat16)
    k = torch.randint(-1, 2, (1, length, kv_heads, 128), generator=generator).to(torch.bfloat16)
    v = torch.randint(-1, 2, (1, length, kv_heads, 128), generator=generator).to(torch.bfloat16)
    *_, idx = prefill_attention_topk(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks)
    _, want_lse, raw = oracle.causal_attention(q[0].float().numpy(), k[0].float().numpy(), v[0].float().numpy(), SCALE)
    for head in range(heads):
        want_idx = oracle.reference_topk(raw[head], want_lse[head], SCALE, sinks)[1]
        assert np.array_equal(idx[0, head].cpu().numpy(), want_idx), head


@pytest.mark.parametrize("kind", ["nan", "inf"])
@pytest.mark.parametrize("heads,kv_heads", [(4, 1), (2, 2)])
def test_reference_topk_rule_with_odd_scores(kind, heads, kv_heads):
    """Whole-number scores with a few keys that make a row's scores infinite or not a number: a NaN or
    -inf is never a neighbour (every row has eight others), a +inf is one and saturates the candidate key."""

    length, sinks = 333, 10
    generator = torch.Generator().manual_seed(length)
    q = torch.randint(0, 2, (1, length, heads, 128), generator=generator).mul(2).sub(1).to(torch.bfloat16)
    k = torch.randint(-1, 2, (1, length, kv_heads, 128), generator=generator).to(torch.bfloat16)
    v = torch.randn((1, length, kv_heads, 128), generator=generator).to(torch.bfloat16)
    if kind == "nan":
        k[0, 45] = float("nan")
        k[0, 200, :, 3] = float("nan")
    else:
        k[0, 77, :, 0] = float("inf")
        k[0, 130, :, 0] = float("inf")
        k[0, 300, :, 5] = float("-inf")
    *_, idx = prefill_attention_topk(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=sinks)
    group = heads // kv_heads
    for head in range(heads):
        raw = q[0, :, head].double().numpy() @ k[0, :, head // group].double().numpy().T
        raw = np.where(np.isnan(raw), -1000.0, raw).astype(np.float32)  # quantises to the least key, as -inf does
        want_idx = oracle.reference_topk(raw, np.zeros(length, np.float32), SCALE, sinks)[1]
        assert np.array_equal(idx[0, head].cpu().numpy(), want_idx), head


@pytest.mark.parametrize("room,shift", [(0, 0), (24, 0), (24, 4)])
def test_plugin_prefill_reads_the_cache_where_it_lies(room, shift):
    """``[B, H, S, D]`` tensors with unused rows, and off the 16-byte boundary that the tile copies need."""

    from types import SimpleNamespace

    from community_kv_b200 import CommunityKVAttention, CommunityKVConfig, CommunityKVRuntime, PartitionConfig

    length, heads, kv_heads = 200, 4, 2
    q, k, v = _inputs(8, length, heads, kv_heads)
    want = prefill_attention_topk(q.cuda(), k.cuda(), v.cuda(), softmax_scale=SCALE, num_sink=10)

    def placed(tensor, rows):
        whole = torch.zeros((tensor.shape[2] * rows * 128 + shift,), dtype=torch.bfloat16, device="cuda")
        view = whole[shift:].view(1, tensor.shape[2], rows, 128)
        view[:, :, :length] = tensor.cuda().transpose(1, 2)
        return view

    edges = {}
    runtime = CommunityKVRuntime(config=CommunityKVConfig(num_sink=10), partition=PartitionConfig(), num_layers=1,
                                 max_decode_tokens=8, partitioner=lambda **found: edges.update(found))
    runtime.start_request()
    out, _ = CommunityKVAttention(runtime).forward(
        SimpleNamespace(layer_idx=0), placed(q, length), placed(k, length + room), placed(v, length + room), None, SCALE)
    assert torch.equal(out, want[0])
    assert torch.equal(edges["topk_indices"], want[5][0]) and torch.equal(edges["topk_scores"], want[4][0])


@pytest.mark.parametrize("kv_heads,batch,length", [(149, 1, 120), (33, 9, 120), (74, 1, 200), (75, 1, 200), (25, 6, 300)])
def test_prefill_items_over_the_ctas(kv_heads, batch, length):
    """One or several tiles per CTA of the head-pair kernel (148 of them), tiles of one key block next to longer ones:
    the bits do not depend on which tiles a CTA works through."""

    generator = torch.Generator(device="cuda").manual_seed(length + kv_heads)

    def rows(heads):
        return torch.randn((batch, length, heads, 128), generator=generator, device="cuda").to(torch.bfloat16)

    q, k, v = rows(2 * kv_heads), rows(kv_heads), rows(kv_heads)
    k = k * 0.3
    out, lse, _, _, val, idx = prefill_attention_topk(q, k, v, softmax_scale=SCALE, num_sink=3)
    plain, plain_lse = prefill_attention(q, k, v, softmax_scale=SCALE)
    for b in {0, batch // 2, batch - 1}:
        for h in {0, 1, kv_heads // 2, kv_heads - 1}:
            alone = prefill_attention_topk(q[b : b + 1, :, 2 * h : 2 * h + 2].contiguous(), k[b : b + 1, :, h : h + 1].contiguous(),
                                           v[b : b + 1, :, h : h + 1].contiguous(), softmax_scale=SCALE, num_sink=3)
            pair = slice(2 * h, 2 * h + 2)
            assert torch.equal(out[b, :, pair], alone[0][0]) and torch.equal(lse[b, pair], alone[1][0])
            assert torch.equal(val[b, pair], alone[4][0]) and torch.equal(idx[b, pair], alone[5][0])
            want = torch.nn.functional.scaled_dot_product_attention(
                q[b, :, pair].float().transpose(0, 1), k[b, :, h].float().expand(2, -1, -1),
                v[b, :, h].float().expand(2, -1, -1), is_causal=True, scale=SCALE).transpose(0, 1)
            assert float((out[b, :, pair].float() - want).abs().max()) <= 2e-2
    # the plain kernel works through the same tiles; its sums are those of the other
    assert torch.equal(plain, out) and torch.equal(plain_lse, lse)


def test_prefill_beside_a_kernel_that_holds_some_sms():
    """Tiles go to whichever SM is free: sixteen SMs held by another stream's long kernel do not keep a share of the
    prompt waiting (shares dealt out before the launch took 1.8 times as long as alone)."""

    generator = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn((1, 16384, heads, 128), generator=generator, device="cuda").to(torch.bfloat16)
               for heads in (32, 8, 8))
    rows = torch.randn((16, 1 << 20), generator=generator, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    main, other = torch.cuda.Stream(), torch.cuda.Stream()

    def milliseconds(beside):
        spans = []
        for _ in range(5):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            if beside:
                with torch.cuda.stream(other):
                    torch.cumsum(rows, 1)  # a CTA per row or so, 1.7 ms
            with torch.cuda.stream(main):
                begin.record()
                out, lse = prefill_attention(q, k, v, softmax_scale=SCALE, status=status)
                end.record()
            torch.cuda.synchronize()
            spans.append(begin.elapsed_time(end))
        return min(spans), out, lse

    torch.cumsum(rows, 1)
    alone, want, want_lse = milliseconds(False)
    beside, out, lse = milliseconds(True)
    assert int(status) == 0
    assert torch.equal(out, want) and torch.equal(lse, want_lse)
    assert beside < 1.4 * alone
