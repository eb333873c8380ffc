"""Decode-state assembly kernels (``ckv_assemble_*``) against the host restatement of the reference's
builders (community_kv/graph/partition.py:382-535), which ``tests/test_host_logic.py`` pins on fixtures
generated from the reference itself."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from community_kv_b200.assembly import (
    aggregation_mappings,
    assemble_layer,
    build_member_csr,
    compute_centroids,
    init_modularity_state,
)
from community_kv_b200.synthetic import zipf_sizes

pytestmark = pytest.mark.gpu


def _labels(graphs, length, communities, seed, zipf=None):
    generator = torch.Generator().manual_seed(seed)
    rows = []
    for _ in range(graphs):
        if zipf is None:
            ids = torch.randint(0, communities, (length,), generator=generator)
            ids[:communities] = torch.randperm(communities, generator=generator)
        else:
            sizes = zipf_sizes(length, communities, zipf, generator)
            ids = torch.repeat_interleave(torch.arange(communities), sizes)[torch.randperm(length, generator=generator)]
        rows.append(ids)
    return torch.stack(rows).to(torch.int32)


@pytest.mark.parametrize(
    "graphs,kv_heads,query_heads,aggregation,length,communities,zipf",
    [
        (2, 2, 8, "query_group", 3000, 37, None),
        (8, 2, 8, "per_query_head", 1000, 11, None),
        (1, 4, 16, "layer_wise", 5000, 130, 1.1),
        (8, 8, 32, "query_group", 32768, 512, 1.1),      # one layer of the whole-model configuration
        (2, 2, 8, "query_group", 131072, 4096, 1.1),     # long-context sizes
    ],
)
def test_member_lists_and_centroids_match_the_host_builders(graphs, kv_heads, query_heads, aggregation, length,
                                                            communities, zipf):
    device = torch.device("cuda", 0)
    sinks, decode = 10, 7
    labels = _labels(graphs, length, communities, seed=length + graphs, zipf=zipf)
    generator = torch.Generator().manual_seed(5)
    keys = (torch.randn((kv_heads, length, 128), generator=generator) / 128**0.5).to(torch.bfloat16)
    counts = (labels.amax(dim=1) + 1).to(torch.int32)
    to_graph, to_kv = aggregation_mappings(aggregation, query_heads=query_heads, kv_heads=kv_heads)

    want_offsets, want_positions = build_member_csr(labels, counts, num_sink=sinks)
    want_centroids, want_sizes = compute_centroids(labels, counts, keys, retrieval_to_graph=to_graph,
                                                   retrieval_to_kv=to_kv, num_sink=sinks, max_decode_tokens=decode)
    got_offsets, got_positions = build_member_csr(labels.to(device), counts.to(device), num_sink=sinks)
    got_centroids, got_sizes = compute_centroids(labels.to(device), counts.to(device), keys.to(device),
                                                 retrieval_to_graph=to_graph.to(device),
                                                 retrieval_to_kv=to_kv.to(device), num_sink=sinks,
                                                 max_decode_tokens=decode)
    assert torch.equal(got_offsets.cpu(), want_offsets)
    assert torch.equal(got_positions.cpu(), want_positions)
    assert torch.equal(got_sizes.cpu(), want_sizes)
    assert got_centroids.shape == want_centroids.shape
    assert torch.equal(got_centroids.cpu().view(torch.uint8), want_centroids.view(torch.uint8))


def test_assembly_fixture_from_the_reference(golden_dir):
    """The reference-generated fixture (labels -> offsets, member positions, sizes, e4m3 centroids)."""

    device = torch.device("cuda", 0)
    data = np.load(golden_dir / "assembly.npz")
    sinks, decode = int(data["meta"][3]), int(data["meta"][4])
    keys = torch.from_numpy(data["keys"])
    keys_are_bf16 = torch.equal(keys, keys.to(torch.bfloat16).float())  # the kernel takes bf16 keys
    for case in range(3):
        labels = torch.from_numpy(data[f"labels_{case}"])
        to_graph = torch.from_numpy(data[f"to_graph_{case}"])
        to_kv = torch.from_numpy(data[f"to_kv_{case}"])
        counts = (labels.amax(dim=1) + 1).to(torch.int32)
        offsets, positions = build_member_csr(labels.to(device), counts.to(device), num_sink=sinks)
        centroids, sizes = compute_centroids(labels.to(device), counts.to(device), keys.to(torch.bfloat16).to(device),
                                             retrieval_to_graph=to_graph.to(device), retrieval_to_kv=to_kv.to(device),
                                             num_sink=sinks, max_decode_tokens=decode)
        assert torch.equal(offsets.cpu(), torch.from_numpy(data[f"offsets_{case}"])), case
        assert torch.equal(positions.cpu(), torch.from_numpy(data[f"positions_{case}"])), case
        assert torch.equal(sizes.cpu(), torch.from_numpy(data[f"sizes_{case}"])), case
        if keys_are_bf16:
            assert torch.equal(centroids.cpu().view(torch.uint8), torch.from_numpy(data[f"centroids_{case}"])), case


def test_modularity_state_from_an_edge_list():
    device = torch.device("cuda", 0)
    graphs, length, communities = 3, 4000, 50
    labels = _labels(graphs, length, communities, seed=9)
    generator = torch.Generator().manual_seed(10)
    edges = 60000
    graph = torch.randint(0, graphs, (edges,), generator=generator)
    source = graph * length + torch.randint(0, length, (edges,), generator=generator)
    destination = graph * length + torch.randint(0, length, (edges,), generator=generator)
    weight = torch.rand((edges,), generator=generator)
    want_weight, want_total = init_modularity_state(labels, source, destination, weight, community_capacity=64)
    got_weight, got_total = init_modularity_state(labels.to(device), source.to(device), destination.to(device),
                                                  weight.to(device), community_capacity=64)
    torch.testing.assert_close(got_weight.cpu(), want_weight, rtol=2e-5, atol=1e-6)
    torch.testing.assert_close(got_total.cpu(), want_total, rtol=2e-5, atol=1e-6)
    empty = torch.empty((0,), dtype=torch.int64, device=device)
    zero_weight, zero_total = init_modularity_state(labels.to(device), empty, empty, empty.float(),
                                                    community_capacity=64)
    assert float(zero_weight.abs().sum()) == 0.0 and float(zero_total.abs().sum()) == 0.0


def test_assembled_layer_on_the_device_equals_the_host_one():
    device = torch.device("cuda", 0)
    labels = _labels(2, 6000, 90, seed=3, zipf=1.1)
    keys = (torch.randn((2, 6000, 128), generator=torch.Generator().manual_seed(4)) / 128**0.5).to(torch.bfloat16)
    host = assemble_layer(labels, keys, aggregation="query_group", query_heads=8, num_sink=10, max_decode_tokens=5)
    dev = assemble_layer(labels.to(device), keys.to(device), aggregation="query_group", query_heads=8, num_sink=10,
                         max_decode_tokens=5)
    for name in host.__slots__:
        a, b = getattr(host, name), getattr(dev, name).cpu()
        if a.dtype == torch.float8_e4m3fn:
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)), name
        elif a.dtype == torch.float32:
            torch.testing.assert_close(b, a, rtol=1e-6, atol=0, msg=name)
        else:
            assert torch.equal(a, b), name


# ---- edge list -> adjacency -----------------------------------------------------------------------
def _adjacency_equal(got, want, where):
    source, destination, weight = (t.cpu().numpy() for t in got)
    assert np.array_equal(source, want[0]), where
    assert np.array_equal(destination, want[1]), where
    assert np.array_equal(weight.view(np.int32), want[2].view(np.int32)), where  # fp32 sums bit for bit


def test_adjacency_fixture_from_the_reference(golden_dir):
    from community_kv_b200.assembly import build_adjacency

    device = torch.device("cuda", 0)
    data = np.load(golden_dir / "adjacency.npz")
    for case in data["cases"].tolist():
        length, lam = int(data[f"scalars_{case}"][0]), float(data[f"scalars_{case}"][1])
        got = build_adjacency(torch.from_numpy(data[f"indices_{case}"]).to(device),
                              torch.from_numpy(data[f"scores_{case}"]).to(device),
                              torch.from_numpy(data[f"positions_{case}"]).to(device), seq_len=length, lam=lam)
        _adjacency_equal(got, (data[f"source_{case}"], data[f"destination_{case}"], data[f"weight_{case}"]),
                         f"case {case}")


@pytest.mark.parametrize("graphs,rows,length,lam", [(8, 4 * 4000, 4096, 0.5), (2, 30000, 32768, 0.5),
                                                    (1, 50000, 131072, 1.0)])
def test_adjacency_against_the_cpu_restatement(graphs, rows, length, lam):
    """Sizes of a real prefill (causal neighbours, hub keys, several heads sharing a graph): every
    distinct edge, in order, with its weight summed in the reference's order."""

    from community_kv_b200.assembly import build_adjacency
    from oracle.adjacency_oracle import build_adjacency as oracle_adjacency

    device = torch.device("cuda", 0)
    rng = np.random.default_rng(rows)
    positions = rng.integers(20, length, size=(graphs, rows)).astype(np.int64)
    # neighbours are earlier positions, a few of them shared hubs; some slots are empty
    indices = (positions[..., None] * rng.uniform(0, 1, size=(graphs, rows, 8))).astype(np.int32)
    hubs = rng.integers(0, 64, size=(graphs, rows, 8)).astype(np.int32)
    indices = np.where(rng.uniform(size=indices.shape) < 0.2, hubs, indices)
    indices = np.where(rng.uniform(size=indices.shape) < 0.05, -1, indices).astype(np.int32)
    scores = rng.uniform(0, 1, size=indices.shape).astype(np.float32)
    want = oracle_adjacency(indices, scores, positions, seq_len=length, lam=lam)
    got = build_adjacency(torch.from_numpy(indices).to(device), torch.from_numpy(scores).to(device),
                          torch.from_numpy(positions).to(device), seq_len=length, lam=lam)
    _adjacency_equal(got, want, f"{graphs}x{rows}")


@pytest.mark.parametrize(
    "graphs,rows,length,kappa,lam",
    [
        (1, 1, 9, 8, 0.5),            # fewer edges than a tile's first warp has lanes for
        (3, 31, 4096, 8, 0.5),        # 4092 edges, a few short of a tile; 4-byte keys
        (2, 47, 65536, 8, 0.5),       # two positions fill 4 bytes: 8-byte keys, two tiles and a bit
        (1, 187, 256, 8, 0.25),       # 8228 edges, a few beyond two tiles
        (1, 600, 5000, 8, 1.0),       # direct edges only
        (5, 260, 3000, 3, 0.5),       # another row width, several graphs in a tile
        (2, 900, 40, 8, 0.5),         # long runs of one edge, across tiles
    ],
)
def test_adjacency_at_the_edges_of_tiles_and_keys(graphs, rows, length, kappa, lam):
    from community_kv_b200.assembly import build_adjacency
    from oracle.adjacency_oracle import build_adjacency as oracle_adjacency

    device = torch.device("cuda", 0)
    rng = np.random.default_rng(rows + length)
    positions = rng.integers(0, length, size=(graphs, rows)).astype(np.int64)
    indices = rng.integers(-1, length, size=(graphs, rows, kappa)).astype(np.int32)
    scores = rng.uniform(0, 1, size=indices.shape).astype(np.float32)
    want = oracle_adjacency(indices, scores, positions, seq_len=length, lam=lam)
    got = build_adjacency(torch.from_numpy(indices).to(device), torch.from_numpy(scores).to(device),
                          torch.from_numpy(positions).to(device), seq_len=length, lam=lam)
    _adjacency_equal(got, want, f"{graphs}x{rows}x{kappa}")


def test_adjacency_leaves_out_direct_edges_of_rows_outside_the_graph():
    """A row's own position beyond its graph, or negative: no direct edge; its neighbours' edges stay."""

    from community_kv_b200.assembly import build_adjacency
    from oracle.adjacency_oracle import build_adjacency as oracle_adjacency

    length, kappa = 100, 8
    rng = np.random.default_rng(3)
    indices = rng.integers(0, length, size=(2, 40, kappa)).astype(np.int32)
    scores = rng.uniform(0.01, 1, size=indices.shape).astype(np.float32)
    positions = rng.integers(0, length, size=(2, 40)).astype(np.int64)
    outside = rng.uniform(size=positions.shape) < 0.3
    moved = np.where(outside, rng.choice([-1, -length, length, length + 7, 2**40], size=positions.shape), positions)
    device = torch.device("cuda", 0)

    def run(lam):
        return build_adjacency(*(torch.from_numpy(a).to(device) for a in (indices, scores, moved)), seq_len=length, lam=lam)

    # direct edges alone: as if those rows had no neighbours
    want = oracle_adjacency(np.where(outside[..., None], -1, indices), scores, positions, seq_len=length, lam=1.0)
    _adjacency_equal(run(1.0), want, "direct")
    # lam = 0: direct edges weigh nothing, and every other edge is there
    got = [t.cpu().numpy() for t in run(0.0)]
    want = oracle_adjacency(indices, scores, positions, seq_len=length, lam=0.0)
    _adjacency_equal([torch.from_numpy(a[got[2] > 0]) for a in got], [a[want[2] > 0] for a in want], "co-attention")


def test_adjacency_reports_a_wait_that_ran_out():
    """Waits inside the sort that give up at their first look: the count says so, or the edges are right.
    More tiles than run at a time, so that some tile does find its predecessors unfinished."""

    from community_kv_b200 import native
    from community_kv_b200.assembly import build_adjacency

    graphs, rows, kappa, length, lam = 4, 12000, 8, 8192, 0.5
    generator = torch.Generator().manual_seed(5)
    indices = torch.randint(0, length, (graphs, rows, kappa), generator=generator, dtype=torch.int32).cuda()
    scores = torch.rand((graphs, rows, kappa), generator=generator).cuda()
    positions = torch.randint(0, length, (graphs, rows), generator=generator).cuda()
    want = build_adjacency(indices, scores, positions, seq_len=length, lam=lam)
    lib = native.library()
    raw = lib.ckv_adjacency_raw_edges(graphs, rows, kappa, lam)
    reported = 0
    for _ in range(20):
        scratch = torch.zeros((lib.ckv_adjacency_scratch_bytes(graphs, rows, kappa, lam),), dtype=torch.uint8,
                              device="cuda")
        source, destination = (torch.empty((raw,), dtype=torch.int32, device="cuda") for _ in range(2))
        weight = torch.empty((raw,), device="cuda")
        count = torch.empty((1,), dtype=torch.int64, device="cuda")
        assert lib.ckv_build_adjacency_polls(
            indices.data_ptr(), scores.data_ptr(), positions.data_ptr(), graphs, rows, kappa, length, lam,
            source.data_ptr(), destination.data_ptr(), weight.data_ptr(), raw, count.data_ptr(),
            scratch.data_ptr(), scratch.numel(), 0, native.current_stream(indices.device)) == 0
        edges = int(count)
        reported += edges == -1
        if edges != -1:
            for got, expected in zip((source, destination, weight), want):
                assert torch.equal(got[:edges], expected)
    assert reported > 0


@pytest.mark.parametrize("host", ["member_offsets", "member_positions", "community_counts"])
def test_member_lists_on_the_host_and_the_device(host):
    """``PrefillCSR.validate`` takes tensors that are not all on one device."""

    from community_kv_b200.state import PrefillCSR

    tensors = {"member_offsets": torch.tensor([[0, 2, 3], [0, 1, 9]], dtype=torch.int32),
               "member_positions": torch.zeros((2, 4), dtype=torch.int32),
               "community_counts": torch.tensor([2, 1], dtype=torch.int32)}
    placed = {name: tensor if name == host else tensor.cuda() for name, tensor in tensors.items()}
    PrefillCSR(**placed).validate()
    placed["community_counts"] = placed["community_counts"] + 1
    with pytest.raises(ValueError, match="count exceeds"):
        PrefillCSR(**placed).validate()


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_modularity_counts_destinations_in_the_sources_graph(dtype):
    """Destinations numbered in another graph, and negative ones: position modulo the length, as on the host."""

    graphs, length, communities = 3, 50, 7
    labels = _labels(graphs, length, communities, seed=12)
    source = torch.tensor([60, 61, 110, 120, 149, 99, 55])
    destination = torch.tensor([3, 149, -1, -50, -51, -99, 60])
    weight = torch.tensor([1.0, 2.0, 4.0, 8.0, 16.0, 32.0, 64.0])
    want = init_modularity_state(labels, source, destination, weight, community_capacity=8)
    got = init_modularity_state(labels.cuda(), source.to(dtype).cuda(), destination.to(dtype).cuda(), weight.cuda(),
                                community_capacity=8)
    assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1])


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("edges", [1, 15, 16, 4097, 9001])
def test_modularity_of_sorted_edges(edges, dtype):
    """Runs of one source, a graph's end inside a thread's run, a ragged tail, unaligned edge arrays."""

    device = torch.device("cuda", 0)
    graphs, length, communities = 3, 700, 20
    labels = _labels(graphs, length, communities, seed=11)
    generator = torch.Generator().manual_seed(edges)
    source = torch.randint(0, graphs * length, (edges + 1,), generator=generator).sort().values
    destination = source // length * length + torch.randint(0, length, (edges + 1,), generator=generator)
    # sixteenths: every sum below 2^20 is exact in fp32, in any order
    weight = torch.randint(1, 17, (edges + 1,), generator=generator) / 16
    for begin in (0, 1):
        part = [t[begin : begin + edges] for t in (source, destination, weight)]
        want_weight, want_total = init_modularity_state(labels, *part, community_capacity=24)
        moved = [t.to(device)[begin : begin + edges] for t in (source.to(dtype), destination.to(dtype), weight)]
        got_weight, got_total = init_modularity_state(labels.to(device), *moved, community_capacity=24)
        assert torch.equal(got_weight.cpu(), want_weight) and torch.equal(got_total.cpu(), want_total)
