"""The level-sweep kernels, which graphs without closure lists, explicit row
kernels and level groupings run: every test asserts that they did. Scores are
the oracle's, paths score the oracle's optimum."""
import numpy as np
import pytest

import chsga_b200 as cb
import oracle as orc
from conftest import gen_graph
from test_gpu_wide_weights import _graph

pytestmark = pytest.mark.gpu

SWEEPS = 8000  # an explicit level grouping selects the sweeps
AUTO_KERNEL = {1: "k_row_t1", 2: "k_row_dpx", 8: "k_row_dpx", 16: "k_row_dpx", 32: "k_row_dpx",
               64: "k_row_stream", 128: "k_row_delta"}


def test_packed_sweeps_with_weights_above_65535(tmp_path):
    """Saturating sums of weights above 65535 and scores up to 64,000 in the
    packed upward and downward kernels (see test_gpu_wide_weights.py)."""
    g, files = _graph(tmp_path, "chain", 2000, lambda i, rng: int(rng.integers(400, 512)))
    reads = g.gen_reads(6, 7, 300, 600, sub_rate=0.02, indel_rate=0.02).to_list()
    want = orc.Oracle(files).scores(reads)
    ctx = cb.Context(0).load(g)
    # a read of N scores its length; clamped weights saturate at any score
    for slots, n in ((8, 64_000), (128, 3000)):
        # a grouping below the vertex count, so that levels run as grid launches
        got = ctx.align_scores_batched(reads + [b"N" * n], slots=slots, top_vertices=1000)
        assert ctx.last_row_kernel() == AUTO_KERNEL[slots] and ctx.profile()["row_bits"] == 16
        np.testing.assert_array_equal(got, list(want) + [n], err_msg=f"{slots} slots")
    ctx.close()


def test_long_vertices_with_weights_above_65535(tmp_path):
    g, files = _graph(tmp_path, "long", 120,
                      lambda i, rng: 66_000 if i in (30, 60, 90) else int(rng.integers(5, 30)))
    reads = g.gen_reads(6, 7, 100, 200, sub_rate=0.02, indel_rate=0.02).to_list()
    want = orc.Oracle(files).scores(reads)
    ctx = cb.Context(0).load(g)
    for slots in (8, 128):
        got = ctx.align_scores_batched(reads, slots=slots, top_vertices=60)
        assert ctx.last_row_kernel() == "k_row_direct"
        np.testing.assert_array_equal(got, want, err_msg=f"{slots} slots")
    ctx.close()


@pytest.mark.parametrize("coop", ["0", "1"])
@pytest.mark.parametrize("top_vertices", [300, SWEEPS])
def test_pull_forms_match_oracle(tmp_path, monkeypatch, top_vertices, coop):
    """Upward levels below the top region, with and without cooperative edge
    loads, on a graph larger than either grouping."""
    g, files = gen_graph(tmp_path, "g", backbone_len=120_000, seed=4)
    assert g.stats()["num_strings"] > SWEEPS
    reads = g.gen_reads(150, 23, 1, 300, sub_rate=0.03, indel_rate=0.02).to_list()
    want = orc.Oracle(files).scores(reads)
    monkeypatch.setenv("CHSGA_PULL_COOP", coop)
    ctx = cb.Context(0).load(g)
    for slots in (64, 128):
        got = ctx.align_scores_batched(reads, slots=slots, top_vertices=top_vertices)
        assert ctx.last_row_kernel() == AUTO_KERNEL[slots]
        np.testing.assert_array_equal(got, want)
    ctx.close()


@pytest.mark.parametrize("top_vertices", [300, SWEEPS])
def test_delta_rows_equal_16bit_rows(small_graph, oracle_small, top_vertices):
    g, _, reads = small_graph
    mix = list(reads) + g.gen_reads(150, 29, 1, 600, sub_rate=0.04, indel_rate=0.03, n_rate=0.01).to_list()
    want = oracle_small.scores(mix)
    ctx = cb.Context(0).load(g)
    for rk, kernel in ((cb.ROW_DELTA, "k_row_delta"), (cb.ROW_STREAM, "k_row_stream"), (cb.ROW_DPX, "k_row_dpx")):
        got = ctx.align_scores_batched(mix, slots=128, top_vertices=top_vertices, row_kernel=rk)
        assert ctx.last_row_kernel() == kernel
        np.testing.assert_array_equal(got, want)
    ctx.close()


@pytest.mark.parametrize("match_n", [False, True])
def test_graph_without_lists(tmp_path, match_n):
    """A graph of one-char vertices gets no closure lists: every call runs the
    sweeps by itself."""
    g, files = gen_graph(tmp_path, "g", backbone_len=6000, seed=6, vlen_min=1, vlen_max=1, bubble_gap_mean=50.0)
    reads = g.gen_reads(140, 8, 1, 120, sub_rate=0.03, indel_rate=0.03, n_rate=0.01).to_list()
    want = orc.Oracle(files, match_n=match_n).scores(reads)
    ctx = cb.Context(0, flags=cb.FLAG_MATCH_N if match_n else 0).load(g)
    np.testing.assert_array_equal(ctx.align_scores(reads[:9]), want[:9])
    assert ctx.last_row_kernel() == "k_row_t1"
    for slots, kernel in AUTO_KERNEL.items():
        np.testing.assert_array_equal(ctx.align_scores_batched(reads, slots=slots), want, err_msg=f"{slots} slots")
        assert ctx.last_row_kernel() == kernel
    np.testing.assert_array_equal(ctx.align_scores_batched(reads, slots=8, row_bits=32), want)
    assert ctx.last_row_kernel() == "k_row_direct"
    np.testing.assert_array_equal(ctx.align_scores_noalloc(reads), want)
    assert ctx.last_row_kernel() == "k_row_direct"
    srv = cb.Server(ctx, slots=32, queue_capacity=64)
    tk = [srv.submit(r) for r in reads]
    res = srv.collect()
    srv.close()
    assert [res[t]["score"] for t in tk] == list(want)
    ctx.close()


def test_forced_row_kernel_everywhere(small_graph, oracle_small, monkeypatch):
    """CHSGA_ROW_KERNEL runs the sweeps in the allocation-free call, the serving
    lane and the batched traceback too."""
    g, files, reads = small_graph
    want = oracle_small.scores(reads)
    labels = open(files[3], "rb").read().replace(b"\n", b"")
    plain = cb.Context(0).load(g)
    for name in ("direct", "stream"):
        monkeypatch.setenv("CHSGA_ROW_KERNEL", name)
        ctx = cb.Context(0).load(g)
        monkeypatch.delenv("CHSGA_ROW_KERNEL")
        np.testing.assert_array_equal(ctx.align_scores_noalloc(reads), want)
        assert ctx.last_row_kernel() == "k_row_direct"
        srv = cb.Server(ctx, slots=64, queue_capacity=64)
        tk = [srv.submit(r) for r in reads]
        res = srv.collect()
        srv.close()
        assert [res[t]["score"] for t in tk] == list(want)
        for slots in (4, 64):
            got = ctx.align_traceback_batched(reads, slots=slots)
            paths = plain.align_traceback_batched(reads, slots=slots)
            for (ops, score, _), (other, _, _), rd, w in zip(got, paths, reads, want):
                assert score == w and orc.rescore(ops, rd, labels) == (w, len(rd) - 1)
                np.testing.assert_array_equal(ops, other)
        ctx.close()
    plain.close()
