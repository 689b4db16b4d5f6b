"""Which candidates the autotuner runs: every row kernel that AUTO does not
run already, and level groupings of kernels that sweep levels."""
import pytest

import chsga_b200 as cb
from conftest import gen_graph

pytestmark = pytest.mark.gpu

AT_SLOTS = {16: {cb.ROW_DPX, cb.ROW_DIRECT}, 32: {cb.ROW_DPX, cb.ROW_DIRECT, cb.ROW_TILED},
            64: {cb.ROW_STREAM, cb.ROW_DPX, cb.ROW_DIRECT, cb.ROW_TILED},
            128: {cb.ROW_DELTA, cb.ROW_STREAM, cb.ROW_DPX, cb.ROW_DIRECT, cb.ROW_TILED}}
SWEEPS_AUTO = {16: cb.ROW_DPX, 32: cb.ROW_DPX, 64: cb.ROW_STREAM, 128: cb.ROW_DELTA}


@pytest.mark.parametrize("lists", [True, False])
def test_candidates(tmp_path, lists):
    over = {} if lists else dict(vlen_min=1, vlen_max=1, bubble_gap_mean=50.0)
    g, _ = gen_graph(tmp_path, "g", backbone_len=8000, seed=3, **over)
    ctx = cb.Context(0).load(g)
    reads = g.gen_reads(140, 4, 30, 200, sub_rate=0.02).to_list()
    _, trials = ctx.autotune(reads, repeats=1)
    ctx.close()
    stage = [t for t in trials if t["row_kernel"] != cb.ROW_AUTO and t["top_vertices"] == 0]
    slots = stage[0]["slots"]
    want = AT_SLOTS[slots] - (set() if lists else {SWEEPS_AUTO[slots]})
    assert {t["row_kernel"] for t in stage} == want
    grouped = [t for t in trials if t["top_vertices"]]
    assert len(grouped) == 2
    if lists:  # AUTO has no levels to group
        fastest = max(stage, key=lambda t: t["measured_gcups"])
        assert {t["row_kernel"] for t in grouped} == {fastest["row_kernel"]}
