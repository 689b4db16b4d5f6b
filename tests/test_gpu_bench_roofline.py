"""bench.py's profiled pass names the row kernel that ran, whatever the graph
and the options select."""
import pytest

import bench
import chsga_b200 as cb
from conftest import gen_graph

pytestmark = pytest.mark.gpu

OPTS = dict(slots=128, steps_per_graph=8, use_graphs=1, row_kernel=cb.ROW_AUTO, top_vertices=0)


def _kernel(g, slots=128, row_bits=0, **opts):
    st = g.stats()
    out = bench.profiled_roofline(cb, g, st, st["num_strings"] - st["single_char_strings"], 0, slots,
                                  dict(OPTS, **opts), 6454.0, "measured", row_bits)
    return out["kernel"]


def test_long_labels_at_many_slots(tmp_path):
    # over 400,000 (vertex, slot) pairs, but labels of more than 512 chars
    g, _ = gen_graph(tmp_path, "g", backbone_len=2_500_000, seed=2, vlen_min=600, vlen_max=900,
                     bubble_gap_mean=2000.0)
    assert g.stats()["num_strings"] * 128 > 400_000
    assert _kernel(g) == "k_row_words<128>"


def test_other_choices(tmp_path):
    g, _ = gen_graph(tmp_path, "g", backbone_len=60_000, seed=2)
    assert _kernel(g) == "k_row_sliced<128>"
    assert _kernel(g, slots=8) == "k_row_words<8>"
    assert _kernel(g, row_bits=32) == "k_row_words<128>"
    assert _kernel(g, top_vertices=1000) == "k_row_delta<128>"
    assert _kernel(g, row_kernel=cb.ROW_STREAM) == "k_row_stream<128>"
