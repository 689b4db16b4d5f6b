"""Every form of the bit-row kernels at 32 to 128 slots, whichever the size of
the graph selects: the word kernel and k_row_sliced with one and with four
items a lane, forced with CHSGA_BIT_ROWS on graphs with labels at the word
boundaries, smaller than and just past a block's window of vertices, against
the oracle; and the forms the sizes select on a 1 Mbp graph, against the level
sweeps. Each test asserts which kernel ran. Uneven reads (one base up), more
than there are slots, end, drain and refill slots together."""
import os
import subprocess
import sys

import numpy as np
import pytest

import chsga_b200 as cb
import oracle as orc
from conftest import ROOT, gen_graph, sprinkle_n

pytestmark = pytest.mark.gpu

GRAPHS = {
    "words_32_34": dict(backbone_len=4000, seed=3, vlen_min=32, vlen_max=34),
    "words_64_66": dict(backbone_len=6000, seed=4, vlen_min=64, vlen_max=66),
    "longest_labels": dict(backbone_len=9000, seed=8, vlen_min=500, vlen_max=512, bubble_gap_mean=2000.0),
    "two_chars": dict(backbone_len=3000, seed=5, vlen_min=2, vlen_max=3),
    "one_window": dict(backbone_len=500, seed=6),
    "past_window": dict(backbone_len=3100, seed=7),
}
FORMS = {"words": "k_row_words", "sliced": "k_row_sliced<{},1>", "sliced4": "k_row_sliced<{},4>"}


def _uneven(g, count, seed):
    reads = g.gen_reads(count, seed, 1, 130, sub_rate=0.02, indel_rate=0.03, n_rate=0.01).to_list()
    return reads + [b"A", b"N", b"ACGT" * 30, b"T" * 61]


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("match_n", [False, True])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_forced_forms_match_oracle(tmp_path, monkeypatch, name, match_n, form):
    g, files = gen_graph(tmp_path, name, **GRAPHS[name])
    if match_n:
        g = sprinkle_n(files, 0.01, 2)
    reads = _uneven(g, 300, 9)
    want = orc.Oracle(files, match_n=match_n).scores(reads)
    monkeypatch.setenv("CHSGA_BIT_ROWS", form)
    ctx = cb.Context(0, flags=cb.FLAG_MATCH_N if match_n else 0).load(g)
    for slots in (32, 64, 128):
        for graphs in (0, 1):
            got = ctx.align_scores_batched(reads, slots=slots, use_graphs=graphs)
            assert ctx.last_row_kernel() == FORMS[form].format(slots)
            np.testing.assert_array_equal(got, want, err_msg=f"{slots} slots")
    srv = cb.Server(ctx, slots=64, queue_capacity=64)
    tk = [srv.submit(r) for r in reads]
    res = srv.collect()
    srv.close()
    assert [res[t]["score"] for t in tk] == list(want)
    ctx.close()


@pytest.mark.parametrize("form", ["sliced", "sliced4"])
def test_reads_past_15_bits(tmp_path, monkeypatch, form):
    """A read of more than 32767 bases (saturating sums, its drain step too)
    beside short ones that take the other sums once it has ended."""
    g, files = gen_graph(tmp_path, "g", **GRAPHS["one_window"])
    rng = np.random.default_rng(4)
    long_read = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 32900).astype(np.uint8))
    reads = [long_read] + _uneven(g, 40, 3)
    want = orc.Oracle(files).scores(reads)
    assert want[0] > 1 << 14
    monkeypatch.setenv("CHSGA_BIT_ROWS", form)
    ctx = cb.Context(0).load(g)
    np.testing.assert_array_equal(ctx.align_scores_batched(reads, slots=32), want)
    assert ctx.last_row_kernel() == FORMS[form].format(32)
    np.testing.assert_array_equal(ctx.align_scores_batched(reads[1:] + reads[:1], slots=32), want[1:].tolist() + [want[0]])
    ctx.close()


@pytest.mark.parametrize("match_n", [False, True])
def test_forms_chosen_by_size(tmp_path, match_n):
    """1 Mbp, 109,000 vertices: four items a lane at 32, 64 and 128 slots;
    100 kbp, 9,500: one at 64 and 128; 20 kbp: words. Scores are the level
    sweeps'."""
    for backbone, want_kernel in ((1_000_000, {32: "k_row_sliced<32,4>", 64: "k_row_sliced<64,4>",
                                               128: "k_row_sliced<128,4>"}),
                                  (100_000, {64: "k_row_sliced<64,1>", 128: "k_row_sliced<128,1>"}),
                                  (20_000, {32: "k_row_words", 64: "k_row_words", 128: "k_row_words"})):
        g, files = gen_graph(tmp_path, f"g{backbone}", backbone_len=backbone, seed=12)
        if match_n:
            g = sprinkle_n(files, 0.001, 2)
        reads = _uneven(g, 150, 5)
        ctx = cb.Context(0, flags=cb.FLAG_MATCH_N if match_n else 0).load(g)
        want = ctx.align_scores_batched(reads, slots=64, row_kernel=cb.ROW_DIRECT)
        assert ctx.last_row_kernel() == "k_row_direct"
        for slots, kernel in want_kernel.items():
            np.testing.assert_array_equal(ctx.align_scores_batched(reads, slots=slots), want)
            assert ctx.last_row_kernel() == kernel
        ctx.close()


CHECKED = os.path.join(ROOT, "chsga_b200", "lib_checked", "libchsga.so")
CHILD = r"""
import sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/oracle", sys.argv[1] + "/tests"]
import numpy as np
import chsga_b200 as cb, oracle as orc
from conftest import gen_graph
from test_gpu_bit_forms import FORMS, GRAPHS, _uneven
assert cb.LIB_PATH.endswith("lib_checked/libchsga.so")
form = sys.argv[3]
for name in sorted(GRAPHS):
    g, files = gen_graph(sys.argv[2], name, **GRAPHS[name])
    reads = _uneven(g, 150, 9)
    want = orc.Oracle(files).scores(reads)
    ctx = cb.Context(0).load(g)
    for slots in (32, 64, 128):
        np.testing.assert_array_equal(ctx.align_scores_batched(reads, slots=slots), want)
        assert ctx.last_row_kernel() == FORMS[form].format(slots)
    ctx.close()
print("checked ok")
"""


@pytest.mark.skipif(not os.path.exists(CHECKED), reason="checked build absent (make -C chsga_b200 checked)")
@pytest.mark.parametrize("form", sorted(FORMS))
def test_forced_forms_pass_the_index_checks(tmp_path, form):
    env = dict(os.environ, CHSGA_LIBRARY=CHECKED, CHSGA_BIT_ROWS=form)
    res = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(tmp_path), form], env=env, capture_output=True,
                         text=True, timeout=600)
    assert res.returncode == 0 and "checked ok" in res.stdout, res.stdout[-3000:] + res.stderr[-3000:]
