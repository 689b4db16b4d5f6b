"""Bit-row kernels against the oracle where they can go wrong: labels at the
word boundaries (32, 33, 34, 64, 65, 66 chars), labels above the sliced
kernel's limit, graphs smaller than and just past a block's window of
vertices, uneven reads (one base up) that end and refill slots together,
both score widths and both scoring schemes. Scores are whole numbers."""
import numpy as np
import pytest

import chsga_b200 as cb
import oracle as orc
from conftest import gen_graph, sprinkle_n

pytestmark = pytest.mark.gpu

GRAPHS = {
    "words_32_34": dict(backbone_len=4000, seed=3, vlen_min=32, vlen_max=34),
    "words_64_66": dict(backbone_len=6000, seed=4, vlen_min=64, vlen_max=66),
    "short_labels": dict(backbone_len=3000, seed=5, vlen_min=1, vlen_max=4, bubble_gap_mean=20.0),
    "one_window": dict(backbone_len=500, seed=6),
    "past_window": dict(backbone_len=3100, seed=7),
    "long_labels": dict(backbone_len=9000, seed=8, vlen_min=600, vlen_max=900, bubble_gap_mean=2000.0),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("match_n", [False, True])
def test_bit_rows_match_oracle(tmp_path, name, match_n):
    g, files = gen_graph(tmp_path, name, **GRAPHS[name])
    if match_n:
        g = sprinkle_n(files, 0.01, 2)
    reads = g.gen_reads(70, 9, 1, 130, sub_rate=0.02, indel_rate=0.03, n_rate=0.01).to_list()
    reads += [b"A", b"N", b"ACGT" * 30, b"T" * 61]
    want = orc.Oracle(files, match_n=match_n).scores(reads)
    with_n = cb.Context(0, flags=cb.FLAG_MATCH_N if match_n else 0).load(g)
    np.testing.assert_array_equal(with_n.align_scores(reads), want)
    for slots in (1, 2, 4, 8, 16, 32, 64, 128):
        for row_bits in (0, 32):
            got = with_n.align_scores_batched(reads, slots=slots, row_bits=row_bits)
            np.testing.assert_array_equal(got, want, err_msg=f"{slots} slots, {row_bits} bits")
    with_n.close()


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_bit_row_tracebacks_equal_level_sweeps(tmp_path, monkeypatch, name):
    """Paths from bit rows (full matrix, checkpoints, two-level segments,
    batched) are the level-sweep engine's, op for op, and score the optimum."""
    g, files = gen_graph(tmp_path, name, **GRAPHS[name])
    reads = g.gen_reads(5, 19, 60, 140, sub_rate=0.03, indel_rate=0.05).to_list() + [b"A", b"T" * 45]
    n = g.view().num_chars
    want = orc.Oracle(files).scores(reads)
    labels = open(files[3], "rb").read().replace(b"\n", b"")
    monkeypatch.setenv("CHSGA_ROW_KERNEL", "direct")
    sweeps = cb.Context(0).load(g)
    monkeypatch.delenv("CHSGA_ROW_KERNEL")
    bits = cb.Context(0).load(g)
    tight = cb.Context(0, hbm_cap_bytes=16 * 4 * n).load(g)
    for rd, w in zip(reads, want):
        ops, score, ck = sweeps.align_traceback(rd)
        assert score == w and not ck
        for ctx, k, cap in ((bits, 500, 0), (bits, 13, 4 * n), (tight, 100, 0)):
            got, gs, _ = ctx.align_traceback(rd, k=k, cap_bytes=cap)
            assert gs == w
            if len(rd) > 1:
                assert orc.rescore(got, rd, labels) == (w, len(rd) - 1)
            np.testing.assert_array_equal(got, ops)
    for slots in (4, 64):
        for (got, gs, _), rd, w in zip(bits.align_traceback_batched(reads, slots=slots), reads, want):
            assert gs == w
            np.testing.assert_array_equal(got, sweeps.align_traceback(rd)[0])
    for c in (sweeps, bits, tight):
        c.close()
