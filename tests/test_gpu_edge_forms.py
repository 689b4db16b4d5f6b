"""Edge-case reads and tiny graphs (conftest.edge_reads, conftest.TINY_GFA) on
every form the defaults do not pick for such small graphs: the level sweeps of
all slot counts and k_row_sliced with one and four items a lane; and the level
sweeps' checkpointed tracebacks, files included. Scores equal the oracle's."""
import os

import numpy as np
import pytest

import chsga_b200 as cb
import oracle as orc
from conftest import TINY_GFA, TINY_READS, edge_reads, gen_graph, tiny_graph
from test_gpu_sweep_kernels import AUTO_KERNEL, SWEEPS

pytestmark = pytest.mark.gpu

GRAPH = dict(backbone_len=600, seed=71, vlen_max=8, bubble_gap_mean=10.0, p_snp=0.5, p_indel=0.3, p_alt=0.2,
             alt_min=3, alt_max=30)


def _case(tmp_path, name):
    if name in TINY_GFA:
        g, files = tiny_graph(tmp_path, name)
        return g, files, TINY_READS
    g, files = gen_graph(tmp_path, name, **GRAPH)
    return g, files, edge_reads(g, 71)


@pytest.mark.parametrize("name", ["edge"] + sorted(TINY_GFA))
def test_scores(tmp_path, monkeypatch, name):
    g, files, reads = _case(tmp_path, name)
    want = orc.Oracle(files).scores(reads)
    ctx = cb.Context(0).load(g)
    for slots, kernel in AUTO_KERNEL.items():
        got = ctx.align_scores_batched(reads, slots=slots, top_vertices=SWEEPS - 1)
        assert ctx.last_row_kernel() == kernel
        np.testing.assert_array_equal(got, want, err_msg=f"{slots} slots")
    ctx.close()
    for form, items in (("sliced", 1), ("sliced4", 4)):
        monkeypatch.setenv("CHSGA_BIT_ROWS", form)
        ctx = cb.Context(0).load(g)
        for slots in (32, 64, 128):
            got = ctx.align_scores_batched(reads, slots=slots)
            if ctx.last_row_kernel().startswith("k_row_sliced"):
                assert ctx.last_row_kernel() == f"k_row_sliced<{slots},{items}>"
            else:  # a graph of one-char vertices may have no lists
                assert name != "edge" and ctx.last_row_kernel() == AUTO_KERNEL[slots]
            np.testing.assert_array_equal(got, want, err_msg=f"{form}, {slots} slots")
        ctx.close()


def test_sweep_checkpoints_are_the_bit_rows(tmp_path, monkeypatch):
    """Full, checkpointed and two-level tracebacks of the level sweeps give the
    bit rows' paths, and their checkpoint files the same bytes."""
    g, files, reads = _case(tmp_path, "edge")
    labels = open(files[3], "rb").read().replace(b"\n", b"")
    n = orc.Oracle(files).num_chars
    monkeypatch.setenv("CHSGA_ROW_KERNEL", "direct")
    sweeps, tight = cb.Context(0).load(g), cb.Context(0, hbm_cap_bytes=16 * 4 * n).load(g)
    monkeypatch.delenv("CHSGA_ROW_KERNEL")
    bits = cb.Context(0).load(g)
    for i, rd in enumerate(r for r in reads if len(r) >= 40):
        a, b = tmp_path / f"a{i}", tmp_path / f"b{i}"
        want, score, ck = bits.align_traceback(rd, k=11, ckpt_dir=str(b), keep_files=True, cap_bytes=15 * n * 4)
        assert ck and orc.rescore(want, rd, labels) == (score, len(rd) - 1)
        got, s, ck = sweeps.align_traceback(rd, k=11, ckpt_dir=str(a), keep_files=True, cap_bytes=15 * n * 4)
        assert ck and s == score and sweeps.last_row_kernel() == "k_row_direct"
        np.testing.assert_array_equal(got, want)
        names = sorted(os.listdir(b))
        assert names and names == sorted(os.listdir(a))
        for nm in names:
            assert (a / nm).read_bytes() == (b / nm).read_bytes(), (i, nm)
        for ctx, k in ((sweeps, 500), (tight, 100)):
            got, s, _ = ctx.align_traceback(rd, k=k)
            assert s == score
            np.testing.assert_array_equal(got, want)
    for c in (sweeps, tight, bits):
        c.close()
