"""Device memory of tracebacks: what a request reports, and what a context
keeps between requests."""
import pytest

import chsga_b200 as cb
from conftest import gen_graph

pytestmark = pytest.mark.gpu


def test_peak_bytes_counts_the_whole_matrix(tmp_path):
    """peak_bytes of a full-matrix traceback depends on the request alone, not
    on the requests its worker ran before: rising, falling and repeated
    lengths, above 1 GiB too."""
    g, _ = gen_graph(tmp_path, "g", backbone_len=100_000, seed=2)
    strings = g.stats()["num_strings"]
    ctx = cb.Context(0).load(g)
    srv = cb.Server(ctx, tb_workers=1, slots=16)
    lens = [60, 60, 200, 200, 300, 300, 320, 320, 1500, 1500, 13000, 13000, 320, 200, 300, 60, 1500, 200, 13000]
    reads = {n: g.gen_reads(1, n, n).to_list()[0] for n in set(lens)}
    peak = []
    for n in lens:
        t = srv.submit(reads[n], cb.REQ_TRACEBACK)
        r = srv.collect()[t]
        assert r["status"] == cb.OK and not r["checkpointed"]
        peak.append(r["peak_bytes"])
    srv.close()
    ctx.close()
    repeated = {n: p for n, p, before in zip(lens[1:], peak[1:], lens) if n == before}
    for i, (n, p) in enumerate(zip(lens, peak)):
        # every row holds two 16-bit scores of every string vertex at least
        assert p >= 4 * strings * n, (i, n, p)
        # the context's own buffers grow with the longest read so far
        if i:
            assert abs(p - repeated[n]) <= 1 << 20, (i, n, p, repeated[n])


def _fill(leave):
    """Takes the device's free memory but `leave` bytes."""
    import torch
    held = []
    step = 1 << 36
    while step >= 1 << 25:
        while torch.cuda.mem_get_info(0)[0] >= leave + step:
            held.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        step >>= 1
    return held


@pytest.mark.parametrize("who", ["same context", "another context", "cost model"])
def test_kept_matrix_gives_way_to_other_allocations(tmp_path, who):
    """On a device that is full but for the matrix a context keeps after a
    traceback, whatever else allocates gets that memory."""
    import torch
    g, _ = gen_graph(tmp_path, "g", backbone_len=100_000, seed=2)
    read = g.gen_reads(1, 3, 9000).to_list()[0]
    short = g.gen_reads(3, 4, 100).to_list()
    want = cb.Context(0).load(g).align_scores(short)
    ctx, other = cb.Context(0).load(g), cb.Context(0).load(g)
    model = cb.CostModel(0, seed=1)
    # kernels of the calls below are loaded before the device is full
    for c in (ctx, other):
        c.align_scores_batched(short, slots=32, row_bits=32, row_kernel=cb.ROW_DIRECT)
        c.align_traceback(short[0])
    model.predict([[1.0] * 8])
    part = read[:7000]
    part_score = ctx.align_scores([part])[0]
    _, score, ck = ctx.align_traceback(read)  # about 0.8 GB
    assert not ck
    held = _fill(64 << 20)
    try:
        assert torch.cuda.mem_get_info(0)[0] < 100 << 20
        if who == "same context":  # about 140 MB of score rows
            got = ctx.align_scores_batched(short, slots=128, row_bits=32, row_kernel=cb.ROW_DIRECT)
            assert list(got) == list(want)
        elif who == "another context":  # a matrix of about 0.6 GB
            assert other.align_traceback(part)[1] == part_score
        else:  # about 400 MB of samples
            assert model.predict([[1.0] * 8] * (10 << 20)).shape == (10 << 20, 2)
    finally:
        del held
        torch.cuda.empty_cache()
    # and the context goes on
    assert ctx.align_traceback(read)[1] == score
    for c in (ctx, other):
        c.close()
    model.close()


def test_workers_keep_no_more_than_the_budget(tmp_path):
    """hbm_budget_bytes bounds what the traceback workers hold between and
    during requests, whichever worker each request falls to: here it has room
    for one request and there are four workers."""
    import torch
    g, _ = gen_graph(tmp_path, "g", backbone_len=100_000, seed=2)
    read = g.gen_reads(1, 3, 9000).to_list()[0]
    ctx = cb.Context(0).load(g)
    need = 2 * g.stats()["num_chars"] * 9100
    srv = cb.Server(ctx, tb_workers=4, slots=16, hbm_budget_bytes=need)
    for _ in range(4):
        srv.submit(read[:50], cb.REQ_TRACEBACK)
    srv.collect()
    before = torch.cuda.mem_get_info(0)[0]
    scores = set()
    for _ in range(24):
        t = srv.submit(read, cb.REQ_TRACEBACK)
        r = srv.collect()[t]
        assert r["status"] == cb.OK and not r["checkpointed"] and r["projected_bytes"] <= need
        scores.add(r["score"])
        assert before - torch.cuda.mem_get_info(0)[0] <= need + (200 << 20)
    assert len(scores) == 1
    srv.close()
    ctx.close()
