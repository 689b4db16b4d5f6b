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
