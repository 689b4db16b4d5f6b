"""Performance cases: the alignment work a user of this library has it do.

Every alignment case runs on a seeded variant-bubble graph held by a loaded
context (what a program keeps between calls) with reads sampled from the
graph; the reads are the inputs and change with the seed. Graphs have string
vertices of 1 to 32 bp, as the benchmark's workloads do, on backbones from
20 kbp (a gene region) over 100 kbp and 1 Mbp to 5 Mbp (the benchmark graph).

  plain       align_scores, one read after another (the score-only driver)
  noalloc     align_scores_noalloc, the same without device allocation
  batched     align_scores_batched at 2 to 128 slots, 16- or 32-bit rows
  tb          align_traceback, full matrix or checkpointed every k rows
  tb_batched  align_traceback_batched
  served      a Server fed with a burst of reads, drained
  cm_train    the learned cost model trained on request logs, then asked

Scores, paths and flags are whole numbers and have no exact() of their own;
the cost model's parameters and predictions are floating-point and do.
"""
import math

import numpy as np

import chsga_b200 as cb

MIX = dict(p_snp=0.7, p_indel=0.2, p_alt=0.1, indel_min=1, indel_max=20, alt_min=50, alt_max=300,
           vlen_min=1, vlen_max=32)
SHORT = dict(sub_rate=0.01, indel_rate=0.003, n_rate=0.001)   # sequencer short reads
ONT = dict(sub_rate=0.02, indel_rate=0.03, n_rate=0.0)        # long reads, 5% errors


def listed():
    return [
        # the shortest call: three reads of 100 bp against a 100 kbp region
        dict(name="plain_3x100_100k", op="plain", backbone=100_000, gap=90.9, count=3, len_min=100, len_max=100,
             err="ont", match_n=False),
        # the score-only driver's five reads on the benchmark graph
        dict(name="plain_5x150_5M", op="plain", backbone=5_000_000, gap=50.0, count=5, len_min=150, len_max=150,
             err="short", match_n=False),
        # 200 short reads on the 100 kbp graph, default options
        dict(name="batched_200x150_100k", op="batched", backbone=100_000, gap=90.9, count=200, len_min=150,
             len_max=150, err="short", match_n=False, slots=64, row_bits=0),
        # a few uneven reads at a time under matchN scoring
        dict(name="batched_8slots_1M", op="batched", backbone=1_000_000, gap=50.0, count=21, len_min=150,
             len_max=700, err="ont", match_n=True, slots=8, row_bits=0),
        # short reads in bulk on the benchmark graph, default options
        dict(name="batched_192x150_5M", op="batched", backbone=5_000_000, gap=50.0, count=192, len_min=150,
             len_max=150, err="short", match_n=False, slots=64, row_bits=0),
        # the benchmark's read mix, capped at 2 kbp, at the throughput setting
        dict(name="batched_mixed_5M", op="batched", backbone=5_000_000, gap=50.0, count=160, len_min=150,
             len_max=2000, err="ont", match_n=False, slots=128, row_bits=0),
        # 32-bit rows, what a batch holding a read over 65 kbp runs with
        dict(name="batched_rows32_100k", op="batched", backbone=100_000, gap=90.9, count=33, len_min=150,
             len_max=1000, err="ont", match_n=False, slots=16, row_bits=32),
        # one read's path on the benchmark graph, full matrix
        dict(name="tb_150_5M", op="tb", backbone=5_000_000, gap=50.0, count=1, len_min=150, len_max=150,
             err="short", match_n=False, k=500, full=True),
        # a long read's path through checkpoints (matrix above the byte cap)
        dict(name="tb_ckpt_1501_100k", op="tb", backbone=100_000, gap=90.9, count=1, len_min=1501, len_max=1501,
             err="ont", match_n=False, k=500, full=False),
        # paths of many short reads
        dict(name="tb_batched_32x150_1M", op="tb_batched", backbone=1_000_000, gap=50.0, count=32, len_min=150,
             len_max=150, err="short", match_n=False, slots=32),
        # a burst of requests to the serving loop: 80% short reads, the rest 1 to 2 kbp
        dict(name="served_mix_1M", op="served", backbone=1_000_000, gap=50.0, count=160, len_min=150, len_max=2000,
             err="ont", match_n=False, slots=128),
        # the admission model retrained on the logged requests
        dict(name="cm_train_279", op="cm_train", n=279, epochs=100, batch=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["plain", "plain", "noalloc", "batched", "batched", "batched", "tb", "tb", "tb_batched", "served",
                     "cm_train"])
    if op == "cm_train":
        return dict(op=op, n=_log(rng, 65, 1000), epochs=rng.randint(5, 60), batch=rng.choice([33, 64, 128, 256]))
    c = dict(op=op, backbone=_log(rng, 20_000, 5_000_000), gap=rng.choice([30.0, 50.0, 90.9]),
             err=rng.choice(["short", "ont"]), match_n=rng.random() < 0.25)
    chars = c["backbone"] * 1.4
    slots = 1
    if op == "batched":
        slots = c["slots"] = rng.choice([2, 4, 8, 16, 32, 64, 64, 128, 128])
        c["row_bits"] = 32 if rng.random() < 0.15 else 0
    elif op == "tb_batched":
        slots = c["slots"] = rng.choice([4, 8, 16, 32, 64])
    elif op == "served":
        slots = c["slots"] = rng.choice([32, 64, 128])
    # rows that fit the time of the largest listed case, by the cells they hold
    row_us = 60 + chars / 1e6 * (8 + 0.9 * slots) * (2 if c.get("row_bits") == 32 else 1)
    rows = 0.7e6 / (row_us * (4 if op in ("tb", "tb_batched") else 1))
    if op == "tb":
        c.update(count=1, k=rng.choice([64, 250, 500]), full=rng.random() < 0.6)
        top = min(2000, rows, 20e9 / (chars * 2) if c["full"] else 1e9)
        c["len_min"] = c["len_max"] = _log(rng, 20, max(21, top))
    elif op in ("plain", "noalloc"):
        c["count"] = rng.randint(3, 5)
        c["len_max"] = _log(rng, 40, max(41, min(2000, rows / c["count"])))
        c["len_min"] = max(20, c["len_max"] // rng.randint(1, 4))
    else:
        c["len_max"] = _log(rng, 40, max(41, min(600 if op == "tb_batched" else 2000, rows / 2)))
        c["len_min"] = max(10, c["len_max"] // rng.randint(1, 8))
        waves = max(0.3, rows / c["len_max"])
        c["count"] = max(5, min(600, int(slots * rng.uniform(0.3, min(3.0, waves)))))
        if op == "tb_batched":
            c["count"] = max(5, min(c["count"], int(20e9 / (chars * 2 * c["len_max"]))))
    return c


_graphs = {}


def _graph(case):
    """The host graph of a case, as a program loads it once (kept for the last few cases)."""
    key = (case["backbone"], case["gap"])
    if key not in _graphs:
        while len(_graphs) >= 6:
            _graphs.pop(next(iter(_graphs)))
        g = cb.HostGraph.generate(backbone_len=case["backbone"], seed=2, bubble_gap_mean=case["gap"], **MIX)
        g.build_pch()
        _graphs[key] = (g, g.stats())
    return _graphs[key]


def _reads(case, g, seed):
    err = SHORT if case["err"] == "short" else ONT
    if case["op"] != "served":
        return g.gen_reads(case["count"], seed, case["len_min"], case["len_max"], **err).to_list()
    longs = max(1, case["count"] // 5)
    lo = min(case["len_max"], max(case["len_min"], case["len_max"] // 2))
    out = g.gen_reads(case["count"] - longs, seed, case["len_min"], case["len_min"], **SHORT).to_list()
    out += g.gen_reads(longs, seed + 1, lo, case["len_max"], **err).to_list()
    np.random.default_rng(seed).shuffle(out)
    return out


def _logs(case, seed):
    """Request logs as the serving loop writes them: 8 features, time in ms and device bytes."""
    r = np.random.default_rng(seed)
    n = case["n"]
    ln = np.exp(r.uniform(np.log(150), np.log(10_000), n))
    big = r.random(n) < 0.3
    chars, strings = np.where(big, 139e6, 6.37e6), np.where(big, 13e6, 549e3)
    tb = r.random(n) < 0.4
    ckpt = tb & (ln > 600)
    k = np.where(ckpt, r.choice([100.0, 250.0, 500.0], n), 1.0)
    slots = np.where(tb, 1.0, r.choice([64.0, 128.0], n))
    x = np.stack([np.log2(ln + 1), np.log2(chars), np.log2(strings), np.log2(2 * strings + 1),
                  np.log2(np.where(big, 46.0, 43.0)), np.log2(slots), tb * 1.0, np.log2(k)], 1)
    ms = ln * (0.04 + chars * 6e-8) * np.where(ckpt, 2.2, 1.0) * np.exp(0.05 * r.standard_normal(n))
    by = np.where(tb, chars * 2 * np.where(ckpt, k, ln), ln + 256) * np.exp(0.01 * r.standard_normal(n))
    y = np.stack([ms, by], 1)
    lim = [math.sqrt(6 / 8)] * (8 * 64) + [0.0] * 64 + [math.sqrt(6 / 64)] * (64 * 64) + [0.0] * 64
    lim += [math.sqrt(6 / 64)] * 128 + [0.0] * 2
    init = (r.uniform(-1, 1, len(lim)) * np.array(lim)).astype(np.float32)
    return x.astype(np.float32), y.astype(np.float32), init


def prepare(case, seed):
    if case["op"] == "cm_train":
        x, y, init = _logs(case, seed)
        return dict(case=case, model=cb.CostModel(0, seed=9), x=x, y=y, init=init, seed=int(seed) % 1000)
    g, _ = _graph(case)
    ctx = cb.Context(0, flags=cb.FLAG_MATCH_N if case["match_n"] else 0).load(g)
    st = dict(case=case, ctx=ctx, reads=_reads(case, g, seed))
    if case["op"] == "served":
        st["server"] = cb.Server(ctx, slots=case["slots"])
    return st


def _padded(paths, case):
    """Paths of different lengths in one array: a path steps to a row or along it, at most once per error."""
    out = np.full((len(paths), 2 * case["len_max"] + 16, 3), -1, np.int64)
    for o, p in zip(out, paths):
        o[:len(p)] = p
    return out


def run(state):
    case, op = state["case"], state["case"]["op"]
    if op == "cm_train":
        m = state["model"]
        m.set_params(state["init"])
        loss = m.train(state["x"], state["y"], epochs=case["epochs"], batch=case["batch"], seed=state["seed"])
        params, norm = m.params()
        return dict(loss=np.array([loss], np.float32), params=params, norm=norm,
                    log_pred=np.log(m.predict(state["x"])))
    ctx, reads = state["ctx"], state["reads"]
    if op == "plain":
        return ctx.align_scores(reads)
    if op == "noalloc":
        return ctx.align_scores_noalloc(reads)
    if op == "batched":
        return ctx.align_scores_batched(reads, slots=case["slots"], row_bits=case["row_bits"])
    if op == "tb":
        ops, score, ck = ctx.align_traceback(reads[0], k=case["k"], cap_bytes=0 if case["full"] else 1 << 20)
        return dict(ops=_padded([ops], case), length=len(ops), score=score, checkpointed=ck)
    if op == "tb_batched":
        res = ctx.align_traceback_batched(reads, slots=case["slots"])
        return dict(ops=_padded([r[0] for r in res], case), lengths=np.array([len(r[0]) for r in res]),
                    scores=np.array([r[1] for r in res]))
    srv = state["server"]
    tickets = [srv.submit(r) for r in reads]
    got = srv.collect()
    return np.array([(got[t]["status"], got[t]["score"], got[t]["vertex"]) for t in tickets], np.int64)


def work(case):
    if case["op"] == "cm_train":
        steps = case["epochs"] * (case["n"] // min(case["n"], case["batch"]))
        mul = 8 * 64 + 64 * 64 + 64 * 2
        return dict(bytes=4 * (10 * case["n"] + 2 * 4866 + 22 + 2 * case["n"]),
                    flops=6.0 * mul * min(case["n"], case["batch"]) * steps + 4.0 * mul * case["n"])
    g, st = _graph(case)
    rows = sum(len(r) for r in _reads(case, g, 1))
    # labels (2 bits and the N flag), vertex offsets and in-edges, hierarchy edges (source and weight)
    graph = st["num_chars"] * 3 / 8 + 4 * st["num_strings"] + 4 * st["num_string_edges"] + 8 * (
        st["pch_up_edges"] + st["pch_down_edges"])
    outputs = 4 * case["count"] if case["op"] in ("plain", "noalloc", "batched") else 24 * rows
    # whole-number operations of a cell: three sums and two minima, and the closure's minimum
    return dict(bytes=graph + rows + outputs, flops=6.0 * rows * st["num_chars"])


def exact(case, seed):
    """The cost model's training in 64 bits; alignments return whole numbers only."""
    if case["op"] != "cm_train":
        return None
    x32, y32, init = _logs(case, seed)
    n, batch, epochs = case["n"], min(case["n"], case["batch"]), case["epochs"]
    x, t = x32.astype(np.float64), np.log(y32.astype(np.float64))
    norm = np.concatenate([x.mean(0), np.maximum(1e-3, x.std(0)), t.mean(0), np.maximum(1e-3, t.std(0))])
    x, t = (x - norm[:8]) / norm[8:16], (t - norm[16:18]) / norm[18:20]
    shapes = [(8, 64), (64,), (64, 64), (64,), (64, 2), (2,)]
    p, at = [], 0
    for s in shapes:
        p.append(init[at:at + int(np.prod(s))].astype(np.float64).reshape(s))
        at += int(np.prod(s))
    m, v = [np.zeros_like(q) for q in p], [np.zeros_like(q) for q in p]

    def forward(q):
        h1 = np.maximum(q @ p[0] + p[1], 0)
        h2 = np.maximum(h1 @ p[2] + p[3], 0)
        return h1, h2, h2 @ p[4] + p[5]

    mask = (1 << 64) - 1
    s, perm, step = ((int(seed) % 1000) ^ 0x7EA1B) & mask, list(range(n)), 0
    b1, b2, lr, eps = (float(np.float32(q)) for q in (0.9, 0.999, 3e-3, 1e-8))
    for _ in range(epochs):
        for i in range(n, 1, -1):
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % i
            perm[i - 1], perm[j] = perm[j], perm[i - 1]
        for off in range(0, n - batch + 1, batch):
            b = perm[off:off + batch]
            h1, h2, o = forward(x[b])
            d = (o - t[b]) / batch
            z2 = (d @ p[4].T) * (h2 > 0)
            z1 = (z2 @ p[2].T) * (h1 > 0)
            grads = [x[b].T @ z1, z1.sum(0), h1.T @ z2, z2.sum(0), h2.T @ d, d.sum(0)]
            step += 1
            for q, gr, a, c in zip(p, grads, m, v):
                a += (1 - b1) * (gr - a)
                c += (1 - b2) * (gr * gr - c)
                q -= lr * (a / (1 - b1 ** step)) / (np.sqrt(c / (1 - b2 ** step)) + eps)
    o = forward(x)[2]
    return dict(loss=np.array([0.5 * ((o - t) ** 2).sum() / n]), params=np.concatenate([q.ravel() for q in p]),
                norm=norm, log_pred=o * norm[18:20] + norm[16:18])
