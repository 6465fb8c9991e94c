"""GPU parity of the batched banded global alignment (g3x_ksw_global2_batch, ksw_global2 of
bwa/src/ksw.cu:706-809) against the oracle's restatement, itself pinned to the reference's
own ksw_global2 (tests/test_global_oracle.py): scores and CIGARs bit-exact, empty CIGARs where
no in-band alignment reaches the last cell, reversed reads, and the job limits."""
import numpy as np
import pytest

import g3sa_b200 as g
from tests import native as nat
from tests.gpu_util import ctx, to_dev

pytestmark = pytest.mark.gpu


def gpu_jobs(cj, flags=0):
    j = np.zeros(len(cj), g.JOB_DT)
    j["q_off"], j["t_off"] = cj["q_off"], cj["t_off"]
    j["qlen"], j["tlen"], j["w"] = cj["qlen"], cj["tlen"], cj["w"]
    j["flags"] = flags
    return j


def run_global(jobs, u8, stride, max_qlen=None, max_tlen=None, max_w=None):
    import torch
    n = len(jobs)
    codes, nmask = g.pack_planes(u8)
    d_score = torch.zeros(n, dtype=torch.int32, device="cuda")
    d_cig = torch.zeros(n * stride, dtype=torch.int32, device="cuda")
    d_nc = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    d_st = torch.full((n,), 99, dtype=torch.int32, device="cuda")
    mq = int(jobs["qlen"].max()) if max_qlen is None else max_qlen
    mt = int(jobs["tlen"].max()) if max_tlen is None else max_tlen
    mw = int(jobs["w"].max()) if max_w is None else max_w
    ctx().global_batch(g.default_score(), to_dev(jobs), n, to_dev(codes), to_dev(nmask), mq, mt, mw, d_score,
                       d_cig, stride, d_nc, d_st)
    torch.cuda.synchronize()
    return (d_score.cpu().numpy(), d_cig.cpu().numpy().view(np.uint32).reshape(n, stride), d_nc.cpu().numpy(),
            d_st.cpu().numpy())


@pytest.mark.parametrize("seed,max_len", [(1, 160), (5, 300), (9, 40)])
def test_gpu_global_matches_oracle(seed, max_len):
    cj, u8 = nat.global_jobs(4000, seed, max_len=max_len)
    stride = int((cj["qlen"] + cj["tlen"]).max()) + 2
    s1, c1, n1, _ = nat.oracle_global(cj, u8, g.default_score(), stride)
    s2, c2, n2, st = run_global(gpu_jobs(cj), u8, stride)
    assert (st == 0).all(), np.unique(st)
    assert np.array_equal(s1, s2)
    assert np.array_equal(n1, n2)
    bad = [k for k in range(len(cj)) if not np.array_equal(c1[k, :n1[k]], c2[k, :n2[k]])]
    assert not bad, bad[:5]


def test_gpu_global_reversed_reads():
    """G3X_JOB_QREV/TREV read the planes backwards: the same as the oracle on reversed copies."""
    cj, u8 = nat.global_jobs(1500, 11)
    stride = int((cj["qlen"] + cj["tlen"]).max()) + 2
    rev = u8.copy()
    for j in cj:
        a, b = int(j["q_off"]), int(j["q_off"] + j["qlen"])
        rev[a:b] = u8[a:b][::-1]
        a, b = int(j["t_off"]), int(j["t_off"] + j["tlen"])
        rev[a:b] = u8[a:b][::-1]
    s1, c1, n1, _ = nat.oracle_global(cj, rev, g.default_score(), stride)
    s2, c2, n2, st = run_global(gpu_jobs(cj, g.JOB_QREV | g.JOB_TREV), u8, stride)
    assert (st == 0).all() and np.array_equal(s1, s2) and np.array_equal(n1, n2)
    assert all(np.array_equal(c1[k, :n1[k]], c2[k, :n2[k]]) for k in range(len(cj)))


def test_gpu_global_limits():
    """Jobs beyond the call's bounds, and CIGARs beyond the stride, get G3X_ERR_TOO_LONG."""
    cj, u8 = nat.global_jobs(600, 13, ws=(3, 5, 17))
    jobs = gpu_jobs(cj)
    stride = 4
    s1, c1, n1, _ = nat.oracle_global(cj, u8, g.default_score(), int((cj["qlen"] + cj["tlen"]).max()) + 2)
    s2, c2, n2, st = run_global(jobs, u8, stride, max_qlen=100, max_w=10)
    over = (cj["qlen"] > 100) | (cj["w"] > 10)
    assert (st[over] == g.G3X_ERR_TOO_LONG).all()
    fits = ~over & (n1 <= stride)
    assert (st[fits] == 0).all() and np.array_equal(s2[fits], s1[fits]) and np.array_equal(n2[fits], n1[fits])
    long_ = ~over & (n1 > stride)
    assert long_.any() and (st[long_] == g.G3X_ERR_TOO_LONG).all() and (n2[long_] == 0).all()


def test_gpu_global_nm_md():
    """NM and MD (the traceback stage's block after ksw_global2) equal the oracle's, itself
    pinned to the reference's own block (tests/test_global_oracle.py)."""
    import torch
    cj, u8 = nat.global_jobs(3000, 21, max_len=200)
    cj["flags"][::3] = g.JOB_MDRC
    jobs = gpu_jobs(cj)
    jobs["flags"] = cj["flags"]
    n = len(cj)
    stride = int((cj["qlen"] + cj["tlen"]).max()) + 2
    md_stride = 4 * stride + 16
    s1, c1, n1, _ = nat.oracle_global(cj, u8, g.default_score(), stride)
    nm1, md1 = nat.oracle_nm_md(cj, u8, c1, n1, md_stride)
    codes, nmask = g.pack_planes(u8)
    d_score = torch.zeros(n, dtype=torch.int32, device="cuda")
    d_cig = torch.zeros(n * stride, dtype=torch.int32, device="cuda")
    d_nc = torch.zeros(n, dtype=torch.int32, device="cuda")
    d_st = torch.full((n,), 99, dtype=torch.int32, device="cuda")
    d_nm = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    d_md = torch.zeros(n * md_stride, dtype=torch.uint8, device="cuda")
    ctx().global_batch(g.default_score(), to_dev(jobs), n, to_dev(codes), to_dev(nmask), int(cj["qlen"].max()),
                       int(cj["tlen"].max()), int(cj["w"].max()), d_score, d_cig, stride, d_nc, d_st,
                       d_nm=d_nm, d_md=d_md, md_stride=md_stride)
    torch.cuda.synchronize()
    assert (d_st.cpu().numpy() == 0).all()
    assert np.array_equal(d_nm.cpu().numpy(), nm1)
    md = d_md.cpu().numpy().reshape(n, md_stride)
    md2 = [bytes(md[k]).split(b"\0")[0].decode() for k in range(n)]
    assert md2 == md1


@pytest.mark.parametrize("long_len", [0, 3500])
def test_gpu_global_both_ring_forms(long_len):
    """Short batches keep H and E as int16 pairs (-2^14 outside the band), batches with long
    sequences as int32 pairs (the reference's -2^30): both equal the oracle, scores from outside
    the band included (jobs whose band misses the last cell)."""
    cj, u8 = nat.global_jobs(1500, 21 + long_len, max_len=120, ws=(0, 1, 3, 10, 40))
    if long_len:
        rng = np.random.default_rng(long_len)
        extra = []
        for k in range(6):
            q = rng.integers(0, 4, long_len - 300 * k).astype(np.uint8)
            t = q.copy()
            t[rng.integers(0, len(t), 40)] = rng.integers(0, 4, 40)
            extra.append((q, t[: len(t) - 20 * k]))
        off = len(u8)
        ej = np.zeros(len(extra), cj.dtype)
        parts = [u8]
        for k, (q, t) in enumerate(extra):
            ej[k]["q_off"], ej[k]["t_off"], ej[k]["qlen"], ej[k]["tlen"], ej[k]["w"] = off, off + len(q), len(q), len(t), 60
            parts += [q, t]
            off += len(q) + len(t)
        cj, u8 = np.concatenate([cj, ej]), np.concatenate(parts)
    # a few jobs whose band cannot reach the last cell: query much longer than target + w
    out_of_band = (cj["qlen"] > cj["tlen"] + cj["w"])
    stride = int((cj["qlen"] + cj["tlen"]).max()) + 2
    s1, c1, n1, _ = nat.oracle_global(cj, u8, g.default_score(), stride)
    s2, c2, n2, st = run_global(gpu_jobs(cj), u8, stride)
    assert (st == 0).all(), np.unique(st)
    assert np.array_equal(s1, s2)
    assert np.array_equal(n1, n2)
    assert all(np.array_equal(c1[k, :n1[k]], c2[k, :n2[k]]) for k in range(len(cj)))
    assert out_of_band.any() and (s1[out_of_band] < -(1 << 29)).any()


def pairs_at_edges(n, seed, ws, lens):
    """Pairs cut to given lengths: targets are edited copies, shortened, lengthened or absent."""
    rng = np.random.default_rng(seed)
    cj, u8 = nat.global_jobs(n, seed, max_len=max(lens) + 1, ws=ws)
    cj["qlen"] = np.minimum(cj["qlen"], rng.choice(lens, n))
    cut = rng.random(n)
    cj["tlen"] = np.where(cut < 0.1, 0, np.where(cut < 0.5, cj["tlen"], np.minimum(cj["tlen"], rng.choice(lens, n))))
    return cj, u8


@pytest.mark.parametrize("n", [1, 3, 1024, 1025, 5000])
@pytest.mark.parametrize("score", [{}, dict(o_del=5, e_del=2, o_ins=7, e_ins=1), dict(a=6, b=9, o_del=0, e_del=5, o_ins=1, e_ins=6)])
def test_gpu_global_group_widths(n, score):
    """Bands on both sides of every group width (2w + 1 columns in 16, 32, 64, 128, 256; a band is
    cut to the longer sequence) and beyond the widest, up to and beyond the batch size that runs
    unsorted: scores, CIGARs, NM and MD equal the oracle's."""
    import torch
    sc = g.default_score(**score)
    for ws in ((0, 1, 3, 4, 7, 8, 15, 16, 31, 32, 63, 64, 126, 127), (2, 7, 100, 127, 128, 200, 500)):
        cj, u8 = pairs_at_edges(n, 31 + n, ws, (0, 1, 2, 7, 8, 9, 16, 33, 64, 127, 128, 200, 255))
        jobs = gpu_jobs(cj)
        stride = int((cj["qlen"] + cj["tlen"]).max()) + 2
        md_stride = 4 * stride + 16
        s1, c1, n1, _ = nat.oracle_global(cj, u8, sc, stride)
        nm1, md1 = nat.oracle_nm_md(cj, u8, c1, n1, md_stride)
        codes, nmask = g.pack_planes(u8)
        out = [torch.full((n * k,), 77, dtype=torch.int32, device="cuda") for k in (1, stride, 1, 1, 1)]
        d_md = torch.zeros(n * md_stride, dtype=torch.uint8, device="cuda")
        ctx().global_batch(sc, to_dev(jobs), n, to_dev(codes), to_dev(nmask), int(cj["qlen"].max()),
                           int(cj["tlen"].max()), int(cj["w"].max()), out[0], out[1], stride, out[2], out[3],
                           d_nm=out[4], d_md=d_md, md_stride=md_stride)
        torch.cuda.synchronize()
        s2, c2, n2, st, nm2 = [t.cpu().numpy() for t in out]
        assert (st == 0).all(), np.unique(st)
        np.testing.assert_array_equal(s2, s1)
        np.testing.assert_array_equal(n2, n1)
        c2 = c2.view(np.uint32).reshape(n, stride)
        for k in range(n):
            assert np.array_equal(c1[k, :n1[k]], c2[k, :n2[k]]), (k, cj[k])
            assert (c2[k, n2[k]:] == 77).all()                  # slots beyond the CIGAR stay
        np.testing.assert_array_equal(nm2, nm1)
        md = d_md.cpu().numpy().reshape(n, md_stride)
        assert [bytes(md[k]).split(b"\0")[0].decode() for k in range(n)] == md1


@pytest.mark.parametrize("n", [1000, 1025, 5000])
@pytest.mark.parametrize("mq,mt,mw", [(250, 260, 100), (120, 120, 300), (250, 260, 400)])
def test_gpu_global_writes_every_refused_pair(n, mq, mt, mw):
    """Jobs beyond the call's bounds or past the planes, their bands on both sides of the widest group's
    (127), with the lane kernel launched (bounds that allow wider bands) and without, unsorted and
    sorted: every output of each is written, whatever the caller's buffers held."""
    import torch
    cj, u8 = nat.global_jobs(n, 41 + n, max_len=250, ws=(5, 20, 100))
    jobs = gpu_jobs(cj)
    k = np.random.default_rng(n).permutation(n)[:200]
    jobs["w"][k[:60]] = np.resize([127, 128, 200, 60000, 0x7FFFFFFF, -1], 60)
    jobs["q_off"][k[60:90]] = len(u8) + 7
    jobs["t_off"][k[90:120]] = 0xFFFFFFF0
    jobs["w"][k[75:105]] = 60000
    q_end, t_end = jobs["q_off"].astype(np.int64) + jobs["qlen"], jobs["t_off"].astype(np.int64) + jobs["tlen"]
    outside = (q_end > len(u8)) | (t_end > len(u8))
    bad = outside | (jobs["qlen"] > mq) | (jobs["tlen"] > mt) | (jobs["w"] > mw) | (jobs["w"] < 0)
    stride, md_stride = 520, 64
    codes, nmask = g.pack_planes(u8)
    out = [torch.full((n * w,), 77, dtype=torch.int32, device="cuda") for w in (1, stride, 1, 1, 1)]
    d_md = torch.full((n * md_stride,), 77, dtype=torch.uint8, device="cuda")
    c = g.Context(0)
    c.global_batch(g.default_score(), to_dev(jobs), n, to_dev(codes), to_dev(nmask), mq, mt, mw, out[0], out[1], stride,
                   out[2], out[3], d_nm=out[4], d_md=d_md, md_stride=md_stride, n_bases=len(u8))
    torch.cuda.synchronize()
    score, _, n_cigar, status, nm = [t.cpu().numpy() for t in out]
    c.close()
    np.testing.assert_array_equal(status[bad], np.where(outside, g.G3X_ERR_INVALID, g.G3X_ERR_TOO_LONG)[bad])
    assert (score[bad] == 0).all() and (n_cigar[bad] == 0).all() and (nm[bad] == 0).all()
    assert (d_md.cpu().numpy().reshape(n, md_stride)[bad, 0] == 0).all()
    taken = cj.copy()
    taken["w"] = jobs["w"]
    s1, _, n1, _ = nat.oracle_global(taken[~bad], u8, g.default_score(), stride)
    assert np.isin(status[~bad], (g.G3X_OK, g.G3X_ERR_TOO_LONG)).all()      # (an MD beyond its stride)
    np.testing.assert_array_equal(score[~bad], s1)
    np.testing.assert_array_equal(n_cigar[~bad], n1)


@pytest.mark.parametrize("max_len,n,md", [(9, 114688, True), (9, 114689, True), (21, 163841, True), (21, 163841, False), (13, 163841, False)])
def test_gpu_global_short_pairs(max_len, n, md):
    """Large batches of very short pairs on both sides of the line from which the lane kernel runs them, in one
    context whose scratch an ordinary batch of the same bounds sized first."""
    import torch
    sc = g.default_score()
    cj, u8 = nat.global_jobs(3000, max_len, max_len=max_len, ws=(0, 3, 5, 20, 50))
    stride, md_stride = int((cj["qlen"] + cj["tlen"]).max()) + 2, 128
    s1, c1, n1, _ = nat.oracle_global(cj, u8, sc, stride)
    nm1, md1 = nat.oracle_nm_md(cj, u8, c1, n1, md_stride)
    codes, nmask = g.pack_planes(u8)
    c = g.Context(0)
    for m in (3000, n):
        jobs = np.resize(gpu_jobs(cj), m)
        out = [torch.full((m * k,), 77, dtype=torch.int32, device="cuda") for k in (1, stride, 1, 1, 1)]
        d_md = torch.zeros(m * md_stride, dtype=torch.uint8, device="cuda")
        c.global_batch(sc, to_dev(jobs), m, to_dev(codes), to_dev(nmask), int(cj["qlen"].max()), int(cj["tlen"].max()),
                       50, out[0], out[1], stride, out[2], out[3], d_nm=out[4] if md else None, d_md=d_md if md else None,
                       md_stride=md_stride if md else 0)
        torch.cuda.synchronize()
        score, cig, nc, status, nm = [t.cpu().numpy() for t in out]
        assert (status == 0).all()
        np.testing.assert_array_equal(score, np.resize(s1, m))
        np.testing.assert_array_equal(nc, np.resize(n1, m))
        used = np.arange(stride)[None, :] < np.resize(n1, m)[:, None]
        want = np.where(used, np.resize(c1, (m, stride)), 77)
        np.testing.assert_array_equal(cig.view(np.uint32).reshape(m, stride), want)
        if md:
            np.testing.assert_array_equal(nm, np.resize(nm1, m))
            text = d_md.cpu().numpy().reshape(m, md_stride)
            for k in range(0, m, 997):
                assert bytes(text[k]).split(b"\0")[0].decode() == md1[k % len(md1)]
    c.close()


def test_gpu_global_captured_after_a_smaller_call():
    """Scratch depends on the call's bounds, not on its pairs (up to the 1,024 that a context's order
    scratch always holds): a call of the same bounds is captured into a graph after a smaller one, and
    the smaller one's graph still runs after it."""
    import torch
    n, small = 1000, 40
    cj, u8 = nat.global_jobs(n, 77, max_len=200, ws=(5, 20))
    codes, nmask = g.pack_planes(u8)
    d_jobs, d_codes, d_nmask = to_dev(gpu_jobs(cj)), to_dev(codes), to_dev(nmask)
    mq, mt = int(cj["qlen"].max()), int(cj["tlen"].max())
    stride = mq + mt + 2
    s1, c1, n1, _ = nat.oracle_global(cj, u8, g.default_score(), stride)
    c = g.Context(0)
    out = [torch.zeros(n * k, dtype=torch.int32, device="cuda") for k in (1, stride, 1, 1)]

    def call(k):
        c.global_batch(g.default_score(), d_jobs, k, d_codes, d_nmask, mq, mt, 20, out[0], out[1], stride, out[2], out[3],
                       stream=st)

    st = torch.cuda.Stream()
    call(small)
    st.synchronize()
    graphs = []
    for k in (small, n):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=st):
            call(k)
    for gr, k in zip(reversed(graphs), (n, small)):
        for t in out:
            t.fill_(77)
        gr.replay()
        torch.cuda.synchronize()
        score, cig, nc, status = [t.cpu().numpy() for t in out]
        assert (status[:k] == 0).all()
        np.testing.assert_array_equal(score[:k], s1[:k])
        np.testing.assert_array_equal(nc[:k], n1[:k])
        cig = cig.view(np.uint32).reshape(n, stride)
        assert all(np.array_equal(cig[j, :n1[j]], c1[j, :n1[j]]) for j in range(k))
    del graphs
    c.close()
