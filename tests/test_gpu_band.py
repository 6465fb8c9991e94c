"""GPU parity of the band kernel's windows and of the split of a last class between it and the
row-parallel kernel (g3x_band.cu, launch_last): long queries on a context as it is created, bands
on both sides of every window and register width, seed scores that leave row -1 in columns the
band has not reached (the stale entries of ksw.cu:388-391), to-end scores, cell and row counts,
against the oracle."""
import numpy as np
import pytest

import g3sa_b200 as g
from tests import native as nat
from tests.gpu_util import to_dev
from tests.test_gpu_group16 import run

pytestmark = pytest.mark.gpu

WS = (1, 5, 31, 32, 63, 64, 111, 112, 127, 128, 191, 192, 255, 256, 383, 384, 511, 512, 700)


def band_jobs(n, seed, ws, h0s, qmin=257):
    wl = g.synth(4, n, seed=seed, w=60, unrelated=0.0)
    rng = np.random.default_rng(seed)
    jobs = wl.jobs.copy()
    jobs["qlen"] = np.minimum(jobs["qlen"], rng.integers(qmin, 1200, n))
    jobs["tlen"] = np.minimum(jobs["tlen"], jobs["qlen"] + rng.integers(-200, 300, n)).astype(np.uint16)
    jobs["w"] = rng.choice(ws, n)
    jobs["h0"] = rng.choice(h0s, n)
    jobs["flags"] = rng.integers(0, 4, n)
    return wl.u8, jobs


@pytest.mark.parametrize("score", [{}, dict(o_del=5, e_del=2, o_ins=7, e_ins=1), dict(a=3, b=2, o_del=1, e_del=9, o_ins=2, e_ins=5),
                                   dict(zdrop=0)])
@pytest.mark.parametrize("n", [60, 6000])
def test_default_context_long_queries(score, n):
    sc = g.default_score(**score)
    for h0s in ((1, 19, 150), (120, 400, 900)):
        u8, jobs = band_jobs(n if n < 1000 else n // 8, 7 + n, WS, h0s)
        if n > 1000:                                   # beyond the batches run as listed: with short ones
            jobs = np.concatenate([jobs] * 8)
            jobs["qlen"][::3] = np.minimum(jobs["qlen"][::3], 200)
        ref, cells, rows = nat.oracle_extend(jobs, u8, sc)
        out, status, gcells, grows, _ = run(u8, jobs, sc)
        assert (status == 0).all()
        np.testing.assert_array_equal(out, ref)
        np.testing.assert_array_equal(gcells, cells)
        np.testing.assert_array_equal(grows, rows)
        np.testing.assert_array_equal(run(u8, jobs, sc, rows=False)[0], ref)


def test_split_keeps_what_no_window_takes():
    """Bands beyond 1,024 columns and scores from 2^21 stay in the row-parallel kernel; refused jobs
    get one status whatever the split."""
    sc = g.default_score()
    u8, jobs = band_jobs(300, 3, (40, 600, 900), (19, 150))
    jobs["h0"][:40] = 1 << 21
    jobs["h0"][40:60] = -1
    jobs["h0"][60:80] = -70000
    jobs["q_off"][80:90] = len(u8) - 5
    want = run(u8, jobs, sc, kernel=g.KERNEL_ROWPAR, n_bases=len(u8))
    got = run(u8, jobs, sc, n_bases=len(u8))
    for a, b in zip(got[:4], want[:4]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kernel_tile", [256, 512, 1024])
def test_band_kernel_small_queries_and_tails(kernel_tile):
    """Every register width of a window on short queries too: lengths 0, 1 and around the band."""
    sc = g.default_score()
    ws = [w for w in WS if 2 * w + 2 <= kernel_tile]
    u8, jobs = band_jobs(400, kernel_tile, ws, (0, 1, 19, 60, 150, 500), qmin=300)
    rng = np.random.default_rng(kernel_tile)
    jobs["qlen"] = rng.choice([0, 1, 2, 30, 64, 101, 128, 300, 600], len(jobs))
    jobs["tlen"] = np.minimum(jobs["tlen"], rng.choice([0, 1, 16, 17, 200, 700], len(jobs)))
    ref, cells, rows = nat.oracle_extend(jobs, u8, sc)
    import torch
    c = g.Context(0)
    n = len(jobs)
    codes, nmask = g.pack_planes(u8)
    out = torch.full((n, 6), -777, dtype=torch.int32, device="cuda")
    status, gcells, grows = (torch.full((n,), 99, dtype=torch.int32, device="cuda") for _ in range(3))
    c.extend_batch(sc, to_dev(jobs), n, to_dev(codes), to_dev(nmask), out, status, int(jobs["qlen"].max()),
                   int(jobs["tlen"].max()), schedule=g.SCHED_SORTED, kernel=g.KERNEL_BAND, tile=kernel_tile, d_cells=gcells,
                   d_rows=grows)
    torch.cuda.synchronize()
    assert (status.cpu().numpy() == 0).all()
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    np.testing.assert_array_equal(gcells.cpu().numpy(), cells)
    np.testing.assert_array_equal(grows.cpu().numpy(), rows)
    c.close()


@pytest.mark.parametrize("n", [9000, 17000])
@pytest.mark.parametrize("kernel,tile", [(g.KERNEL_AUTO, 0), (g.KERNEL_BAND, 512), (g.KERNEL_BAND, 256)])
def test_negative_bands_beside_wide_ones(n, kernel, tile):
    """A warp's jobs share the registers that the widest of its bands needs (two and four jobs a warp from
    8,000 and 16,000 jobs on); a band below 0, which has no cells, changes nothing for the others."""
    import torch
    sc = g.default_score()
    u8, base = band_jobs(340, 5, (100, 120) if tile == 256 else (100, 240), (19, 150))
    base["tlen"] = np.minimum(base["tlen"], np.random.default_rng(1).choice([300, 420, 600], len(base)))
    ref, cells, rows = nat.oracle_extend(base, u8, sc)
    jobs = np.resize(base, n)
    at, neg = np.arange(n) % len(base), np.arange(n) % 7 == 3
    jobs["w"][neg] = np.where(np.arange(n)[neg] % 2, -1, -5)
    codes, nmask = g.pack_planes(u8)
    out = torch.full((n, 6), -777, dtype=torch.int32, device="cuda")
    status, gcells, grows = (torch.full((n,), 99, dtype=torch.int32, device="cuda") for _ in range(3))
    c = g.Context(0)
    c.extend_batch(sc, to_dev(jobs), n, to_dev(codes), to_dev(nmask), out, status, int(jobs["qlen"].max()),
                   int(jobs["tlen"].max()), schedule=g.SCHED_SORTED, kernel=kernel, tile=tile, d_cells=gcells,
                   d_rows=grows)
    torch.cuda.synchronize()
    c.close()
    assert (status.cpu().numpy() == 0).all()
    ok = ~neg
    np.testing.assert_array_equal(out.cpu().numpy()[ok], ref[at[ok]])
    np.testing.assert_array_equal(gcells.cpu().numpy()[ok], cells[at[ok]])
    np.testing.assert_array_equal(grows.cpu().numpy()[ok], rows[at[ok]])


def test_tuned_last_class_runs_each_job_once():
    """The last class of a tuned table may refill a warp's groups together (warp_batch), a path that takes
    every job; it is tuned when the sample holds queries beyond the bound given for it.  Longer jobs
    then: every result, and the row and cell counts, as from one run of each job."""
    import torch
    sc = g.default_score()
    u8, jobs = band_jobs(600, 11, (40, 100), (19, 150))
    jobs["qlen"][::4] = 180
    ref, cells, rows = nat.oracle_extend(jobs, u8, sc)
    codes, nmask = g.pack_planes(u8)
    d = to_dev(jobs), len(jobs), to_dev(codes), to_dev(nmask)
    mq, mt = int(jobs["qlen"].max()), int(jobs["tlen"].max())
    c = g.Context(0)
    for _ in range(4):
        c.autotune(sc, *d, 200, mt)
        out = torch.full((len(jobs), 6), -777, dtype=torch.int32, device="cuda")
        status, gcells, grows = (torch.full((len(jobs),), 99, dtype=torch.int32, device="cuda") for _ in range(3))
        c.extend_batch(sc, *d, out, status, mq, mt, schedule=g.SCHED_SORTED, d_cells=gcells, d_rows=grows)
        torch.cuda.synchronize()
        assert (status.cpu().numpy() == 0).all()
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
        np.testing.assert_array_equal(grows.cpu().numpy(), rows)
        np.testing.assert_array_equal(gcells.cpu().numpy(), cells)
    c.close()


@pytest.mark.parametrize("w,n,ordered", [(60, 3000, False), (200, 2000, False), (200, 2100, True), (500, 512, False), (500, 600, True)])
def test_long_jobs_of_wide_bands_stay_ordered(w, n, ordered):
    """Long jobs that wait for a warp are sorted (the jobs per class show the sort: all in the rest of the
    groups' classes), those that start at once are taken as they come; the bounds show the band."""
    import torch
    sc = g.default_score()
    wl = g.synth(4, n, seed=w, w=w, unrelated=0.0)
    jobs = wl.jobs[wl.jobs["qlen"] > 256]
    jobs = np.resize(jobs, n)
    jobs["qlen"] = np.minimum(jobs["qlen"], 700)
    jobs["tlen"] = np.minimum(jobs["tlen"], jobs["qlen"] + 2 * w)
    ref, _, _ = nat.oracle_extend(jobs, wl.u8, sc)
    codes, nmask = wl.planes()
    d_codes, d_nmask, mq = to_dev(codes), to_dev(nmask), int(jobs["qlen"].max())
    c = g.Context(0)
    seen = []
    for k in (513 if w == 500 else 2049 if w == 200 else 4097, n):        # a sorted batch first
        more = np.resize(jobs, k)
        out = torch.zeros((k, 6), dtype=torch.int32, device="cuda")
        status = torch.full((k,), 9, dtype=torch.int32, device="cuda")
        c.extend_batch(sc, to_dev(more), k, d_codes, d_nmask, out, status, mq, mq + 2 * w, schedule=g.SCHED_SORTED)
        torch.cuda.synchronize()
        assert (status.cpu().numpy() == 0).all()
        np.testing.assert_array_equal(out.cpu().numpy(), np.resize(ref, (k, 6)))
        seen.append(c.class_times()[4][1])
    c.close()
    assert seen[0] > 0 and (seen[1] == n) == ordered and (ordered or seen[1] == seen[0])
