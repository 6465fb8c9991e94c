"""GPU parity of the int16x2 group-per-job kernel (g3x_group16.cu), which small scheduled batches
take on a context whose width classes were not given: against the oracle, and for every kind of job
it may not take against the row-parallel kernel (the general path).  Sizes: queries on both sides
of every group width (31 | 32, 63 | 64, 127 | 128, 255 | 256), batches on both sides of the limits
up to which jobs run as they are listed (4096) and with one block a lane (32768), and one- and
two-job batches."""
import numpy as np
import pytest

import g3sa_b200 as g
from tests import native as nat
from tests.gpu_util import to_dev

pytestmark = pytest.mark.gpu

SCORES = {"bwa": {}, "uneven": dict(o_del=5, e_del=2, o_ins=7, e_ins=1), "steep": dict(a=3, b=2, o_del=1, e_del=30, o_ins=1, e_ins=40),
          "nozdrop": dict(zdrop=0)}


def run(u8, jobs, sc, schedule=g.SCHED_SORTED, kernel=g.KERNEL_AUTO, mq=None, mt=None, n_bases=None, rows=True):
    import torch
    c = g.Context(0)
    n = len(jobs)
    codes, nmask = g.pack_planes(u8)
    out = torch.full((n, 6), -777, dtype=torch.int32, device="cuda")
    status = torch.full((n,), 99, dtype=torch.int32, device="cuda")
    cells = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    d_rows = torch.full((n,), -1, dtype=torch.int32, device="cuda") if rows else None
    c.extend_batch(sc, to_dev(jobs), n, to_dev(codes), to_dev(nmask), out, status,
                   int(jobs["qlen"].max()) if mq is None else mq, int(jobs["tlen"].max()) if mt is None else mt,
                   schedule=schedule, kernel=kernel, d_cells=cells if rows else None, d_rows=d_rows, n_bases=n_bases)
    torch.cuda.synchronize()
    stats = c.last_stats()
    res = [t.cpu().numpy() for t in (out, status, cells)]
    c.close()
    return res + [d_rows.cpu().numpy() if rows else None, stats]


def edge_jobs(n, seed, w):
    """Jobs of the long generator cut to query lengths around the group widths and to targets from
    none to twice the query; reversed reads among them."""
    wl = g.synth(4, n // 4 + 1, seed=seed, w=w, unrelated=0.0)
    rng = np.random.default_rng(seed)
    jobs = np.repeat(wl.jobs, 4)[:n].copy()
    edges = [0, 1, 2, 7, 8, 9, 15, 16, 17, 30, 31, 32, 33, 62, 63, 64, 65, 126, 127, 128, 129, 200, 254, 255, 256, 257, 300]
    jobs["qlen"] = rng.choice(edges, n)
    jobs["tlen"] = np.minimum(jobs["tlen"], rng.choice([0, 1, 15, 16, 17, 64, 300, 480], n))
    jobs["h0"] = rng.choice([0, 1, 5, 19, 60, 150], n)
    jobs["w"] = rng.choice([1, 3, w], n)
    jobs["flags"] = rng.integers(0, 4, n)
    return wl.u8, jobs


@pytest.mark.parametrize("score", list(SCORES))
@pytest.mark.parametrize("n", [1, 2, 63, 4096, 4097, 36000])
def test_edges_match_oracle(score, n):
    sc = g.default_score(**SCORES[score])
    u8, jobs = edge_jobs(n, 17 + n, 40)
    ref, cells, rows = nat.oracle_extend(jobs, u8, sc)
    out, status, gcells, grows, _ = run(u8, jobs, sc)
    assert (status == 0).all()
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(gcells, cells)
    np.testing.assert_array_equal(grows, rows)


@pytest.mark.parametrize("kind,w,units", [(1, 100, 900), (1, 5, 11000), (1, 5, 20000), (2, 100, 500), (2, 100, 12000), (2, 13, 9000),
                                          (2, 13, 12000), (2, 100, 18000)])
@pytest.mark.parametrize("score", ["bwa", "uneven"])
def test_generated_jobs_match_oracle(kind, w, units, score):
    """Batches on both sides of the line that falls with the band: beyond it the lane classes run them."""
    sc = g.default_score(**SCORES[score])
    wl = g.synth(kind, units, seed=units + w, w=w, unrelated=0.3)
    ref, cells, rows = nat.oracle_extend(wl.jobs, wl.u8, sc)
    out, status, gcells, grows, stats = run(wl.u8, wl.jobs, sc)
    assert (status == 0).all()
    # the group kernel counts rows, the lane kernels row blocks
    assert (stats[0] == rows.sum()) == ((kind, w, units) not in ((1, 5, 20000), (2, 13, 12000)))
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(gcells, cells)
    np.testing.assert_array_equal(grows, rows)
    out, status, _, _, _ = run(wl.u8, wl.jobs, sc, rows=False)
    np.testing.assert_array_equal(out, ref)


@pytest.mark.parametrize("n", [200, 9000, 40000])
def test_refused_and_misfit_jobs_as_on_the_general_path(n):
    sc = g.default_score()
    u8, jobs = edge_jobs(n, 5, 40)
    rng = np.random.default_rng(n)
    k = rng.permutation(n)
    jobs["h0"][k[:20]] = 20000                        # outside int16
    jobs["h0"][k[20:30]] = -1                         # refused
    jobs["h0"][k[30:40]] = -50000                     # negative and taken
    jobs["q_off"][k[40:50]] = len(u8) - 3             # past the planes
    jobs["t_off"][k[50:60]] = 0xFFFFFFF0
    jobs["h0"][k[60:70]] = 2000000
    want = run(u8, jobs, sc, kernel=g.KERNEL_ROWPAR, mq=260, mt=400, n_bases=len(u8))
    got = run(u8, jobs, sc, mq=260, mt=400, n_bases=len(u8))
    # a job both too long and past the planes may be refused as either
    both = (jobs["qlen"] > 260) | (jobs["tlen"] > 400)
    np.testing.assert_array_equal(got[1][~both], want[1][~both])
    assert ((got[1] != 0) == (want[1] != 0)).all()
    for a, b in zip(got[:1] + got[2:4], want[:1] + want[2:4]):
        np.testing.assert_array_equal(a, b)


def negative_band_results(jobs):
    """What the row loop gives a band below 0: an empty row 0 from column -w on, which ends the job; a
    to-end score of 0 when that column is the query's end.  Returns (ext[n, 6], rows[n])."""
    ran = jobs["tlen"] > 0
    ends = ran & (jobs["qlen"] == -jobs["w"].astype(np.int64))
    out = np.zeros((len(jobs), 6), np.int32)
    out[:, 0], out[:, 3], out[:, 4] = jobs["h0"], ends, np.where(ends, 0, -1)
    return out, ran.astype(np.int32)


def test_negative_band_rule_matches_oracle():
    """(the oracle, like the reference, writes before its row for bands below -1)"""
    u8, jobs = edge_jobs(2000, 3, 40)
    jobs["w"] = -1
    ref, cells, rows = nat.oracle_extend(jobs, u8, g.default_score())
    want, want_rows = negative_band_results(jobs)
    np.testing.assert_array_equal(want, ref)
    np.testing.assert_array_equal(want_rows, rows)
    assert (cells == 0).all() and (want[:, 4] == 0).any()


@pytest.mark.parametrize("kernel,n", [(k, n) for k in (g.KERNEL_AUTO, g.KERNEL_ROWPAR, g.KERNEL_BAND) for n in (63, 4096, 9000)]
                         + [(g.KERNEL_AUTO, 40000)])
def test_negative_bands(n, kernel):
    """Negative bands among others, queries that end where such a band's row 0 begins and empty queries
    among them: in the group kernel as they are listed and sorted, the row-parallel and the band
    kernel, and the lane classes (40,000), whose sort keys hold the width of the widest row."""
    u8, jobs = edge_jobs(n, 23 + n, 40)
    rng = np.random.default_rng(n)
    neg = rng.random(n) < 0.3
    to_end = -np.maximum(jobs["qlen"].astype(np.int32), 1)
    jobs["w"][neg] = np.where(rng.random(n) < 0.5, to_end, rng.choice([-1, -2, -30, -60000], n))[neg]
    want, want_rows = negative_band_results(jobs)
    assert (want[neg, 4] == 0).any()
    sc = g.default_score()
    out, status, cells, rows, _ = run(u8, jobs, sc, kernel=kernel)
    assert (status == 0).all()
    np.testing.assert_array_equal(out[neg], want[neg])
    np.testing.assert_array_equal(rows[neg], want_rows[neg])
    assert (cells[neg] == 0).all()
    ref, ref_cells, ref_rows = nat.oracle_extend(jobs[~neg], u8, sc)
    np.testing.assert_array_equal(out[~neg], ref)
    np.testing.assert_array_equal(rows[~neg], ref_rows)
    np.testing.assert_array_equal(cells[~neg], ref_cells)


@pytest.mark.parametrize("kind,units", [(2, 3000), (4, 400)])
def test_autotuned_classes_run_as_the_same_classes_set(kind, units):
    """g3x_autotune's table in its context and handed to another through g3x_set_tiles: the same jobs per
    class, the same results; and a context without either sorts the batch into the groups' classes."""
    import torch
    wl = g.synth(kind, units, seed=9, w=60, unrelated=0.2 if kind == 2 else 0.0)
    codes, nmask = wl.planes()
    d = to_dev(wl.jobs), wl.n, to_dev(codes), to_dev(nmask)
    mq, mt = int(wl.jobs["qlen"].max()), int(wl.jobs["tlen"].max())
    sc = g.default_score()
    ref, _, _ = nat.oracle_extend(wl.jobs, wl.u8, sc)
    tuned, same, plain = g.Context(0), g.Context(0), g.Context(0)
    same.set_tiles(tuned.autotune(sc, *d, mq, mt))
    jobs = []
    for c in (tuned, same, plain):
        out = torch.zeros((wl.n, 6), dtype=torch.int32, device="cuda")
        status = torch.full((wl.n,), 9, dtype=torch.int32, device="cuda")
        c.extend_batch(sc, *d, out, status, mq, mt, schedule=g.SCHED_SORTED)
        torch.cuda.synchronize()
        assert (status.cpu().numpy() == 0).all()
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
        jobs.append([k for _, k in c.class_times()])
    for c in (tuned, same, plain):
        c.close()
    assert jobs[0] == jobs[1] and sum(jobs[0]) == wl.n
    if kind == 2:
        assert jobs[2] != jobs[0]


@pytest.mark.parametrize("units,w", [(700, 100), (9000, 100), (60000, 100), (15000, 10), (60000, 10)])
def test_counters_of_seed_calls(units, w):
    """A seed-level call's waves add to the context's occupancy counters in groups too (direct and
    sorted), as in the lane classes, which take narrow bands from fewer seeds on."""
    import torch
    wl = g.synth(2, units, seed=3, w=w, unrelated=0.2)
    codes, nmask = wl.planes()
    ds = g.device_seeds(wl.seeds)
    regs = torch.zeros(len(ds) * g.REG_DT.itemsize, dtype=torch.uint8, device="cuda")
    status = torch.zeros(len(ds), dtype=torch.int32, device="cuda")
    _, _, rows = nat.oracle_extend(wl.jobs, wl.u8, g.default_score())
    c = g.Context(0)
    c.extend_seeds(g.default_opt(w=w), to_dev(ds), len(ds), to_dev(codes), to_dev(nmask), regs, status,
                   int(wl.seeds["l_query"].max()), int((wl.seeds["rmax1"] - wl.seeds["rmax0"]).max()))
    torch.cuda.synchronize()
    got = c.last_stats()[0]
    c.close()
    # the left and right extensions are the workload's jobs, but for the right ones' seed scores; the
    # lane kernels count a row's blocks (three and more at w = 10)
    lanes = (units, w) == (60000, 10)
    assert rows.sum() * (2 if lanes else 0.5) < got < rows.sum() * (8 if lanes else 1.5)
