"""Passes cut into short resident launches: a server whose launches run a step or a few of a pass each
returns the images of the uncut pass bit for bit, whatever blocks and neighbours the cuts meet."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _request(engine, nx, nz, th, nt, slices, seed, **kw):
    from rtmuq2d_gb300 import workloads
    p = workloads.params_tiny(nx=nx, nz=nz, th=16, nt=nt, time_slices=slices, n_wavelet=30)
    p = p.replace(th_left=th[0], th_right=th[1], th_up=th[2], th_down=th[3], **kw)
    rng = np.random.default_rng(seed)
    ext = engine.extend_matrix(p, (1600 + 800 * rng.random((nx, nz))).astype(np.float32))
    return (p, ext, workloads.wavelet_for(p, 60.0),
            (0.1 * rng.standard_normal((p.rec_count, nt))).astype(np.float32))


def _serve(engine, requests, steps_per_launch):
    srv = engine.Server(0, max_members=16, steps_per_launch=steps_per_launch)
    ids = [srv.submit(*r) for r in requests]
    out = srv.run_all()
    srv.close()
    return [out[i][:2] for i in ids]


# Strips that span several blocks along both axes, blocks of one, two and more columns a thread.
RUNS = [
    (97, 61, (17, 21, 14, 19), 61, 1, {}),
    (400, 200, (40, 40, 40, 40), 40, 4, {}),
    (700, 33, (60, 12, 13, 64), 40, 1, dict(storage=0)),
    (333, 600, (64, 60, 64, 45), 24, 2, {}),
    (1201, 403, (41, 37, 30, 45), 24, 4, {}),
]


@pytest.mark.parametrize("steps_per_launch", (1, 2, 3))
@pytest.mark.parametrize("case", range(len(RUNS)))
def test_launches_of_a_step_or_a_few(engine, case, steps_per_launch):
    nx, nz, th, nt, slices, kw = RUNS[case]
    r = _request(engine, nx, nz, th, nt, slices, case, **kw)
    (img, slf), = _serve(engine, [r], steps_per_launch)
    want = engine.migrate_shot(*r)
    assert np.abs(want[0]).max() > 0
    assert np.array_equal(img, want[0]) and np.array_equal(slf, want[1])


def test_members_share_the_steps_at_large_launches(engine):
    """Three members that fill the chip, 256 steps a launch: they finish within a few server steps of one
    another, each with the image of its own uncut migration."""
    rs = [_request(engine, 2600, 600, (50, 50, 50, 50), 4000, 40, k) for k in range(3)]
    srv = engine.Server(0, max_members=8, steps_per_launch=256)
    ids = [srv.submit(*r) for r in rs]
    done, at, step = {}, {}, 0
    while len(done) < len(ids):
        srv.step()
        step += 1
        assert step < 60
        while (r := srv.poll()) is not None:
            done[r[0]], at[r[0]] = r[1:3], step
    srv.close()
    # two of the three waves run at a server step, so a turn takes two; admissions may lie two steps apart
    assert max(at.values()) - min(at.values()) <= 4, at
    for i, r in zip(ids, rs):
        want = engine.migrate_shot(*r)
        assert np.array_equal(done[i][0], want[0]) and np.array_equal(done[i][1], want[1])


def _peak_serve(engine, requests, budget, steps_per_launch=64):
    """Results, the most bytes the server said it held and the most device memory it took."""
    import torch
    torch.cuda.synchronize()
    free, held, taken = torch.cuda.mem_get_info()[0], 0, 0
    srv = engine.Server(budget, max_members=8, steps_per_launch=steps_per_launch)
    base = free - torch.cuda.mem_get_info()[0]             # what every server takes, of any budget
    ids, out, steps = [srv.submit(*r) for r in requests], {}, 0
    while len(out) < len(ids):
        srv.step()
        steps += 1
        assert steps < 20000
        held = max(held, srv.stats()["bytes_in_use"])
        taken = max(taken, free - torch.cuda.mem_get_info()[0] - base)
        while (r := srv.poll()) is not None:
            out[r[0]] = r[1:3]
    srv.close()
    return [out[i] for i in ids], held, taken


@pytest.mark.parametrize("storage", (0, 1))
def test_sixteen_bit_members_stay_within_the_budget(engine, storage):
    """16-bit members whose launches would stage far more than the budget leaves: shorter runs of steps, the
    device memory within the budget, and the images of a server with all the room, bit for bit."""
    rs = [_request(engine, 800, 300, (40, 40, 40, 40), 256, 1, k, storage=storage, precision=1 + k % 2) for k in range(2)]
    want, _, _ = _peak_serve(engine, rs, 0, 256)
    fp = max(engine.footprint_bytes(r[0]) for r in rs)
    slack = 8 << 20                                        # allocations are rounded up to 2 MB pages
    for extra in (64 << 20, 34 << 20):
        got, held, taken = _peak_serve(engine, rs[:1], fp + extra, 256)
        assert held <= fp + extra and taken <= fp + extra + slack, (held, taken, fp + extra)
        assert np.array_equal(got[0][0], want[0][0]) and np.array_equal(got[0][1], want[0][1])


def test_members_without_room_for_resident_launches(engine):
    """A budget that holds a member but not what its resident launches need: the member still runs, and a
    large request is admitted after resident members although their buffers were in its way."""
    small = _request(engine, 200, 100, (40, 40, 40, 40), 60, 4, 1)
    big = _request(engine, 900, 400, (40, 40, 40, 40), 400, 4, 2, storage=0)
    fps, fpb = engine.footprint_bytes(small[0]), engine.footprint_bytes(big[0])
    assert fpb > (40 << 20) + fps
    (got,), held, _ = _peak_serve(engine, [small], fps + (64 << 10))
    assert held <= fps + (64 << 10)
    want = engine.migrate_shot(*small)
    assert np.linalg.norm(got[0].astype(np.float64) - want[0]) <= 1e-5 * np.linalg.norm(want[0])
    (a, b, c), held, _ = _peak_serve(engine, [small, big, small], fpb + (64 << 10))
    assert held <= fpb + (64 << 10)
    assert np.array_equal(a[0], want[0]) and np.array_equal(c[0], want[0])
    want = engine.migrate_shot(*big)
    assert np.linalg.norm(b[0].astype(np.float64) - want[0]) <= 1e-5 * np.linalg.norm(want[0])


@pytest.mark.parametrize("kw", ({}, dict(storage=0, precision=2), dict(precision=1), dict(compute=1), dict(tile_x=16)))
def test_plan_bytes_are_what_it_takes(engine, kw):
    """A plan's bytes against the device memory that plans of it take: the footprint, and with passes on the
    chip (no tile width forced) their mailboxes, tables and staging."""
    import torch
    from rtmuq2d_gb300 import workloads
    p = workloads.params_tiny(nx=1201, nz=403, th=40, nt=400, time_slices=4).replace(**kw)
    engine.Plan(p).close()                                 # what the process loads once
    free = torch.cuda.mem_get_info()[0]
    plans = [engine.Plan(p) for _ in range(3)]
    taken = free - torch.cuda.mem_get_info()[0]
    said = sum(plan.nbytes for plan in plans)
    for plan in plans:
        plan.close()
    fp = engine.footprint_bytes(p)
    assert (said == 3 * fp) == bool(kw.get("tile_x")) and said >= 3 * fp
    # two allocations a plan, each rounded up to 2 MB pages
    assert said <= taken + (2 << 20) and taken <= said + 3 * 2 * (2 << 20) + (2 << 20)


def test_more_snapshots_than_a_grid_has_rows(engine):
    """16-bit snapshots of more steps than the 65535 blocks of a launch's second dimension, staged at once."""
    nt = 66000
    p, vel, wav, seis = _request(engine, 1, 4, (12, 12, 12, 12), nt, 1, 3, storage=0, precision=2, rec_count=1,
                                 shot_x=0, shot_z=1)
    got = engine.migrate_shot(p, vel, wav, seis)
    want = engine.migrate_shot(p.replace(tile_x=16), vel, wav, seis)
    assert np.abs(want[0]).max() > 0
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("steps_per_launch", (3, 16))
def test_more_members_than_run_at_a_step(engine, steps_per_launch):
    """Eleven members that fill the chip and six small ones: two or more of the waves run at a server step, and
    every image equals the member's own."""
    rs = [_request(engine, 2600, 600, (50, 50, 50, 50), 40, 4, k % 3, precision=0) for k in range(11)]
    rs += [_request(engine, 96 + 7 * k, 64, (16, 16, 16, 16), 60 + 20 * k, 4, 20 + k, storage=k % 2) for k in range(6)]
    srv = engine.Server(0, max_members=32, steps_per_launch=steps_per_launch)
    ids = [srv.submit(*r) for r in rs]
    out = srv.run_all()
    srv.close()
    want = {}
    for k, r in enumerate(rs):
        key = k % 3 if k < 11 else k
        if key not in want:
            want[key] = engine.migrate_shot(*r)
        assert np.array_equal(out[ids[k]][0], want[key][0]) and np.array_equal(out[ids[k]][1], want[key][1]), k
