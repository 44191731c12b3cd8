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
