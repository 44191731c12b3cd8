"""Passes on the chip of several plans at once: each on its stream and thread, they run side by side on parts
of the chip, and each image equals the plan's own on the whole chip bit for bit."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _job(engine, torch, nx, nz, th, nt, slices, seed, **kw):
    from rtmuq2d_gb300 import workloads
    p = workloads.params_tiny(nx=nx, nz=nz, th=th, nt=nt, time_slices=slices, n_wavelet=30).replace(**kw)
    rng = np.random.default_rng(seed)
    ext = engine.extend_matrix(p, (1600 + 800 * rng.random((nx, nz))).astype(np.float32))
    vel, wav = torch.from_numpy(ext).cuda(), torch.from_numpy(workloads.wavelet_for(p, 60.0)).cuda()
    seis = torch.from_numpy((0.1 * rng.standard_normal((p.rec_count, nt))).astype(np.float32)).cuda()
    out = [torch.zeros((nx, nz), device="cuda", dtype=torch.float64) for _ in range(2)]
    return engine.Plan(p), vel, wav, seis, out


def _shot(j):
    plan, vel, wav, seis, out = j
    plan.forward(vel, wav)
    plan.adjoint(seis)
    plan.read_image(0, out[0], True)
    plan.read_image(1, out[1], True)
    plan.sync()


def _together(jobs, shots, check=None):
    errors = []

    def work(j, want):
        import torch
        torch.cuda.set_device(0)
        try:
            for _ in range(shots):
                if want is not None:
                    for o in j[4]:
                        o.zero_()
                    torch.cuda.current_stream().synchronize()
                _shot(j)
                if want is not None:
                    assert all(torch.equal(a, b) for a, b in zip(j[4], want))
        except Exception as e:          # noqa: BLE001 -- a thread's failure is the test's
            errors.append(e)

    threads = [threading.Thread(target=work, args=(j, check[k] if check else None)) for k, j in enumerate(jobs)]
    t = time.perf_counter()
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not errors, errors
    return time.perf_counter() - t


def test_plans_share_the_chip_with_the_same_images(engine):
    """Grids and options that take 1 to 12 columns a thread at a half to an eighth of the chip, together with
    one that has no part smaller than the whole."""
    import torch
    jobs = [_job(engine, torch, 96, 64, 16, 400, 4, 0), _job(engine, torch, 400, 200, 40, 200, 4, 1),
            _job(engine, torch, 401, 203, 41, 200, 4, 2, storage=0), _job(engine, torch, 700, 300, 40, 160, 4, 3),
            _job(engine, torch, 1201, 403, 40, 100, 4, 4, precision=1), _job(engine, torch, 333, 141, 30, 200, 4, 5, precision=2, storage=0),
            _job(engine, torch, 150, 90, 20, 200, 4, 6, compute=1), _job(engine, torch, 2600, 600, 50, 40, 4, 7)]
    want = []
    for j in jobs:
        _shot(j)
        want.append([o.clone() for o in j[4]])
        assert float(want[-1][0].abs().max()) > 0
    _together(jobs, 8, want)
    for j in jobs:
        j[0].close()


def test_small_plans_do_not_queue_for_the_whole_chip(engine):
    """Eight small plans on eight streams take less than three quarters of eight times one's time: in turn they
    took all of it, side by side 2.3 (96 x 64) and 4.0 times one's."""
    import torch
    for nx, nz, th, nt in ((96, 64, 16, 2000), (400, 200, 40, 1000)):
        jobs = [_job(engine, torch, nx, nz, th, nt, 20, k) for k in range(8)]
        for j in jobs:
            _shot(j)
        alone = min(_together(jobs[:1], 6) for _ in range(3))
        all_ = min(_together(jobs, 6) for _ in range(3))
        assert all_ < 0.75 * 8 * alone, (alone, all_)
        for j in jobs:
            j[0].close()


def test_pass_beside_a_capture_leaves_it_valid(engine):
    """A pass on one stream, with another in flight, while this thread captures a third in global mode."""
    import torch
    a, b = _job(engine, torch, 400, 200, 40, 200, 4, 1), _job(engine, torch, 96, 64, 16, 200, 4, 2)
    for j in (a, b):
        _shot(j)
    want = [o.clone() for o in b[4]]
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    a[0].forward(a[1], a[2])
    with torch.cuda.graph(graph):
        x += 1
        b[0].forward(b[1], b[2])
        x += 1
    b[0].adjoint(b[3])
    b[0].read_image(0, b[4][0], True)
    b[0].sync()
    a[0].sync()
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 2.0 and torch.equal(b[4][0], want[0])
    for j in (a, b):
        j[0].close()
