"""Resident passes (k_resident) against the per-step kernels (a plan with tile_x set) on the same
inputs: the same arithmetic in the same order, so the fields after a pass stay within 1e-5 and the
images within 1e-4 (FP64: 1e-10, 1e-8) of each other -- the bars both hold against the oracle -- at
sizes where a block or a strip can go wrong: odd grids, a CPML different on every side, strips wider
than the model, one-column models, blocks of one, two and more columns a thread."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # nx, nz, (left, right, up, down), nt, slices, other parameters
    (96, 64, (16, 16, 16, 16), 60, 4, {}),
    (97, 61, (17, 21, 14, 19), 60, 4, {}),
    (97, 61, (17, 21, 14, 19), 60, 4, dict(storage=0)),
    (1, 4, (12, 12, 12, 12), 40, 2, dict(rec_count=1, shot_x=0, shot_z=1)),
    (700, 33, (60, 12, 13, 64), 40, 1, {}),
    (33, 600, (12, 60, 64, 13), 40, 2, dict(rec_spacing=1, rec_count=5)),
    (500, 303, (30, 31, 32, 33), 40, 2, {}),
    (1201, 403, (41, 37, 30, 45), 40, 20, {}),
    (3400, 700, (50, 50, 50, 50), 20, 4, {}),
    (1777, 555, (23, 57, 36, 41), 20, 4, dict(storage=0)),
    (150, 90, (33, 20, 25, 40), 40, 4, dict(compute=1)),
    (150, 90, (33, 20, 25, 40), 40, 4, dict(compute=1, storage=0)),
    (601, 203, (33, 20, 25, 40), 20, 4, dict(compute=1)),
    # 16-bit storage: more steps than a staged run, runs that do not divide nt, every kind of group
    (97, 61, (17, 21, 14, 19), 150, 2, dict(precision=1)),
    (500, 303, (30, 31, 32, 33), 70, 2, dict(precision=2)),
    (97, 61, (17, 21, 14, 19), 60, 4, dict(storage=0, precision=2)),
    (901, 301, (40, 40, 40, 40), 120, 2, dict(storage=0, precision=1)),
]


def _run(eng, torch, p, vel, wav, seis):
    real = torch.float64 if p.compute == 1 else torch.float32
    plan, out = eng.Plan(p), {}
    rec = torch.zeros((max(1, p.rec_count), p.nt), device="cuda", dtype=real)
    plan.forward(vel, wav, rec)
    plan.sync()
    launches = plan.launches
    out["seismogram"] = rec
    for k in (0, 1):
        out["u%d" % k] = torch.empty((p.dim_x, p.dim_z), device="cuda", dtype=real)
        plan.read_field(k, out["u%d" % k])
    plan.adjoint(seis)
    for k in (0, 1):
        out["image%d" % k] = torch.empty((p.nx, p.nz), device="cuda", dtype=torch.float64)
        plan.read_image(k, out["image%d" % k], True)
    out["receiver"] = torch.empty((p.dim_x, p.dim_z), device="cuda", dtype=real)
    plan.read_field(2, out["receiver"])
    plan.sync()
    plan.close()
    return launches, {k: v.cpu().numpy().astype(np.float64) for k, v in out.items()}


@pytest.mark.parametrize("case", range(len(CASES)))
def test_resident_pass_matches_step_kernels(engine, case):
    import torch
    from rtmuq2d_gb300 import workloads
    nx, nz, th, nt, slices, kw = CASES[case]
    p = workloads.params_tiny(nx=nx, nz=nz, th=16, nt=nt, time_slices=slices, n_wavelet=30)
    p = p.replace(th_left=th[0], th_right=th[1], th_up=th[2], th_down=th[3], **kw)
    rng = np.random.default_rng(case)
    ext = engine.extend_matrix(p, (1600 + 800 * rng.random((nx, nz))).astype(np.float32))
    vel = torch.from_numpy(ext).cuda()
    wav = torch.from_numpy(workloads.wavelet_for(p, 60.0)).cuda()
    seis = torch.from_numpy((0.1 * rng.standard_normal((p.rec_count, nt))).astype(np.float32)).cuda()
    n_res, a = _run(engine, torch, p, vel, wav, seis)
    # 16 columns: the default tile, whose groups the 16-bit scales of both plans belong to
    n_step, b = _run(engine, torch, p.replace(tile_x=16), vel, wav, seis)
    assert n_res < 12 and n_step >= nt          # a few launches for the pass, one a step
    for k, y in b.items():
        tol = (1e-8 if k.startswith("image") else 1e-10) if p.compute == 1 else (1e-4 if k.startswith("image") else 1e-5)
        assert np.linalg.norm(a[k] - y) <= tol * np.linalg.norm(y), k


def test_resident_plans_on_two_threads_and_streams(engine):
    """Two plans, each on its own stream and thread, repeat their solo results bit for bit: their
    cooperative launches run one after the other on the device."""
    import threading
    import torch
    from rtmuq2d_gb300 import workloads
    jobs, want, got = [], [], [[], []]
    for k, (nx, nz) in enumerate(((180, 90), (333, 141))):
        p = workloads.params_tiny(nx=nx, nz=nz, th=16, nt=80, time_slices=4)
        rng = np.random.default_rng(k)
        ext = engine.extend_matrix(p, (1600 + 800 * rng.random((nx, nz))).astype(np.float32))
        wav = workloads.wavelet_for(p, 60.0)
        seis = (0.1 * rng.standard_normal((p.rec_count, p.nt))).astype(np.float32)
        jobs.append((p, ext, wav, seis))
        want.append(engine.migrate_shot(*jobs[-1]))

    def work(k):
        p, ext, wav, seis = jobs[k]
        torch.cuda.set_device(0)
        for _ in range(6):
            got[k].append(engine.migrate_shot(p, ext, wav, seis))

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert len(got[k]) == 6
        for img, slf in got[k]:
            assert np.array_equal(img, want[k][0]) and np.array_equal(slf, want[k][1])


def test_capturing_stream_keeps_the_step_kernels(engine):
    """A forward pass with recording on a stream under capture stays a sequence of capturable
    launches, and its replay gives the resident pass's seismogram."""
    import torch
    from rtmuq2d_gb300 import workloads
    p = workloads.params_tiny(nx=120, nz=70, th=16, nt=40, time_slices=4)
    rng = np.random.default_rng(5)
    ext = engine.extend_matrix(p, (1600 + 800 * rng.random((p.nx, p.nz))).astype(np.float32))
    vel, wav = torch.from_numpy(ext).cuda(), torch.from_numpy(workloads.wavelet_for(p, 60.0)).cuda()
    plan = engine.Plan(p)
    want = torch.zeros((p.rec_count, p.nt), device="cuda")
    plan.forward(vel, wav, want)
    plan.sync()
    stream = torch.cuda.Stream()
    plan.set_stream(stream.cuda_stream)
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        plan.forward(vel, wav, out)
    graph.replay()
    torch.cuda.synchronize()
    assert float(want.abs().max()) > 0
    assert float((out - want).norm()) <= 1e-5 * float(want.norm())


@pytest.mark.parametrize("steps_per_launch", (16, 7))
def test_server_members_resident_and_batched_agree(engine, steps_per_launch):
    """A server's resident members (small ones sharing a launch, 16-bit stores packed by strip block
    or tile) against the batched kernels (tile_x = 32): within 1e-5, the bar of the batched engine."""
    from rtmuq2d_gb300 import workloads
    grids = [(97, 61, (17, 21, 14, 19), 60, 4, {}), (200, 100, (40, 40, 40, 40), 60, 20, dict(precision=1)),
             (640, 303, (41, 37, 30, 45), 40, 20, {}), (97, 61, (17, 21, 14, 19), 50, 5, dict(storage=0, precision=2)),
             (300, 133, (60, 12, 13, 64), 49, 7, dict(precision=2)), (301, 150, (33, 20, 25, 40), 60, 4, dict(storage=0)),
             (1500, 500, (50, 50, 50, 50), 40, 20, dict(precision=1)), (120, 80, (16, 16, 16, 16), 33, 1, {})]
    requests = []
    for k, (nx, nz, th, nt, slices, kw) in enumerate(grids):
        p = workloads.params_tiny(nx=nx, nz=nz, th=16, nt=nt, time_slices=slices)
        p = p.replace(th_left=th[0], th_right=th[1], th_up=th[2], th_down=th[3], **kw)
        rng = np.random.default_rng(k)
        ext = engine.extend_matrix(p, (1600 + 800 * rng.random((nx, nz))).astype(np.float32))
        requests.append((p, ext, workloads.wavelet_for(p, 60.0),
                         (0.1 * rng.standard_normal((p.rec_count, nt))).astype(np.float32)))
    results = []
    for tile_x in (0, 32):
        srv = engine.Server(0, max_members=16, steps_per_launch=steps_per_launch)
        ids = [srv.submit(r[0].replace(tile_x=tile_x), *r[1:]) for r in requests]
        out = srv.run_all()
        srv.close()
        results.append([out[i][:2] for i in ids])
    for k, (a, b) in enumerate(zip(*results)):
        for x, y in zip(a, b):
            assert np.linalg.norm(x.astype(np.float64) - y) <= 1e-5 * np.linalg.norm(y), k
