"""Resident passes against the per-step kernels bit for bit: recorded seismograms, images, and every field
after either pass, in float and double, on blocks of one, two and more columns a thread
(tests/resident_wait.cu holds these grids to those kinds), with the shot and the receivers beside each
corner of the grid in turn so that waves cross all four strips and their corners."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [
    # nx, nz, (left, right, up, down), nt, slices, other parameters
    (96, 64, (16, 16, 16, 16), 120, 4, {}),
    (97, 61, (17, 21, 14, 19), 120, 2, dict(storage=0)),
    (400, 200, (40, 40, 40, 40), 80, 4, {}),
    (901, 301, (40, 40, 40, 40), 60, 4, {}),
    (901, 301, (41, 37, 30, 45), 60, 4, dict(storage=0)),
    (1201, 403, (40, 40, 40, 40), 60, 4, {}),
    (1201, 403, (41, 37, 30, 45), 60, 4, dict(storage=0)),
    (3400, 700, (50, 50, 50, 50), 80, 4, {}),
    (150, 90, (20, 20, 20, 20), 120, 4, dict(compute=1)),
    (1000, 300, (40, 40, 40, 40), 60, 4, dict(compute=1)),
    (1000, 300, (41, 37, 30, 45), 60, 4, dict(compute=1, storage=0)),
    (1201, 403, (41, 37, 30, 45), 80, 4, dict(precision=1)),
    (901, 301, (40, 40, 40, 40), 60, 2, dict(precision=2, storage=0)),
]


def _outputs(eng, torch, p, vel, wav, seis):
    real = torch.float64 if p.compute == 1 else torch.float32
    plan, out = eng.Plan(p), {}
    out["seismogram"] = torch.zeros((p.rec_count, p.nt), device="cuda", dtype=real)
    plan.forward(vel, wav, out["seismogram"])
    plan.sync()
    launches = plan.launches

    def fields(when, ids):
        for k in ids:
            out["%s %d" % (when, k)] = torch.empty((p.dim_x, p.dim_z), device="cuda", dtype=real)
            plan.read_field(k, out["%s %d" % (when, k)])

    fields("forward", (0, 1))
    plan.adjoint(seis)
    for k in (0, 1):
        out["image %d" % k] = torch.empty((p.nx, p.nz), device="cuda", dtype=torch.float64)
        plan.read_image(k, out["image %d" % k], True)
    fields("adjoint", (2,))
    plan.sync()
    plan.close()
    return launches, {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("corner", ("top left", "bottom right"))
@pytest.mark.parametrize("case", range(len(GRIDS)))
def test_resident_pass_equals_step_kernels(engine, case, corner):
    import torch
    from rtmuq2d_gb300 import workloads
    nx, nz, th, nt, slices, kw = GRIDS[case]
    far = corner == "bottom right"
    p = workloads.params_tiny(nx=nx, nz=nz, th=16, nt=nt, time_slices=slices, n_wavelet=30)
    p = p.replace(th_left=th[0], th_right=th[1], th_up=th[2], th_down=th[3], shot_x=nx - 3 if far else 2,
                  shot_z=nz - 3 if far else 2, rec_depth=nz - 2 if far else 1, **kw)
    rng = np.random.default_rng(100 + case)
    ext = engine.extend_matrix(p, (1600 + 800 * rng.random((nx, nz))).astype(np.float32))
    vel = torch.from_numpy(ext).cuda()
    wav = torch.from_numpy(workloads.wavelet_for(p, 60.0)).cuda()
    seis = torch.from_numpy((0.1 * rng.standard_normal((p.rec_count, nt))).astype(np.float32)).cuda()
    n_res, a = _outputs(engine, torch, p, vel, wav, seis)
    n_step, b = _outputs(engine, torch, p.replace(tile_x=16), vel, wav, seis)   # the tiles the 16-bit scales belong to
    assert n_res < 12 and n_step >= nt
    u = b["forward 0"]
    w = 4 + 4
    assert np.abs(u[-w:, -w:] if far else u[:w, :w]).max() > 0        # the waves reached the corner of the strips
    for k, y in b.items():
        assert np.abs(y).max() > 0, k
        assert np.array_equal(a[k], y), (k, float(np.abs(a[k].astype(np.float64) - y).max()))


def test_members_of_one_launch_equal_their_own(engine):
    """A launch takes the kernel of its widest member: members of one and two columns a thread beside one of
    more (whose kernel keeps the values elsewhere and rounds by rule, not by the compiler's choice) return
    what each returns by itself."""
    from rtmuq2d_gb300 import workloads
    requests = []
    for k, (nx, nz, th) in enumerate(((96, 64, 16), (400, 200, 40), (1201, 403, 40), (333, 141, 30), (97, 61, 17))):
        p = workloads.params_tiny(nx=nx, nz=nz, th=th, nt=120, time_slices=4, n_wavelet=30)
        rng = np.random.default_rng(k)
        ext = engine.extend_matrix(p, (1600 + 800 * rng.random((nx, nz))).astype(np.float32))
        requests.append((p, ext, workloads.wavelet_for(p, 60.0),
                         (0.1 * rng.standard_normal((p.rec_count, p.nt))).astype(np.float32)))
    srv = engine.Server(0, max_members=8, steps_per_launch=16)
    ids = [srv.submit(*r) for r in requests]
    out = srv.run_all()
    srv.close()
    for i, r in zip(ids, requests):
        want = engine.migrate_shot(*r)
        assert np.abs(want[0]).max() > 0
        assert np.array_equal(out[i][0], want[0]) and np.array_equal(out[i][1], want[1])


@pytest.mark.parametrize("kw", ({}, dict(precision=1)))
def test_resident_forward_with_an_adjoint_by_steps(engine, kw):
    """3600 x 700 with rings: the forward pass fits the chip, the adjoint with its two fields does not."""
    import torch
    from rtmuq2d_gb300 import workloads
    p = workloads.params_tiny(nx=3600, nz=700, th=50, nt=80, time_slices=4, n_wavelet=30).replace(**kw)
    rng = np.random.default_rng(9)
    ext = engine.extend_matrix(p, (1600 + 800 * rng.random((p.nx, p.nz))).astype(np.float32))
    vel = torch.from_numpy(ext).cuda()
    wav = torch.from_numpy(workloads.wavelet_for(p, 60.0)).cuda()
    seis = torch.from_numpy((0.1 * rng.standard_normal((p.rec_count, p.nt))).astype(np.float32)).cuda()
    plan = engine.Plan(p)
    plan.forward(vel, wav)
    forward = plan.launches
    plan.adjoint(seis)
    plan.sync()
    assert forward < 12 and plan.launches - forward >= p.nt
    plan.close()
    _, a = _outputs(engine, torch, p, vel, wav, seis)
    _, b = _outputs(engine, torch, p.replace(tile_x=16), vel, wav, seis)
    for k, y in b.items():
        assert np.abs(y).max() > 0 and np.array_equal(a[k], y), k
