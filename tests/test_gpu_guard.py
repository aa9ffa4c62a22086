"""Failure detection during propagation: the wavefield watchdog and the
stability checks of the reference's set-up code.

Divergence is made on the host side of the physics, never by a fault: a
pseudo-acoustic VTI medium with delta > epsilon is unstable (in the
reference as much as here) and overflows to Inf within a few hundred
steps.  The watchdog sees it at its next scan, the run stops queueing
steps and returns GEO_ERR_NAN; the context stays usable."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEO_ERR_CFL, GEO_ERR_NAN = 5, 8


def _unstable3d(n=24):
    v = np.full((n, n, n), 2500.0, np.float32)
    return v, np.zeros_like(v), np.full_like(v, 0.4)


def _step_of(err):
    m = re.search(r"by time step (\d+)", str(err))
    return int(m.group(1)) if m else None


KW3 = dict(npd=8, dx=10.0, dy=10.0, dz=10.0, dt=np.float32(1e-3), favg=25.0, pfac=10.0, fsx=12, fsy=12, fsz=3)


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_fd3d_watchdog_stops_a_diverging_shot(geo, mode):
    v, e, d = _unstable3d()
    with pytest.raises(geo.GeoError) as ei:
        geo.fd3d_shot(v, e, d, nt=2000, mode=mode, **KW3)
    assert ei.value.status == GEO_ERR_NAN, str(ei.value)
    assert _step_of(ei.value) in (100, 200, 300), str(ei.value)
    # the context and the library still compute correctly afterwards
    from tests.util import random_model_3d
    vs, es, ds = random_model_3d(24, 24, 24, seed=1)
    out = geo.fd3d_shot(vs, es, ds, nt=150, mode=mode, **KW3)
    assert np.isfinite(out).all() and np.abs(out).max() > 0


def test_fd3d_watchdog_interval_and_off(geo, monkeypatch):
    v, e, d = _unstable3d()
    monkeypatch.setenv("GEO_WATCH_EVERY", "50")
    with pytest.raises(geo.GeoError) as ei:
        geo.fd3d_shot(v, e, d, nt=1000, mode="fast", **KW3)
    assert ei.value.status == GEO_ERR_NAN and _step_of(ei.value) % 50 == 0
    # off: the run completes as the reference's would, with non-finite values
    monkeypatch.setenv("GEO_WATCH_EVERY", "0")
    out = geo.fd3d_shot(v, e, d, nt=600, mode="fast", **KW3)
    assert not np.isfinite(out).all()


def test_fd3d_watchdog_checks_the_last_step(geo):
    """nt not a multiple of the interval: the last step is scanned too."""
    v, e, d = _unstable3d()
    with pytest.raises(geo.GeoError) as ei:
        geo.fd3d_shot(v, e, d, nt=399, mode="fast", **KW3)
    assert ei.value.status == GEO_ERR_NAN


def test_rtm3d_watchdog(geo):
    v, e, d = _unstable3d(20)
    kw = dict(KW3, fsx=10, fsy=10)
    with pytest.raises(geo.GeoError) as ei:
        geo.rtm3d(v, e, d, nt=700, method="boundary", **kw)
    assert ei.value.status == GEO_ERR_NAN


def _unstable2d(nx=48, nz=48):
    v = np.full((nx, nz), 2500.0, np.float32)
    return v, np.zeros_like(v), np.full_like(v, 0.4)


KW2 = dict(npd=10, dx=10.0, dz=10.0, dt=np.float32(1e-3), favg=20.0, pfac=10.0, fs=24.0, zs=5.0)


@pytest.mark.parametrize("variant", ["cpu", "gpu", "mpi"])
@pytest.mark.parametrize("snap_every", [0, 50])
def test_fd2d_watchdog(geo, variant, snap_every):
    v, e, d = _unstable2d()
    with pytest.raises(geo.GeoError) as ei:
        geo.fd2d_shot(v, e, d, nt=1200, variant=variant, snap_every=snap_every, **KW2)
    assert ei.value.status == GEO_ERR_NAN, str(ei.value)


def test_tti2d_watchdog(geo):
    v, e, d = _unstable2d()
    th = np.full_like(v, 20.0)
    with pytest.raises(geo.GeoError) as ei:
        geo.tti2d_shot(v, e, d, th, nt=1200, **KW2)
    assert ei.value.status == GEO_ERR_NAN


def test_rtm2d_batch_watchdog(geo):
    nx, nz = 121, 40
    v = np.full((nx, nz), 2500.0, np.float32)
    e, d = np.zeros_like(v), np.full_like(v, 0.4)
    with pytest.raises(geo.GeoError) as ei:
        geo.rtm2d_batch(v, e, d, npd=12, nt=900, dx=10.0, dz=10.0, dt_ms=1.0, favg=20.0, pfac=1000.0, zs=1,
                        shot_x=[41, 81], shot_nxs=[41, 51])
    assert ei.value.status == GEO_ERR_NAN, str(ei.value)
    assert "forward" in str(ei.value)


def test_rtm2d_gpu_watchdog(geo):
    v, e, d = _unstable2d(60, 40)
    with pytest.raises(geo.GeoError) as ei:
        geo.rtm2d_gpu(v, e, d, npml=15, nt=900, dx=10.0, dz=10.0, dt=np.float32(1e-3), favg=20.0, fs=30, zs=2)
    assert ei.value.status == GEO_ERR_NAN, str(ei.value)


def test_stability_condition_refused_everywhere(geo):
    """dt*vmax*sqrt(sum 1/d^2) >= 0.777 (the set-up code's limit for the
    8th-order operator) is refused with GEO_ERR_CFL before any step."""
    from tests.util import layered_model, random_model_3d
    v3, e3, d3 = random_model_3d(20, 20, 20, seed=2, vlo=2000, vhi=4500)
    with pytest.raises(geo.GeoError) as ei:       # 0.002*4500*sqrt(3)/10 = 1.56
        geo.fd3d_shot(v3, e3, d3, nt=20, **dict(KW3, dt=np.float32(2e-3), fsx=10, fsy=10))
    assert ei.value.status == GEO_ERR_CFL
    v, e, d = layered_model(50, 40, seed=1)        # vp up to 4000: 0.002*4000*sqrt(2)/10 = 1.13
    for variant in ("cpu", "gpu", "mpi"):
        with pytest.raises(geo.GeoError) as ei:
            geo.fd2d_shot(v, e, d, nt=20, variant=variant, **dict(KW2, dt=np.float32(2e-3)))
        assert ei.value.status == GEO_ERR_CFL
    with pytest.raises(geo.GeoError) as ei:
        geo.rtm2d_batch(v, e, d, npd=12, nt=20, dx=10.0, dz=10.0, dt_ms=2.0, favg=20.0, pfac=1000.0, zs=1,
                        shot_x=[25], shot_nxs=[21])
    assert ei.value.status == GEO_ERR_CFL
    with pytest.raises(geo.GeoError) as ei:
        geo.tti2d_shot(v, e, d, np.full_like(v, 10.0), nt=20, **dict(KW2, dt=np.float32(2e-3)))
    assert ei.value.status == GEO_ERR_CFL


def test_cpu_program_limits(geo):
    """CPU_vti2dfd's get_constant limits (spacing above vmin/favg*0.2, dt
    above 0.5*min(d)/vmax) are refused for the CPU form only: the program
    leaves its sponge constant undefined there; the GPU programs have no
    such check."""
    from tests.util import layered_model
    v, e, d = layered_model(50, 40, seed=1)        # vmin >= 2000: 2000/150*0.2 = 2.7 < 10
    with pytest.raises(geo.GeoError) as ei:
        geo.fd2d_shot(v, e, d, nt=20, variant="cpu", **dict(KW2, favg=150.0))
    assert ei.value.status == GEO_ERR_CFL
    out = geo.fd2d_shot(v, e, d, nt=20, variant="gpu", **dict(KW2, favg=150.0))
    assert np.isfinite(out).all()


@pytest.mark.parametrize("array,value,text", [(0, np.nan, "velocity[37]"), (0, -1.0, "velocity[37]"),
                                              (1, np.inf, "eps/del[37]"), (2, -0.6, "1+2*delta[37]"),
                                              (3, np.nan, "theta[37]")])
def test_2d_model_check_names_the_first_bad_cell(geo, array, value, text):
    """Every 2D entry point, host and device arrays: the first failing cell
    (a later one fails too) is reported and nothing runs."""
    import torch
    nx, nz = 21, 19
    m = [np.full((nx, nz), x, np.float32) for x in (2000.0, 0.1, 0.05, 20.0)]
    m[array].reshape(-1)[[37, 300]] = value
    kw = dict(nt=5, dx=10.0, dz=10.0, dt=np.float32(1e-3), favg=20.0)
    calls = [lambda a: geo.tti2d_shot(*a, npd=8, fs=10, zs=3, **kw), lambda a: geo.rtm2d_tti(*a, npml=8, fs=10, **kw)]
    if array < 3:
        calls += [lambda a: geo.fd2d_shot(*a[:3], npd=8, fs=10, zs=3, **kw),
                  lambda a: geo.rtm2d_gpu(*a[:3], npml=8, fs=10, **kw),
                  lambda a: geo.rtm2d_batch(*a[:3], npd=8, nt=5, dx=10.0, dz=10.0, dt_ms=1.0, favg=20.0, pfac=10.0,
                                            zs=3, shot_x=[10], shot_nxs=[9])]
    for dev in (False, True):
        a = [torch.from_numpy(x).cuda() for x in m] if dev else m
        for call in calls:
            with pytest.raises(geo.GeoError) as err:
                call(a)
            assert text in str(err.value), str(err.value)


@pytest.mark.parametrize("widths", [[3], [5, 31]])
def test_batch_backward_overflow_found_at_the_first_scan(geo, widths):
    """Overflow in cells that the next step's lines replace (a window of three
    columns has no others at its sides) is found by the scan after the step
    that computed it, not at the end of the pass."""
    nx, nz = 80, 40
    g = np.random.default_rng(4)
    v = (2000 + 900 * g.random((nx, nz))).astype(np.float32)
    r = ((v - 2000) / 2000).astype(np.float32)
    kw = dict(npd=5, nt=330, dx=10.0, dz=10.0, dt_ms=1.0, favg=20.0, pfac=3e38, zs=1, shot_x=[41] * len(widths),
              shot_nxs=widths)
    with pytest.raises(geo.GeoError) as err:
        geo.rtm2d_batch(v, 0.3 * r, 0.15 * r, **kw)
    assert "pass: wavefield non-finite by time step 100" in str(err.value)


def test_calls_in_threads_beside_captures(geo):
    """Batched RTM captures its time loop; shots, RTM and 3D runs of other host
    threads neither fail beside that nor break it."""
    import threading
    import torch
    g = torch.Generator(device="cuda").manual_seed(2)
    v = 2000 + 800 * torch.rand((90, 70), generator=g, device="cuda")
    m = (v, 0.3 * (v - 2000) / 2000, 0.15 * (v - 2000) / 2000)
    v3 = 2000 + 800 * torch.rand((20, 22, 24), generator=g, device="cuda")
    m3 = (v3, 0.3 * (v3 - 2000) / 2000, 0.15 * (v3 - 2000) / 2000)
    kw = dict(nt=60, dx=10.0, dz=10.0, favg=20.0)
    jobs = [lambda: geo.rtm2d_batch(*m, npd=10, dt_ms=1.0, pfac=10.0, zs=2, shot_x=[40, 50], shot_nxs=[31, 41], **kw),
            lambda: geo.fd2d_shot(*m, npd=10, dt=1e-3, fs=40, zs=2, **kw),
            lambda: geo.fd2d_shot(*m, npd=10, dt=1e-3, fs=40, zs=2, variant="mpi", **kw),
            lambda: geo.rtm2d_gpu(*m, npml=10, dt=1e-3, fs=40, zs=2, **kw)["illum"],
            lambda: geo.fd3d_shot(*m3, npd=8, dy=10.0, dt=1e-3, fsx=10, fsy=10, fsz=2, **kw)]
    ref = [j() for j in jobs]
    bad = []

    def run(first):
        with torch.cuda.stream(torch.cuda.Stream()):
            for k in range(15):
                i = (first + k) % len(jobs)
                try:
                    out = jobs[i]()
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(out, ref[i]):
                        bad.append((i, "differs"))
                except Exception as ex:
                    bad.append((i, repr(ex)[:200]))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
