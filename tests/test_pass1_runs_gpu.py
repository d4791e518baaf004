"""GPU: pass 1 of the float sinc in runs of eight outputs (k_fl_pass1_runs) against the FP64 oracle, at the sizes and
spacings where a run can go wrong: fewer samples than a tile, tile and pulse-group remainders, odd row lengths and a
signal that starts on an 8-byte boundary (the bulk copies move 16-byte units), output spacings up to and past the
limit of the dispatch, and non-finite samples next to the taps.  Tolerance: the float mode's stated 1e-6 relative L2."""
import numpy as np
import pytest

from oracle import float_pfa as fp
from pfa_b200 import engine, geometry, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("aperture_deg,bw", [(3.0, 600e6), (3.0, 113.6e6), (6.0, 113.6e6), (6.7, 113.6e6), (10.0, 113.6e6)])
@pytest.mark.parametrize("m,n", [(33, 64), (64, 127), (100, 129), (257, 1000), (65, 4097)])
def test_runs_against_fp64(torch_cuda, m, n, aperture_deg, bw, offset):
    torch = torch_cuda
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=m + n, jitter=0.2, aperture_deg=aperture_deg, bw=bw)
    t = geometry.prepare_tables_from_scene(sc)
    flat = torch.zeros(m * n + offset, dtype=torch.complex64, device="cuda")
    sig = flat[offset:].view(m, n)
    sig.copy_(torch.from_numpy(sc.signal))
    with engine.FloatPlan(m, n, True, True) as plan:
        plan.set_tables(t)
        img = plan.form(sig, detect="complex").cpu().numpy()
    ref = fp.pfa_image(sc.signal, t["freq"], t["ax"], t["ay"], t["sgn"], precision="f64", interp="sinc")
    assert fp.rel_l2(img, ref) <= 1e-6


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_samples_beside_the_taps_are_not_used(torch_cuda, bad):
    # an output grid that starts 40 samples into every pulse: samples below 25 feed no output
    torch = torch_cuda
    m, n = 96, 700
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=5)
    job = geometry.float_job(geometry.prepare_tables_from_scene(sc))
    step = 2.0 / synth.C * job["pr"].max() * job["df"][0]
    job["KR"] = 2.0 / synth.C * job["f0"][0] * job["pr"].max() + step * (40.3 + 1.01 * np.arange(n))
    clean, dirty = sc.signal.copy(), sc.signal.copy()
    clean[:, :25] = 0
    dirty[:, :25] = bad
    with engine.FloatPlan(m, n, True, True) as plan:
        plan.set_job(job)
        a = plan.form(torch.from_numpy(clean).cuda(), detect="complex")
        b = plan.form(torch.from_numpy(dirty).cuda(), detect="complex")
    assert torch.isfinite(torch.view_as_real(a)).all() and torch.equal(a, b)


@pytest.mark.parametrize("mixed,az", [(True, False), (False, True)])
def test_a_lost_copy_ends_the_frame(torch_cuda, mixed, az):
    # the test hook of the window copies (lines below 2048 points: mixed plans have no other wait here; FP32: both passes run
    # out): zeros, the timeout status, and a plan without the hook forms the frame right after
    from pfa_b200 import _lib
    m, n = 900, 1000
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=12, jitter=0.1)
    t = geometry.prepare_tables_from_scene(sc)
    img = np.ones((1024, 1024), np.float32)
    with engine.FloatPlan(m, n, True, az, mixed=mixed, test_wait_polls=500) as plan:
        plan.set_tables(t)
        for _ in range(2):
            with pytest.raises(_lib.PfaError) as ei:
                plan.form_host(sc.signal, img)
            assert ei.value.status == _lib.TIMEOUT and not img.any()
    with engine.FloatPlan(m, n, True, True, mixed=mixed) as plan:
        plan.set_tables(t)
        img = plan.form_host(sc.signal, detect="complex")
    ref = fp.pfa_image(sc.signal, t["freq"], t["ax"], t["ay"], t["sgn"], precision="f64", interp="sinc")
    assert fp.rel_l2(img, ref) <= 1e-6


def test_an_end_sample_short_of_the_axis(torch_cuda):
    # a job whose f_last lies inside the axis: bins past that end are zero for every pulse, whichever run they fall in
    torch = torch_cuda
    m, n, j_end = 96, 300, 100
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=6)
    job = geometry.float_job(geometry.prepare_tables_from_scene(sc))
    cut = dict(job, f_last=(job["KR"][j_end] + 0.3 * (job["KR"][1] - job["KR"][0])) * synth.C / (2.0 * job["pr"]))
    sig, rows = torch.from_numpy(sc.signal).cuda(), []
    with engine.FloatPlan(m, n, True, False) as plan:
        for j in (job, cut):
            plan.set_job(j, window=False, centred=False)
            rows.append(np.fft.ifft2(plan.form(sig, detect="complex").cpu().numpy().astype(complex))[:m, :n])
    scale = np.abs(rows[0]).max()
    assert np.abs(rows[1][:, :j_end + 1] - rows[0][:, :j_end + 1]).max() <= 1e-5 * scale
    assert np.abs(rows[1][:, j_end + 1:]).max() <= 1e-5 * scale
