"""GPU: the float sinc pass 2 with the resample in its own kernel (k_fl_resample2, k_fl_row_fft) against the FP64 oracle
at the sizes and pulse spacings where a run of eight can go wrong: fewer cross samples than a tile, tile and row-group
remainders, pulses displaced by up to nearly half their spacing (runs given up one by one, then whole jobs on the fused
kernel), and spacings past the dispatch's limit.  Tolerance: the float mode's stated 1e-6 relative L2."""
import numpy as np
import pytest

from oracle import float_pfa as fp
from pfa_b200 import autofocus, engine, geometry, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("jitter", [0.0, 0.3, 0.45, 2.0])
@pytest.mark.parametrize("bw,aperture_deg", [(600e6, 3.0), (1200e6, 3.0), (2000e6, 12.0)])
@pytest.mark.parametrize("m,n", [(64, 40), (256, 64), (257, 33), (300, 100), (384, 64), (1025, 65)])
def test_resample_against_fp64(torch_cuda, m, n, bw, aperture_deg, jitter):
    torch = torch_cuda
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=m + n, jitter=jitter, bw=bw, aperture_deg=aperture_deg)
    t = geometry.prepare_tables_from_scene(sc)
    with engine.FloatPlan(m, n, True, True) as plan:
        plan.set_tables(t)
        sig = torch.from_numpy(sc.signal).cuda()
        img = plan.form(sig, detect="complex").cpu().numpy()
        plan.set_tables(t, window=False, centred=False)
        raw = plan.form(sig, detect="complex").cpu().numpy()
    ref = fp.pfa_image(sc.signal, t["freq"], t["ax"], t["ay"], t["sgn"], precision="f64", interp="sinc")
    assert fp.rel_l2(img, ref) <= 1e-6
    g2, _ = fp.resample_kspace(sc.signal, t["freq"], t["ax"], t["ay"], "f64", "sinc", window=False)
    pad = np.zeros(raw.shape, complex)
    pad[:m, :n] = g2
    assert fp.rel_l2(raw, np.fft.fft2(pad)) <= 1e-6


def test_a_plan_changes_between_the_kernels(torch_cuda):
    # the job decides: a regular scene, an irregular one and the regular one again on one plan, frames and gradients
    torch = torch_cuda
    m, n = 290, 90
    out = {}
    with engine.FloatPlan(m, n, True, True) as plan:
        for k, jitter in enumerate((0.0, 2.0, 0.0)):
            sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=7, jitter=jitter)
            plan.set_tables(geometry.prepare_tables_from_scene(sc))
            sig = torch.from_numpy(sc.signal).cuda()
            ent, g = autofocus.entropy_grad(plan, sig, torch.linspace(-1, 1, m, device="cuda") ** 2)
            out[k] = plan.form(sig), float(ent), g
    assert torch.equal(out[0][0], out[2][0]) and abs(out[0][1] - out[2][1]) < 1e-6
    assert float((out[0][2] - out[2][2]).norm() / out[0][2].norm()) < 1e-5
    assert not torch.equal(out[0][0], out[1][0])


def test_plans_of_two_threads(torch_cuda):
    # jobs of other spacings need other amounts of shared memory of the same kernels: plans on two host threads, each on its own
    # stream, must not take each other's opt-in away between the call that raises it and the launch
    import threading
    torch = torch_cuda
    m, n, errors, images = 300, 64, [], {}
    jobs = []
    for bw, aperture in ((600e6, 3.0), (113.6e6, 6.5)):
        sc = synth.make_scene(m, n, n_targets=4, snr_db=15.0, seed=9, bw=bw, aperture_deg=aperture)
        jobs.append((geometry.prepare_tables_from_scene(sc), torch.from_numpy(sc.signal).cuda()))
    torch.cuda.synchronize()

    def work(k):
        try:
            t, sig = jobs[k]
            stream = torch.cuda.Stream()
            with engine.FloatPlan(m, n, True, True) as p, engine.FixedPlan(m, n, 512, True, True) as q:
                p.set_tables(t)
                q.set_tables(t)
                a, b = torch.empty((p.m2, p.n2), device="cuda"), torch.empty((512, 512), dtype=torch.uint16, device="cuda")
                stream.wait_stream(torch.cuda.current_stream())
                for _ in range(1500):
                    p.form(sig, out=a, stream=stream)
                    q.form(sig, out=b, stream=stream)
                stream.synchronize()
                images[k] = a, b
        except Exception as e:                               # (reported by the main thread)
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors
    for k, (t, sig) in enumerate(jobs):
        with engine.FloatPlan(m, n, True, True) as p, engine.FixedPlan(m, n, 512, True, True) as q:
            p.set_tables(t)
            q.set_tables(t)
            assert torch.equal(images[k][0], p.form(sig)) and torch.equal(images[k][1].view(torch.int16), q.form(sig).view(torch.int16))
