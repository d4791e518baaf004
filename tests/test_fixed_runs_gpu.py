"""GPU: the fixed-point passes in runs of eight outputs (k_fx_quant, k_fx_pass1_runs, k_fx_resample2), bit-exact against the emulator
restatement at the sizes, spacings and input forms where a run can go wrong: fewer samples than a tile, tile and pulse-group
remainders, rows and int16 inputs that start off the bulk copies' 16-byte units, output spacings up to and past the
dispatch's limit, and signals whose block exponent leaves the normal floats."""
import numpy as np
import pytest

from oracle import fixed_emulator as fe
from pfa_b200 import engine, geometry, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("aperture_deg,bw", [(3.0, 600e6), (3.0, 113.6e6), (6.0, 113.6e6), (10.0, 113.6e6)])
@pytest.mark.parametrize("m,n,G", [(33, 64, 64), (64, 127, 128), (100, 129, 256), (257, 200, 512), (40, 1000, 1024)])
def test_bit_exact(torch_cuda, m, n, G, aperture_deg, bw):
    torch = torch_cuda
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=m + n, jitter=0.2, aperture_deg=aperture_deg, bw=bw)
    t = geometry.prepare_tables_from_scene(sc)
    ref, _ = fe.form_image(sc.signal, t, G, True, True)
    with engine.FixedPlan(m, n, G, True, True) as plan:
        plan.set_tables(t)
        assert np.array_equal(plan.form(torch.from_numpy(sc.signal).cuda()).cpu().numpy(), ref)
        # the same frame from quantised I/Q that starts 0..3 samples off a 16-byte boundary
        e = plan.exponents()[2]
        q = np.clip(np.floor(np.stack([sc.signal.real, sc.signal.imag], -1) / np.float32(2.0 ** e)), -32768, 32767)
        for off in range(4):
            flat = torch.zeros((m * n + off, 2), dtype=torch.int16, device="cuda")
            iq = flat[off:].view(m, n, 2)
            iq.copy_(torch.from_numpy(q.astype(np.int16)))
            assert np.array_equal(plan.form_iq16(iq).cpu().numpy(), ref), off


@pytest.mark.parametrize("scale", [1e-41, 1e-37, 1e-20, 1e30])
def test_block_exponents(torch_cuda, scale):
    torch = torch_cuda
    sc = synth.make_scene(90, 75, n_targets=5, snr_db=15.0, seed=3)
    t = geometry.prepare_tables_from_scene(sc)
    sig = (sc.signal.astype(np.complex128) * scale).astype(np.complex64)
    ref, _ = fe.form_image(sig, t, 128, True, True)
    with engine.FixedPlan(90, 75, 128, True, True) as plan:
        plan.set_tables(t)
        assert np.array_equal(plan.form(torch.from_numpy(sig).cuda()).cpu().numpy(), ref)


@pytest.mark.parametrize("jitter", [0.0, 0.3, 0.45, 2.0])
@pytest.mark.parametrize("m,n,G,bw,aperture_deg", [(64, 40, 64, 600e6, 3.0), (256, 64, 256, 1200e6, 3.0), (257, 33, 512, 600e6, 3.0),
                                                   (385, 100, 512, 2000e6, 12.0), (1025, 65, 2048, 113.6e6, 3.0)])
def test_pass2_bit_exact(torch_cuda, m, n, G, bw, aperture_deg, jitter):
    # pulses displaced by up to nearly half their spacing (runs given up one by one), then jobs on the fused kernel;
    # lerp pass 1 as well, so that the split pass 2 runs alone
    torch = torch_cuda
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=m + n, jitter=jitter, bw=bw, aperture_deg=aperture_deg)
    t = geometry.prepare_tables_from_scene(sc)
    for rs in (True, False):
        ref, _ = fe.form_image(sc.signal, t, G, rs, True)
        with engine.FixedPlan(m, n, G, rs, True) as plan:
            plan.set_tables(t)
            img = plan.form(torch.from_numpy(sc.signal).cuda()).cpu().numpy()
            assert np.array_equal(img, ref), rs


@pytest.mark.parametrize("rs,az", [(True, False), (False, True), (True, True)])
def test_a_lost_copy_ends_the_frame(torch_cuda, rs, az):
    # a wait that runs out (the test hook pfa_config.test_wait_polls) with copies in flight and many tiles left: the CTA uses
    # no window, stages nothing more, waits for its copies and writes zeros; the frame is flagged, the context stays usable
    from pfa_b200 import _lib
    m, n, G = 2000, 1500, 2048
    sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=11, jitter=0.1)
    t = geometry.prepare_tables_from_scene(sc)
    img = np.ones((G, G), np.uint16)
    with engine.FixedPlan(m, n, G, rs, az, test_wait_polls=500) as plan:
        plan.set_tables(t)
        for _ in range(2):                                   # cleared once reported, raised by the next frame again
            with pytest.raises(_lib.PfaError) as ei:
                plan.form_host(sc.signal, img)
            assert ei.value.status == _lib.TIMEOUT and not img.any()
        with pytest.raises(_lib.PfaError) as ei:
            plan.form_host_frames([sc.signal] * 2)
        assert ei.value.status == _lib.TIMEOUT
    ref, _ = fe.form_image(sc.signal, t, G, rs, az)
    with engine.FixedPlan(m, n, G, rs, az) as plan:
        plan.set_tables(t)
        assert np.array_equal(plan.form_host(sc.signal), ref)


def test_a_flag_of_an_asynchronous_frame_stays_out_of_a_later_call(torch_cuda):
    # an asynchronous frame leaves the timeout flag (test hook; its job takes the pass in runs); a host frame of a job
    # that the fused pass takes is valid on the same plan, and empty calls report nothing
    from pfa_b200 import _lib
    torch = torch_cuda
    m, n, G = 300, 90, 512
    scenes = [synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=13, jitter=j) for j in (0.0, 2.0)]
    tables = [geometry.prepare_tables_from_scene(s) for s in scenes]
    ref, _ = fe.form_image(scenes[1].signal, tables[1], G, False, True)
    with engine.FixedPlan(m, n, G, False, True, test_wait_polls=500) as plan:
        for _ in range(2):
            plan.set_tables(tables[0])
            assert not plan.form(torch.from_numpy(scenes[0].signal).cuda()).view(torch.int16).any()
            plan.form_host_frames([])
            plan.set_tables(tables[1])
            assert np.array_equal(plan.form_host(scenes[1].signal), ref)
            assert np.array_equal(plan.form_host_frames([scenes[1].signal] * 3)[2], ref)
        plan.set_tables(tables[0])
        with pytest.raises(_lib.PfaError):
            plan.form_host(scenes[0].signal)


def test_the_quantised_signal_takes_no_memory_of_its_own(torch_cuda):
    # it lies where FFT-1 writes its rows later: a sinc plan holds what a lerp plan holds, and frames in a row stay right
    m, n, G = 200, 210, 256
    with engine.FixedPlan(m, n, G, True, True) as a, engine.FixedPlan(m, n, G, False, False) as b:
        assert a.workspace_bytes == b.workspace_bytes
        for seed in (1, 2):
            sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=seed)
            t = geometry.prepare_tables_from_scene(sc)
            a.set_tables(t)
            ref, _ = fe.form_image(sc.signal, t, G, True, True)
            assert np.array_equal(a.form(sc.signal), ref) and np.array_equal(a.form(sc.signal), ref)
