"""GPU: a frame or a gradient captured in a CUDA graph, then another job on the same plan.  The graph keeps the kernels that the first job
chose; they read the job's vectors from the plan, so a replay gives what the plan gives eagerly under the new job: another
regular scene, displaced pulses that the passes in runs do not take, and descending source axes.  Frames: the same bits (fixed) or
1e-6 relative L2 (float); the gradient's sums have no fixed order, 1e-4."""
import numpy as np
import pytest

from oracle import fixed_emulator as fe
from pfa_b200 import autofocus, engine, geometry, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _tables(m, n):
    """The captured job and three to replay under: other spacing, irregular, descending (signal, tables)."""
    out = []
    for k, (jitter, bw, aperture) in enumerate([(0.1, 600e6, 3.0), (0.3, 113.6e6, 5.0), (2.0, 600e6, 3.0), (0.4, 600e6, 3.0)]):
        sc = synth.make_scene(m, n, n_targets=6, snr_db=15.0, seed=40 + k, jitter=jitter, bw=bw, aperture_deg=aperture)
        t = dict(geometry.prepare_tables_from_scene(sc))
        if k == 3:
            t["freq"] = -t["freq"]
            t["KR"] = -t["KR"][::-1]
        out.append((sc.signal, t))
    return out


@pytest.mark.parametrize("rs,az", [(True, True), (True, False), (False, True)])
def test_fixed(torch_cuda, rs, az):
    torch = torch_cuda
    m, n, G = 290, 150, 512
    jobs = _tables(m, n)
    sig = torch.from_numpy(jobs[0][0]).cuda()
    img = torch.empty((G, G), dtype=torch.uint16, device="cuda")
    with engine.FixedPlan(m, n, G, rs, az) as plan:
        plan.set_tables(jobs[0][1])
        plan.form(sig, out=img)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.form(sig, out=img)
        for signal, t in jobs[1:] + jobs[:1]:
            plan.set_tables(t)
            sig.copy_(torch.from_numpy(signal))
            graph.replay()
            ref, _ = fe.form_image(signal, t, G, rs, az)
            assert np.array_equal(img.cpu().numpy(), ref)
        del graph


@pytest.mark.parametrize("rs,az,mixed", [(True, True, False), (True, False, False), (False, True, False), (False, False, True),
                                         (True, True, True)])
def test_float(torch_cuda, rs, az, mixed):
    torch = torch_cuda
    m, n = (2050, 70) if mixed else (290, 150)
    jobs = _tables(m, n)
    sig = torch.from_numpy(jobs[0][0]).cuda()
    with engine.FloatPlan(m, n, rs, az, mixed=mixed) as plan, engine.FloatPlan(m, n, rs, az, mixed=mixed) as other:
        img = torch.empty((plan.m2, plan.n2), dtype=torch.complex64, device="cuda")
        plan.set_tables(jobs[0][1])
        plan.form(sig, out=img, detect="complex")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.form(sig, out=img, detect="complex")
        for signal, t in jobs[1:] + jobs[:1]:
            plan.set_tables(t)
            other.set_tables(t)
            sig.copy_(torch.from_numpy(signal))
            graph.replay()
            ref = other.form(sig, detect="complex")
            assert float((img - ref).norm() / ref.norm()) <= 1e-6
        del graph


@pytest.mark.parametrize("rs,az", [(True, True), (False, True)])
def test_gradient(torch_cuda, rs, az):
    torch = torch_cuda
    m, n = 290, 150
    jobs = _tables(m, n)
    sig = torch.from_numpy(jobs[0][0]).cuda()
    theta = torch.linspace(-1, 1, m, device="cuda") ** 2
    with engine.FloatPlan(m, n, rs, az) as plan, engine.FloatPlan(m, n, rs, az) as other:
        plan.set_tables(jobs[0][1])
        ent, g = autofocus.entropy_grad(plan, sig, theta)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            autofocus.entropy_grad(plan, sig, theta, g, ent)
        for signal, t in jobs[1:] + jobs[:1]:
            plan.set_tables(t)
            other.set_tables(t)
            sig.copy_(torch.from_numpy(signal))
            graph.replay()
            ent2, g2 = autofocus.entropy_grad(other, sig, theta)
            assert abs(float(ent) - float(ent2)) <= 1e-5 * abs(float(ent2))
            assert float((g - g2).norm() / g2.norm()) <= 1e-4
        del graph
