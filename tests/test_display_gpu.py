"""GPU: the device display scaling of save_detected_geotiff (pfa_display_u8, src/form_image_pfa.py:287-292)
against the reference arithmetic (np.percentile(amp, 99.7), clip, uint8), bit for bit: random magnitudes
of many sizes (vector tails, a single element, heavy ties, constant images, a range of scales), other
percentiles, and the detected image of a focused scene; plus the whole GeoTIFF path on that image."""
import numpy as np
import pytest

from oracle import geotiff_ref
from pfa_b200 import engine, geocode, geometry, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _check(torch, amp, pct=99.7):
    x = torch.from_numpy(amp).cuda()
    out, hi = geocode.display_u8(x, pct)
    ref_amp = amp.astype(np.float32)
    ref_hi = np.percentile(ref_amp, pct)
    ref = np.clip(ref_amp / (ref_hi + 1e-12) * 255.0, 0, 255).astype(np.uint8)
    assert float(hi) == float(ref_hi), (float(hi), float(ref_hi), amp.size)
    got = out.cpu().numpy()
    assert np.array_equal(got, ref), (amp.size, int((got != ref).sum()))


@pytest.mark.parametrize("n", [1, 2, 5, 1023, 4096, 100003, 1 << 20, 3_000_001])
def test_random_sizes(torch_cuda, n):
    rng = np.random.default_rng(n)
    _check(torch_cuda, (rng.random(n) * rng.choice([1e-3, 1.0, 7.5, 3e4])).astype(np.float32))


def test_ties_constants_and_percentiles(torch_cuda):
    rng = np.random.default_rng(3)
    ties = rng.integers(0, 40, 500000).astype(np.float32) * 0.25
    _check(torch_cuda, ties)
    _check(torch_cuda, np.full(77777, 3.5, np.float32))
    _check(torch_cuda, np.zeros(1000, np.float32) + np.float32(1e-30))
    ray = rng.rayleigh(1.0, 2_000_000).astype(np.float32)
    for pct in (0.0, 50.0, 99.0, 99.7, 99.99, 100.0):
        _check(torch_cuda, ray, pct)


def test_focused_image_and_geotiff(torch_cuda, tmp_path):
    torch = torch_cuda
    sc = synth.make_scene(1500, 1300, n_targets=32, clutter_db=-10.0, snr_db=20.0, seed=31)
    tb = geometry.prepare_tables_from_scene(sc)
    with engine.FloatPlan(1500, 1300) as plan:
        plan.set_tables(tb)
        mag = plan.form(torch.from_numpy(sc.signal).cuda())
    cz = None
    ref, ref_hi = geotiff_ref.display_u8(mag.cpu().numpy())
    got, hi = geocode.display_u8(mag)
    assert float(hi) == float(ref_hi) and np.array_equal(got.cpu().numpy(), ref)
    # the file: the synthetic scene sits at the Earth's centre, so give it a real place for the projection
    tbg = dict(tb)
    tbg["center_ecef"] = geocode.geodetic_to_ecef(-96.8, 46.9, 270.0)
    tbg["uiax"], tbg["uiay"] = np.array([0.11, 0.99, 0.0]), np.array([-0.73, 0.08, 0.68])
    path, epsg, aff = geocode.save_detected_geotiff(mag, tbg, tmp_path / "img.tif")
    Image = pytest.importorskip("PIL.Image")
    assert np.array_equal(np.array(Image.open(path)), ref) and epsg == 32614
    del cz


def _shaped(kind, n, rng):
    if kind == "rayleigh":
        return rng.rayleigh(1.0, n)
    if kind == "ties_below":            # the value of rank k also fills the window's lower end
        return np.where(rng.random(n) < 0.9965, 2.0, 2.0 + rng.random(n))
    if kind == "ties_at_rank":          # one heavy value around the rank
        return np.where(rng.random(n) < 0.02, 5.0, np.where(rng.random(n) < 0.99, rng.random(n), 9.0))
    if kind == "mostly_zero":           # a zero-padded product
        return np.where(rng.random(n) < 0.002, rng.rayleigh(3.0, n), 0.0)
    if kind == "few_values":            # candidates that crowd single values
        return rng.integers(0, 3000, n) * 0.5
    if kind == "one_block_bright":      # a bright patch that the strata see, far above everything else
        a = rng.random(n) * 1e-6
        a[n // 3: n // 3 + n // 300] += 1e6
        return a
    # "unsampled": a sample of one 16-byte group per stratum says nothing about the image (the radix sweeps answer)
    lg, n4 = (13 if n >= 1 << 23 else 10), n >> 2
    g = np.arange(1 << lg, dtype=np.uint64)
    r = (g * 2654435761) & 0xffffffff
    r ^= r >> 15
    r = (r * 2246822519) & 0xffffffff
    r ^= r >> 13
    a0, a1 = (g * n4) >> lg, ((g + 1) * n4) >> lg
    hit = (a0 + (((a1 - a0) * r) >> 32)).astype(np.int64)
    a = rng.random(n)
    a[(4 * hit[:, None] + np.arange(4)).ravel()] = 7.0
    return a


@pytest.mark.parametrize("n", [4095, 4096, 4097, 200_003, 9_000_001])
@pytest.mark.parametrize("kind", ["rayleigh", "ties_below", "ties_at_rank", "mostly_zero", "few_values", "one_block_bright",
                                  "unsampled"])
def test_window_select_and_radix_sweeps(torch_cuda, kind, n):
    rng = np.random.default_rng(n + len(kind))
    amp = _shaped(kind, n, rng).astype(np.float32)
    for pct in (99.7, 50.0, 0.01, 99.999, 100.0):
        _check(torch_cuda, amp, pct)


def test_candidates_past_the_buffer(torch_cuda):
    # the median of a large image: more elements inside the window than the candidate list holds
    x = torch_cuda.rand(100_000_007, generator=torch_cuda.Generator(device="cuda").manual_seed(5), device="cuda")
    out, hi = geocode.display_u8(x, 50.0)
    v = np.float32(x.numel() - 1) * (np.float32(50.0) / np.float32(100.0))
    k = int(np.floor(v))
    s = x.sort().values[k:k + 2].cpu().numpy()
    ref = s[0] + (s[1] - s[0]) * np.float32(v - np.floor(v))
    assert float(hi) == float(np.float32(ref))
    ref8 = ((x / torch_cuda.tensor(np.float32(ref) + np.float32(1e-12)).cuda()) * 255.0).clamp(0, 255).to(torch_cuda.uint8)
    assert torch_cuda.equal(out, ref8)


def test_more_candidates_than_expected(torch_cuda):
    # the sample's groups (their places as in _shaped) are spread over [0, 1), every other element lies inside the window
    # that they give: the list overflows and the radix sweeps answer
    torch = torch_cuda
    n, lg = 40_000_003, 13
    n4 = n >> 2
    g = np.arange(1 << lg, dtype=np.uint64)
    r = (g * 2654435761) & 0xffffffff
    r ^= r >> 15
    r = (r * 2246822519) & 0xffffffff
    r ^= r >> 13
    a0, a1 = (g * n4) >> lg, ((g + 1) * n4) >> lg
    hit = (a0 + (((a1 - a0) * r) >> 32)).astype(np.int64)
    rng = np.random.default_rng(8)
    amp = np.full(n, 0.997, np.float32)
    amp[(4 * hit[:, None] + np.arange(4)).ravel()] = rng.random(4 << lg).astype(np.float32)
    for pct in (99.7, 50.0):
        _check(torch, amp, pct)


@pytest.mark.parametrize("n,pct", [(3000, 99.7), (300_001, 99.7), (300_001, 50.0), (70_000_000, 50.0)])
def test_captured_in_a_graph(torch_cuda, n, pct):
    # the call's launches inside a CUDA graph: replays on new images give what the eager call gives
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand(n, generator=g, device="cuda")
    geocode.display_u8(x, pct)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, hi = geocode.display_u8(x, pct)
    for _ in range(2):
        x.copy_(torch.rand(n, generator=g, device="cuda").square() * 3.0)
        graph.replay()
        ref, ref_hi = geocode.display_u8(x, pct)
        assert torch.equal(out, ref) and float(hi) == float(ref_hi)
