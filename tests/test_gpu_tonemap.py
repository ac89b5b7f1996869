"""GPU tests of the LDR colour chain (lum_tonemap_device, lum_render_ldr) against the f64 oracle.

The device computes the chain in f64 without FMA contraction, so bytes equal the oracle's
except where a last-bit difference of pow/log/exp (CUDA's versus the host's) lands on a
quantisation boundary: >= 99.99% of channel bytes identical and no byte off by more than 1.
"""
import numpy as np
import pytest

import luminara_b200 as L
from luminara_b200 import abi
from luminara_b200 import workloads as W
from oracle import tonemap as OT

pytestmark = pytest.mark.gpu

CHAINS = [
    {},
    {"tone_map": OT.REINHARD, "gamma": 2.2, "dither": True, "vignette": 0.4, "exposure": 1.7},
    {"tone_map": OT.FILMIC, "auto_exposure": True, "saturation": 1.3, "white_balance": 0.5, "hue_shift": 25.0,
     "grade_shadows": (0.9, 1.0, 1.15), "grade_highlights": (1.1, 1.0, 0.9)},
    {"tone_map": OT.NONE, "brightness": 0.05, "contrast": 1.4, "sepia": 0.3, "tint": (1.0, 0.9, 0.8),
     "color_balance": (1.1, 1.0, 0.95), "posterize": 6},
    {"auto_exposure": True, "exposure": 0.5, "dither": True, "hue_shift": -40.0, "saturation": 0.6},
]


def tm_config(d):
    tm = L.ToneMapConfig()
    for k, v in d.items():
        setattr(tm, k, v)
    return tm


def compare(got, want):
    diff = np.abs(got.astype(int) - want.astype(int))
    assert diff.max() <= 1, diff.max()
    assert (diff == 0).mean() >= 0.9999, (diff == 0).mean()


def hdr_image(h, w, seed=0):
    rng = np.random.default_rng(seed)
    img = np.exp(rng.normal(-1.0, 1.5, (h, w, 3))).astype(np.float32)        # 5 decades of radiance
    img[rng.random((h, w)) < 0.02] = 0.0
    img[0, 0] = (-0.5, 2.0, 1e4)
    return img


@pytest.mark.parametrize("chain", range(len(CHAINS)))
@pytest.mark.parametrize("shape", [(135, 240), (23, 37)])
def test_tonemap_device_matches_oracle(chain, shape):
    import torch
    h, w = shape
    img = hdr_image(h, w, chain)
    d_hdr = torch.from_numpy(img).cuda()
    d_out = torch.empty((h, w, 4), dtype=torch.uint8, device="cuda")
    scratch = torch.empty(abi.TONEMAP_SCRATCH_BYTES, dtype=torch.uint8, device="cuda")
    L.tonemap_device(d_hdr.data_ptr(), w, h, tm_config(CHAINS[chain]), scratch.data_ptr(), d_out.data_ptr())
    torch.cuda.synchronize()
    compare(d_out.cpu().numpy(), OT.tonemap(img, CHAINS[chain]))


def test_unaligned_buffers_take_the_scalar_path():
    import torch
    h, w = 31, 17
    img = hdr_image(h, w, 5)
    flat = torch.zeros(h * w * 3 + 1, dtype=torch.float32, device="cuda")
    flat[1:] = torch.from_numpy(img).reshape(-1).cuda()
    out = torch.zeros(h * w * 4 + 3, dtype=torch.uint8, device="cuda")
    L.tonemap_device(flat.data_ptr() + 4, w, h, tm_config(CHAINS[1]), 0, out.data_ptr() + 3)
    torch.cuda.synchronize()
    compare(out[3:].cpu().numpy().reshape(h, w, 4), OT.tonemap(img, CHAINS[1]))


def test_auto_exposure_needs_scratch_and_bad_tone_map_is_rejected():
    import torch
    d = torch.ones((4, 4, 3), dtype=torch.float32, device="cuda")
    o = torch.empty((4, 4, 4), dtype=torch.uint8, device="cuda")
    with pytest.raises(L.LuminaraError):
        L.tonemap_device(d.data_ptr(), 4, 4, tm_config({"auto_exposure": True}), 0, o.data_ptr())
    with pytest.raises(L.LuminaraError):
        L.tonemap_device(d.data_ptr(), 4, 4, tm_config({"tone_map": 7}), 0, o.data_ptr())


@pytest.mark.parametrize("chain", [0, 2, 3])
def test_render_ldr_is_the_chain_over_the_hdr_render(chain):
    world, cfg = W.box_room(width=96, height=64, spp=16)
    world.camera.aspect_ratio = 96 / 64
    cfg.exposure = 1.5
    sc = L.GpuScene(world)
    ldr, st = sc.render_ldr(cfg, tm_config(CHAINS[chain]))
    assert st.paths == 96 * 64 * 16 and ldr.shape == (64, 96, 4)
    cfg1 = L.RenderConfig(**{**cfg.__dict__, "exposure": 1.0})
    hdr, _ = sc.render(cfg1)
    want = OT.tonemap(hdr, {**CHAINS[chain], "exposure": 1.5})       # the render's exposure, not tm's
    compare(ldr, want)
    assert ldr[..., :3].max() > 100


@pytest.mark.parametrize("exposure", [1.0, 4.0, 0.25, 2.0 ** -20])
def test_power_of_two_exposure_integer_keys(exposure):
    """An exposure 2^k takes the byte table with keys formed from the f32 bits (x = v * 2^k is
    exact); zero, negative, NaN, denormal and very large values fall back to the f64 key.  The
    bytes must be the chain's over eight decades and at those edges."""
    import torch
    rng = np.random.default_rng(7)
    h, w = 64, 256
    img = np.exp(rng.uniform(-12.0, 12.0, (h, w, 3))).astype(np.float32)
    edges = np.array([np.nan, 0.0, -0.0, -1.0, 1e-45, 1e-39, 1.17e-38, 2.0 ** 99, 6.4e29, 1e30, 1e35, 3e38],
                     dtype=np.float32)
    img.reshape(-1)[: edges.size] = edges
    d_hdr = torch.from_numpy(img).cuda()
    d_out = torch.empty((h, w, 4), dtype=torch.uint8, device="cuda")
    scratch = torch.empty(abi.TONEMAP_SCRATCH_BYTES, dtype=torch.uint8, device="cuda")
    L.tonemap_device(d_hdr.data_ptr(), w, h, tm_config({"exposure": exposure}), scratch.data_ptr(), d_out.data_ptr())
    torch.cuda.synchronize()
    got = d_out.cpu().numpy()
    want = OT.tonemap(img, {"exposure": exposure})
    compare(got, want)
    np.testing.assert_array_equal(got.reshape(-1, 4)[:4, :3].reshape(-1), want.reshape(-1, 4)[:4, :3].reshape(-1))


@pytest.mark.parametrize("curve", [OT.ACES, OT.REINHARD, OT.FILMIC, OT.NONE])
@pytest.mark.parametrize("exposure", [1.0, 2.0 ** -20, 2.0 ** 19, 2.0 ** 20, 1.7, 0.0])
def test_common_chain_over_tiles_and_rare_values(curve, exposure):
    """Pixel counts around the 4-pixel groups and 128-pixel tiles, with zeros, negatives, denormals,
    huge values, infinities and NaN among them, at exposures on both sides of each key form."""
    import torch
    rare = np.array([0.0, -0.0, -1.0, 1e-45, 1e-38, 3.4e38, np.inf, -np.inf, np.nan, 1e29, 2.0 ** 97], np.float32)
    for n in (1, 3, 4, 127, 128, 131, 516, 5003):
        img = hdr_image(1, n, n) / np.float32(exposure if exposure > 0 else 1.0)
        flat = img.reshape(-1)
        flat[:: 7][: len(rare)] = rare[: len(flat[::7])]
        d_hdr, d_out = torch.from_numpy(img).cuda(), torch.zeros((1, n, 4), dtype=torch.uint8, device="cuda")
        chain = {"tone_map": curve, "exposure": exposure}
        L.tonemap_device(d_hdr.data_ptr(), n, 1, tm_config(chain), 0, d_out.data_ptr())
        torch.cuda.synchronize()
        with np.errstate(all="ignore"):
            compare(d_out.cpu().numpy(), OT.tonemap(img, chain))


@pytest.mark.parametrize("chain", [
    {"saturation": 1.3, "vignette": 0.5}, {"hue_shift": 30.0, "contrast": 1.3, "brightness": -0.1, "gamma": 2.2},
    {"tone_map": OT.REINHARD, "sepia": 0.6, "posterize": 5, "white_balance": -0.7},
    {"tone_map": OT.NONE, "tint": (0.9, 1.0, 0.7), "color_balance": (1.2, 0.9, 1.0), "auto_exposure": True,
     "grade_shadows": (0.8, 1.0, 1.2), "grade_highlights": (1.1, 1.0, 0.9)}])
def test_graded_chain_over_ragged_tiles_and_rare_values(chain):
    """The optional steps at widths and pixel counts around the 32-pixel tiles, with zeros, negatives,
    huge values and NaN among the pixels (infinities would make the auto-exposure's mean infinite)."""
    import torch
    rare = np.array([0.0, -0.0, -1.0, 1e-45, 1e30, 3e37, np.nan, 1e20], np.float32)
    for w, h in ((1, 1), (1, 33), (31, 1), (5, 13), (64, 3), (127, 9)):
        img = hdr_image(h, w, w * h)
        if not chain.get("auto_exposure"):
            flat = img.reshape(-1)
            flat[::11][: len(rare)] = rare[: len(flat[::11])]
        d_hdr, d_out = torch.from_numpy(img).cuda(), torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
        scratch = torch.empty(abi.TONEMAP_SCRATCH_BYTES, dtype=torch.uint8, device="cuda")
        L.tonemap_device(d_hdr.data_ptr(), w, h, tm_config(chain), scratch.data_ptr(), d_out.data_ptr())
        torch.cuda.synchronize()
        with np.errstate(all="ignore"):
            compare(d_out.cpu().numpy(), OT.tonemap(img, chain))


def test_graded_chain_can_be_captured_before_its_table_exists():
    """The first call of a graded chain inside a stream capture records kernels only (its byte table is
    not uploaded there), and the replayed graph gives the bytes of a direct call."""
    import torch
    img = hdr_image(40, 52, 1)
    tm = tm_config({"saturation": 1.4, "gamma": 1.9371})                  # a gamma no other test uses
    d_hdr = torch.from_numpy(img).cuda()
    a, b = (torch.zeros((40, 52, 4), dtype=torch.uint8, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        L.tonemap_device(d_hdr.data_ptr(), 52, 40, tm, 0, a.data_ptr(), torch.cuda.current_stream().cuda_stream)
    graph.replay()
    L.tonemap_device(d_hdr.data_ptr(), 52, 40, tm, 0, b.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    compare(a.cpu().numpy(), b.cpu().numpy())
    compare(b.cpu().numpy(), OT.tonemap(img, {"saturation": 1.4, "gamma": 1.9371}))


@pytest.mark.parametrize("steps", [{}, {"saturation": 1.2}])
def test_gammas_without_a_table_and_new_pairs_after_them(steps):
    """A gamma whose curve fits no byte table (ACES at 4) over many calls, then pairs of their own: the chain's
    bytes from whichever kernel takes them (which pairs get tables is checked in test_table_cache)."""
    import torch
    img = hdr_image(16, 32, 3)
    d_hdr, d_out = torch.from_numpy(img).cuda(), torch.zeros((16, 32, 4), dtype=torch.uint8, device="cuda")
    for chain in [{**steps, "gamma": g} for g in [4.0] * 40 + [1.2345, 2.2, 4.0, 1.5]]:
        L.tonemap_device(d_hdr.data_ptr(), 32, 16, tm_config(chain), 0, d_out.data_ptr())
        torch.cuda.synchronize()
        compare(d_out.cpu().numpy(), OT.tonemap(img, chain))


@pytest.mark.parametrize("steps", [{}, {"saturation": 1.2}])
@pytest.mark.parametrize("mode", ["global", "thread_local"])
@pytest.mark.parametrize("blocking", [False, True])
@pytest.mark.parametrize("own", [False, True])
def test_first_call_of_a_pair_leaves_stream_captures_whole(steps, mode, blocking, own):
    """The first call of a (curve, gamma) pair uploads its table.  Made while a stream (one that waits for
    the default stream, or not) is being captured, it neither breaks the capture nor is broken by it: on a
    stream beside the captured one it runs at once, on the captured stream it becomes part of the graph."""
    import ctypes

    import torch
    chain = {**steps, "gamma": 1.61 + 0.01 * len(steps) + 0.1 * own + (0.2 if mode == "global" else 0.0) + 0.4 * blocking}
    img = hdr_image(24, 36, 2)
    d_hdr = torch.from_numpy(img).cuda()
    out, x = torch.zeros((24, 36, 4), dtype=torch.uint8, device="cuda"), torch.zeros(8, device="cuda")
    beside = torch.cuda.Stream()
    captured = None
    if blocking:
        handle = ctypes.c_void_p()
        assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
        captured = torch.cuda.ExternalStream(handle.value)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=captured, capture_error_mode=mode):
        x.add_(1.0)
        stream = torch.cuda.current_stream() if own else beside
        L.tonemap_device(d_hdr.data_ptr(), 36, 24, tm_config(chain), 0, out.data_ptr(), stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 1.0).all()
    compare(out.cpu().numpy(), OT.tonemap(img, chain))
