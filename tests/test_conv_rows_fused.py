"""The row form of the denoiser's convolution in the sizes it is chosen for
(enough 8 x 16-pixel tiles an SM for the row pairs of a run): the edges of its
128-pixel strips, row pairs and runs, and its fused epilogues - pooling at 32
and 48 channels, nearest upsampling, the training step's ReLU mask - in networks
where every resolution runs by rows. Bounds as test_denoiser_conv,
test_denoiser_unet and test_denoiser_training."""
import ctypes as C

import numpy as np
import pytest

import test_denoiser_conv as conv
import test_denoiser_training as training
from helpers import pinhole, rig_of
from ray_tracing_gb300 import denoiser, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,cin,cout,relu,ych,yoff", [
    (100, 1, 80, 16, 32, 1, 32, 0),    # one row: no neighbours above or below
    (96, 2, 127, 32, 32, 1, 80, 0),    # a strip's last pixel missing
    (60, 3, 128, 32, 48, 0, 48, 0),    # exactly a strip, an odd height
    (40, 5, 129, 48, 48, 1, 112, 0),   # a last strip of one pixel
    (2, 200, 257, 32, 48, 1, 48, 0),
    (2, 144, 385, 32, 32, 1, 32, 0),
    (1, 112, 513, 16, 64, 1, 64, 0),
    (4, 72, 256, 48, 64, 1, 64, 0),
    (4, 33, 230, 112, 48, 1, 48, 0),   # two row stages
    (8, 33, 160, 112, 48, 1, 48, 0),
    (4, 90, 333, 80, 32, 1, 32, 0),
    (2, 300, 120, 16, 64, 0, 64, 0),
    (1, 700, 1000, 64, 64, 1, 112, 48),  # long runs over several columns, four TMEM slots
])
def test_rows_match_torch(n, h, w, cin, cout, relu, ych, yoff):
    conv.test_conv3x3_matches_torch(n, h, w, cin, cout, relu, ych, yoff)


@pytest.mark.parametrize("cameras,w,h", [
    (4, 1000, 200),  # pooling and upsampling at both levels by rows
    (4, 1004, 206),  # upsampling into half resolution by its own kernel, into the full one fused
    (4, 1002, 201),  # odd sizes: pooled edges, upsampling by its own kernel
    (1, 648, 360),   # full and half resolution by rows, the quarter by tiles
])
def test_unet_by_rows(cameras, w, h):
    torch = pytest.importorskip("torch")
    from ray_tracing_gb300.renderer import Renderer
    torch.manual_seed(2)
    model = denoiser.build_model()
    flat = denoiser.flatten(model)
    denoiser.unflatten(model, denoiser.from_bf16_bits(denoiser.to_bf16_bits(flat)))
    base = scenes.default_rig("random_spheres", cameras)
    cams = []
    for i in range(cameras):
        cam = pinhole(w, h, 80.0)
        cam.rotation[:] = base.cameras[i].rotation[:]
        cam.translation[:] = base.cameras[i].translation[:]
        cams.append(cam)
    prof = scenes.profile("balanced", samples_per_pixel=1, max_bounces=2, enable_denoise=1, enable_restir_di=0)
    sc = scenes.HostScene("random_spheres", seed=3, detail=64)
    model = model.cuda().eval()
    with Renderer() as r:
        r.prepare_scene(sc.view)
        r.set_denoiser(flat)
        r.render_frame(rig_of(*cams), prof, cameras)
        for cam in range(cameras):
            x = denoiser.make_input(*(r.buffer(cam, b)[None] for b in ("beauty", "albedo", "denoiser_normal", "depth")))
            with torch.no_grad():
                y = model(torch.from_numpy(np.ascontiguousarray(x)).cuda(), bf16_activations=True)
            want = np.expm1(np.maximum(y[0].permute(1, 2, 0).cpu().numpy(), 0.0))
            got = r.buffer(cam, "denoised")[..., :3]
            rel = np.abs(got - want) / np.maximum(np.abs(want), 1e-2)
            assert np.median(rel) <= 2e-3, f"camera {cam}: median {np.median(rel):.2e}"
            assert np.quantile(rel, 0.999) <= 5e-2, f"camera {cam}: 99.9% {np.quantile(rel, 0.999):.2e}"


@pytest.mark.parametrize("n,h,w", [(4, 200, 1000), (2, 400, 512), (1, 16, 320)])
def test_gradients_by_rows(n, h, w):
    torch = pytest.importorskip("torch")
    torch.manual_seed(3)
    model = denoiser.build_model()
    flat = denoiser.from_bf16_bits(denoiser.to_bf16_bits(denoiser.flatten(model))).astype(np.float32)
    denoiser.unflatten(model, flat)
    x, t = training._batch(np.random.default_rng(5), n, h, w)
    dev = torch.device("cuda", 0)
    xb = torch.from_numpy(training._blocked(x)).to(dev).to(torch.bfloat16).contiguous()
    tt = torch.from_numpy(t).to(dev).contiguous()
    lib, tr = training._trainer(torch, flat, n, h, w)
    try:
        loss = C.c_float()
        st = lib.rtgb_trainer_step(tr, C.c_void_p(xb.data_ptr()), C.c_void_p(tt.data_ptr()), 0.0, C.byref(loss))
        assert st == 0, lib.rtgb_trainer_last_error(tr)
        got = np.empty_like(flat)
        assert lib.rtgb_trainer_gradients(tr, got.ctypes.data) == 0
    finally:
        lib.rtgb_trainer_destroy(tr)
    model = model.to(dev)
    out = model(torch.from_numpy(x[:, :10]).to(dev), bf16_activations=True)
    ref_loss = torch.nn.functional.l1_loss(out, tt.permute(0, 3, 1, 2))
    ref_loss.backward()
    ref = np.concatenate([p.grad.detach().float().cpu().numpy().ravel() for c in model.convs for p in (c.weight, c.bias)])
    assert abs(float(loss.value) - float(ref_loss.item())) <= 1e-3 * float(ref_loss.item())
    cos = float(np.dot(got, ref) / (np.linalg.norm(got) * np.linalg.norm(ref)))
    assert cos > 0.999, cos
    off = 0
    for li, (ci, co) in enumerate(denoiser.LAYERS):
        nw = co * ci * 9
        g, r = got[off:off + nw], ref[off:off + nw]
        rel = float(np.linalg.norm(g - r) / max(np.linalg.norm(r), 1e-12))
        assert rel < 0.05, f"layer {li}: weight gradient relative error {rel:.3e}"
        off += nw + co
