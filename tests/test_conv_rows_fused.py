"""The row form of the denoiser's convolution with its fused epilogues: pooling
at 32 and 48 channels, nearest upsampling and the training step's ReLU mask, in
networks wide enough that every resolution runs by rows (a width must fill five
eighths of its 128-pixel strips). Bounds as test_denoiser_unet,
test_denoiser_training and test_denoiser_conv."""
import ctypes as C

import numpy as np
import pytest

import test_denoiser_conv as conv
import test_denoiser_training as training
from helpers import pinhole, rig_of
from ray_tracing_gb300 import denoiser, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,cin,cout", [
    (1, 9, 257, 32, 48),
    (2, 5, 385, 32, 32),
    (1, 6, 513, 16, 64),
])
def test_last_strip_of_one_pixel(n, h, w, cin, cout):
    conv.test_conv3x3_matches_torch(n, h, w, cin, cout, 1, cout, 0)


@pytest.mark.parametrize("cameras,w,h", [
    (1, 324, 36),   # quarter resolution 81 wide: pooling and upsampling at both levels by rows
    (2, 320, 20),   # two images
    (1, 330, 37),   # odd sizes: pooled edges, upsampling by its own kernel
    (1, 326, 6),    # upsampling into half resolution by its own kernel, into the full one fused
    (3, 640, 4),
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


@pytest.mark.parametrize("n,h,w", [(1, 16, 320), (2, 12, 324), (1, 8, 640), (2, 20, 164)])
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
