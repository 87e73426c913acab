"""rtgb_trainer_step refuses an input that is not 16-byte aligned, whichever form
of the convolution the width takes, and the trainer stays usable."""
import ctypes as C

import numpy as np
import pytest

import test_denoiser_training as training
from ray_tracing_gb300 import abi, denoiser

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(8, 40), (8, 320), (128, 1024)])  # by tiles; by tiles; by rows
@pytest.mark.parametrize("shift", [1, 4])     # elements of two bytes
def test_misaligned_input_is_refused(h, w, shift):
    torch = pytest.importorskip("torch")
    torch.manual_seed(3)
    flat = denoiser.flatten(denoiser.build_model()).astype(np.float32)
    n = 1
    x, t = training._batch(np.random.default_rng(5), n, h, w)
    dev = torch.device("cuda", 0)
    flat_x = torch.from_numpy(training._blocked(x)).to(dev).to(torch.bfloat16).reshape(-1)
    room = torch.zeros(flat_x.numel() + 8, dtype=torch.bfloat16, device=dev)
    tt = torch.from_numpy(t).to(dev).contiguous()
    lib, tr = training._trainer(torch, flat, n, h, w)
    try:
        room[shift:shift + flat_x.numel()] = flat_x
        torch.cuda.synchronize()
        loss = C.c_float()
        st = lib.rtgb_trainer_step(tr, C.c_void_p(room[shift:].data_ptr()), C.c_void_p(tt.data_ptr()), 1e-3, C.byref(loss))
        assert abi.STATUS_NAMES[st] == "RUNTIME_ERROR"
        params = np.empty_like(flat)
        assert lib.rtgb_trainer_params(tr, params.ctypes.data) == 0
        assert np.array_equal(params, flat)
        st = lib.rtgb_trainer_step(tr, C.c_void_p(flat_x.data_ptr()), C.c_void_p(tt.data_ptr()), 0.0, C.byref(loss))
        assert st == 0, lib.rtgb_trainer_last_error(tr)
        assert np.isfinite(loss.value)
    finally:
        lib.rtgb_trainer_destroy(tr)
