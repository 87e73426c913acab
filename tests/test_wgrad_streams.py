"""Weight gradients on several streams at once: every call has partials of its
own, so results equal a serial run's bit for bit (the sums have a fixed order;
128 input channels, whose bias sums are atomic, are left out)."""
import ctypes as C

import numpy as np
import pytest

from ray_tracing_gb300 import abi

pytestmark = pytest.mark.gpu

LAYERS = [(4, 100, 110, 80, 32), (6, 96, 130, 64, 64), (2, 64, 64, 16, 16)]  # n, h, w, c_in, c_out


def test_calls_in_flight_on_several_streams():
    torch = pytest.importorskip("torch")
    lib, dev = abi.load(), torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(1)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    data = []
    for n, h, w, cin, cout in LAYERS:
        x = torch.randn((n, cin // 8, h, w, 8), generator=g, device=dev).to(torch.bfloat16)
        dy = torch.randn((n, cout // 8, h, w, 8), generator=g, device=dev).to(torch.bfloat16)
        data.append((x, dy))

    def call(k, dw, db, stream):
        n, h, w, cin, cout = LAYERS[k]
        msg = C.create_string_buffer(256)
        st = lib.rtgb_conv3x3_wgrad_bf16(data[k][0].data_ptr(), n, h, w, cin, data[k][1].data_ptr(), cout, dw.data_ptr(),
                                         db.data_ptr(), err.data_ptr(), C.c_void_p(stream.cuda_stream), msg, 256)
        assert st == 0, msg.value.decode()

    def outputs():
        return [(torch.zeros((cout, cin, 3, 3), device=dev), torch.zeros(cout, device=dev)) for _, _, _, cin, cout in LAYERS]

    want = outputs()
    for k, (dw, db) in enumerate(want):
        call(k, dw, db, torch.cuda.current_stream(dev))
        torch.cuda.synchronize(dev)
    streams = [torch.cuda.Stream(dev) for _ in LAYERS]
    got = [outputs() for _ in range(8)]
    torch.cuda.synchronize(dev)
    for out in got:
        for k, stream in enumerate(streams):
            call(k, *out[k], stream)
    torch.cuda.synchronize(dev)
    assert int(err.item()) == 0
    for out in got:
        for (dw, db), (want_w, want_b) in zip(out, want):
            assert np.array_equal(dw.cpu().numpy(), want_w.cpu().numpy())
            assert np.array_equal(db.cpu().numpy(), want_b.cpu().numpy())


def test_captured_call():
    """A call captured into a graph owns its partials there."""
    torch = pytest.importorskip("torch")
    lib, dev = abi.load(), torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(2)
    n, h, w, cin, cout = LAYERS[1]
    x = torch.randn((n, cin // 8, h, w, 8), generator=g, device=dev).to(torch.bfloat16)
    dy = torch.randn((n, cout // 8, h, w, 8), generator=g, device=dev).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    results = []

    def call(dw, db):
        msg = C.create_string_buffer(256)
        stream = torch.cuda.current_stream(dev).cuda_stream
        st = lib.rtgb_conv3x3_wgrad_bf16(x.data_ptr(), n, h, w, cin, dy.data_ptr(), cout, dw.data_ptr(), db.data_ptr(),
                                         err.data_ptr(), C.c_void_p(stream), msg, 256)
        assert st == 0, msg.value.decode()

    for captured in (False, True):
        dw, db = torch.zeros((cout, cin, 3, 3), device=dev), torch.zeros(cout, device=dev)
        torch.cuda.synchronize(dev)
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                call(dw, db)
            for _ in range(3):
                graph.replay()
        else:
            call(dw, db)
        torch.cuda.synchronize(dev)
        results.append((dw.cpu().numpy(), db.cpu().numpy()))
    assert int(err.item()) == 0
    assert all(np.array_equal(a, b) for a, b in zip(*results))
