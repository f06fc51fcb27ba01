"""The entries that hold no host memory past their return run inside a
caller's stream capture: the replayed graph computes what the call did."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
NT = 30


@pytest.mark.parametrize("name,nd,models,pre,grads", [
    ("Acoustic", 2, 1, "acoustic", 1), ("Acoustic3D", 3, 1, "acoustic", 1), ("Elastic", 2, 3, "elastic", 3),
    ("Elastic3D", 3, 3, "elastic3d", 3), ("AcousticVTI1st", 2, 4, "vti", 4), ("AcousticVTI1st3D", 3, 4, "vti3d", 4)])
def test_captured_call_replays(name, nd, models, pre, grads):
    import sweep_b200 as sb
    from sweep_b200 import _lib
    shape = (17, 15, 34) if nd == 3 else (17, 34)
    s = sb.PropTorch(getattr(sb, name)(spatial_order=4, device=DEV), shape=shape, dh=10.0, dt=5e-4, abcn=5, device=DEV)
    rng = np.random.default_rng(7)
    src, rec = rng.integers(3, 12, (3, nd)), rng.integers(0, 15, (3, 6, nd))
    vp = torch.tensor(2500 + 100 * rng.standard_normal(shape), dtype=torch.float32, device=DEV)
    ms = {1: [vp], 3: [vp, vp / 1.8, vp], 4: [vp, vp * 1e-4, vp * 5e-5, vp]}[models]
    geo, padded, _, fields = s._probe(NT, src, rec, ms)
    padded = [m.contiguous() for m in padded]
    wavelet = torch.tensor(rng.standard_normal((3, 1, NT)), dtype=torch.float32, device=DEV)
    desc = s._desc(geo, padded, wavelet, fields)
    ws_b, tape_b = _lib.c_i64(), _lib.c_i64()
    _lib.call(f"sweep_b200_{pre}_sizes", desc, _lib.MEM_BOUNDARY, 0, ws_b, tape_b)
    ws = torch.empty(ws_b.value, dtype=torch.uint8, device=DEV)
    tape = torch.empty(tape_b.value, dtype=torch.uint8, device=DEV)
    record = torch.empty((3, NT, 6, len(fields[1]) if fields else 1), device=DEV)
    adj = torch.tensor(rng.standard_normal(record.shape), dtype=torch.float32, device=DEV)
    out = [torch.empty_like(padded[0]) for _ in range(grads)]
    extra = [None] * 3 if models == 1 else []       # no wavelet gradient, no illumination

    def call():
        stream = torch.cuda.current_stream(DEV).cuda_stream
        _lib.call(f"sweep_b200_{pre}_forward", desc, _lib.MEM_BOUNDARY, 0, record.data_ptr(), tape.data_ptr(),
                  ws.data_ptr(), ws.numel(), stream)
        _lib.call(f"sweep_b200_{pre}_backward", desc, _lib.MEM_BOUNDARY, 0, adj.data_ptr(), tape.data_ptr(),
                  *[g.data_ptr() for g in out], *extra, ws.data_ptr(), ws.numel(), stream)

    call()
    torch.cuda.synchronize()
    want = [t.clone() for t in (record, *out)]
    assert all(float(t.abs().max()) > 0 for t in want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for _ in range(2):
        for t in (ws, tape, record, *out):
            t.fill_(0 if t.dtype == torch.uint8 else float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        for t, w in zip((record, *out), want):
            assert torch.allclose(t, w, rtol=1e-4, atol=1e-5 * float(w.abs().max()))   # atomics at shared cells
