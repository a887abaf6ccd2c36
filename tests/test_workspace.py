"""Scratch buffers of the operator front-end: what a captured graph uses stays its own."""
import contextlib
import types
import weakref

import pytest
import torch

import mlx_b200 as mb
from mlx_b200 import ops


def test_an_outgrown_buffer_stays(monkeypatch):
    """Kernels of a CUDA graph keep the address of the buffer that was there at capture."""
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=7))
    monkeypatch.setattr(torch.cuda, "device", lambda dev: contextlib.nullcontext())
    told = []
    monkeypatch.setattr(ops, "_front", types.SimpleNamespace(scratch=lambda *a: told.append(a)))
    spaces, dev = ops._Workspaces(), torch.device("cpu:0")
    first = weakref.ref(spaces.get(dev, 1000, "qmm"))
    assert spaces.get(dev, 1001, "qmm").numel() >= 2000
    assert first() is not None and first().numel() == 1000
    last = spaces.get(dev, 5000, "qmm")
    assert told[-1][3:] == (last.data_ptr(), last.numel())
    assert sum(b.numel() for _, b in spaces.all()) <= 2 * last.numel()


@pytest.mark.gpu
def test_graph_replay_after_the_workspace_has_grown():
    """A decode step (whose kernel keeps counters and partial sums in its workspace) is captured; then a prompt goes
    through the same layer, which needs a larger one; the memory around is written; the step must replay as before."""
    N, K, bits, g = 4000, 1280, 6, 64
    G = torch.Generator(device="cuda").manual_seed(0)
    w = mb.quantize(torch.randn(N, K, generator=G, device="cuda", dtype=torch.bfloat16) * 0.02, g, bits)
    x = torch.randn(16, K, generator=G, device="cuda", dtype=torch.bfloat16)
    long = torch.randn(700, K, generator=G, device="cuda", dtype=torch.bfloat16)
    assert mb.qmm_kernel_name(torch.bfloat16, 16, N, K, g, bits) == "qmv_mma"
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        ref = mb.quantized_matmul(x, *w, group_size=g, bits=bits)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            y = mb.quantized_matmul(x, *w, group_size=g, bits=bits)
        before = ops._workspaces.get(x.device, 0, "qmm").numel()
        mb.quantized_matmul(long, *w, group_size=g, bits=bits)
        ops._workspaces.get(x.device, before + 1, "qmm")
        others = [torch.full((before,), 0x55, dtype=torch.uint8, device="cuda") for _ in range(8)]
        graph.replay()
    st.synchronize()
    assert torch.allclose(y.float(), ref.float(), rtol=1e-2, atol=1e-2 * float(ref.float().abs().max()))
    assert all(int((o != 0x55).sum()) == 0 for o in others)


@pytest.mark.gpu
@pytest.mark.parametrize("transpose", (True, False))
def test_first_tensor_core_call_of_a_thread_inside_a_capture(transpose):
    import threading

    M, N, K = 64, 256, 256
    G = torch.Generator(device="cuda").manual_seed(1)
    w = mb.quantize(torch.randn(N, K, generator=G, device="cuda", dtype=torch.bfloat16) * 0.02)
    x = torch.randn(M, N if not transpose else K, generator=G, device="cuda", dtype=torch.bfloat16)
    ref = mb.quantized_matmul(x, *w, transpose=transpose)
    torch.cuda.synchronize()
    out, errors = [], []

    def capture():
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                out.append(mb.quantized_matmul(x, *w, transpose=transpose))
            graph.replay()
            torch.cuda.synchronize()
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    t = threading.Thread(target=capture)
    t.start()
    t.join()
    assert not errors, errors
    assert torch.equal(out[0], ref)
