"""N-sharded linear with the all_gather fused into the matmul epilogue (peer stores), 2 GPUs."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs on one machine")
def test_sharded_matmul_allgather_two_ranks():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, NCCL_NVLS_ENABLE="0")
    res = subprocess.run([sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2",
                          "--master-addr", "127.0.0.1", "--master-port", "29541",
                          os.path.join(root, "tests", "peer_worker.py")], cwd=root, env=env, capture_output=True,
                         text=True, timeout=600)
    assert res.returncode == 0 and res.stdout.count("PEER-OK") == 2, res.stdout[-3000:] + res.stderr[-3000:]


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs on one machine")
def test_sharded_matmul_through_the_copy_kernel_two_ranks():
    """The same worker with B200Q_PUSH=1: prefill-size products store their block locally and
    peer_push_kernel moves it to the other rank and signals (the form chosen by default above four
    ranks); every gathered result is checked against the oracle as before."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, NCCL_NVLS_ENABLE="0", B200Q_PUSH="1")
    res = subprocess.run([sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2",
                          "--master-addr", "127.0.0.1", "--master-port", "29543",
                          os.path.join(root, "tests", "peer_worker.py")], cwd=root, env=env, capture_output=True,
                         text=True, timeout=600)
    assert res.returncode == 0 and res.stdout.count("PEER-OK") == 2, res.stdout[-3000:] + res.stderr[-3000:]


def test_bounded_wait_runs_out_and_is_reported():
    """A rank that never signals: the bounded wait of the exchange gives up after its limit (set to
    50 ms here), stores code 6 in the status word and lets the stream go on; the host-side check
    turns that into an exception and hands back a zeroed workspace.  Nothing is made to fault: the
    flag is simply never raised."""
    import ctypes
    import time

    from mlx_b200 import _lib, ops

    lib = _lib.load()
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    sync = torch.zeros(64, dtype=torch.int32, device="cuda")     # flag at word 0 (stays 0), epoch at word 32
    sync[32] = 2                                                 # two signals expected, none will come
    ws = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    ws[100] = 7                                                  # stale scratch that a later kernel would trip over
    status = ctypes.c_void_p(ws.data_ptr() + ws.numel() - 16)
    stream = torch.cuda.current_stream().cuda_stream
    lib.b200q_set_peer_wait_limit_ms(50)
    try:
        t0 = time.perf_counter()
        rc = lib.b200q_peer_wait(P(sync), ctypes.c_void_p(sync.data_ptr() + 128), status, ctypes.c_void_p(stream))
        assert rc == 0, _lib.last_error()
        with pytest.raises(ops.DeviceStatusError) as ei:
            ops.read_workspace_status(ws, stream, "peer exchange")
        waited = time.perf_counter() - t0
    finally:
        lib.b200q_set_peer_wait_limit_ms(0)
    assert ei.value.code == 6 and "peer" in str(ei.value)
    assert 0.02 < waited < 5.0, waited
    assert int(ws.to(torch.int32).sum()) == 0          # the check re-zeroed the workspace
    ops.read_workspace_status(ws, stream, "peer exchange")   # and the status is clear again
    # a wait whose flag is already there returns at once and reports nothing
    sync[0] = 2
    rc = lib.b200q_peer_wait(P(sync), ctypes.c_void_p(sync.data_ptr() + 128), status, ctypes.c_void_p(stream))
    assert rc == 0
    ops.read_workspace_status(ws, stream, "peer exchange")


class OneRank:
    """The buffers of an exchange with only this process in it (or with copies of the output in the place of other ranks' buffers):
    flag at word 0, epoch at word 32, the count of finished blocks at word 64."""

    def __init__(self, M, N_total, copies=1):
        self.sync = torch.zeros(96, dtype=torch.int32, device="cuda")
        self.y = torch.zeros(copies, M, N_total, dtype=torch.bfloat16, device="cuda")
        self.ws = torch.zeros(8 << 20, dtype=torch.uint8, device="cuda")

    def product(self, x, w, g, bits, col0=0, wait=False, wait_before_x=0):
        import ctypes

        from mlx_b200 import _lib
        lib, P = _lib.load(), lambda t, off=0: ctypes.c_void_p(t.data_ptr() + off)
        n, M, N, (copies, _, ld) = x.shape[-1], x.shape[0], w[0].shape[0], self.y.shape
        ys = (ctypes.c_void_p * copies)(*[self.y[i].data_ptr() for i in range(copies)])
        flags = (ctypes.c_void_p * copies)(*[self.sync.data_ptr()] * copies)
        _lib.check(lib.b200q_qmm_sharded_signal(P(x), P(w[0]), P(w[1]), P(w[2]), ys, copies, ld, col0, _lib.BF16, M, N, n, g, bits, flags,
                                                P(self.sync, 128), P(self.sync, 256), P(self.sync) if wait else None, wait_before_x, 0,
                                                P(self.ws), self.ws.numel(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))

    def check_status(self):
        from mlx_b200 import ops
        ops.read_workspace_status(self.ws, torch.cuda.current_stream().cuda_stream, "peer exchange")


def quantized(N, K, g, bits, seed):
    import mlx_b200 as mb
    G = torch.Generator(device="cuda").manual_seed(seed)
    return mb.quantize(torch.randn(N, K, generator=G, device="cuda", dtype=torch.bfloat16) * 0.02, g, bits)


@pytest.mark.parametrize("then_plain", (False, True))
@pytest.mark.parametrize("wait_before_x", (0, 1))
def test_a_peer_later_than_the_waits_inside_a_block(wait_before_x, then_plain):
    """The flag of the step before is raised after 1.2 s (by a copy: no kernel waits for another), within the limit for peers of 3 s
    but later than what the roles of a block wait for one another (0.65 s).  The rows of a block are more stages than its ring
    has, and with a second product behind it, under the promise of constant weights, that one has filled its own ring long before.
    Results and status are those of a punctual peer."""
    import time

    import mlx_b200 as mb
    from mlx_b200 import _lib, ops

    M, K, g, bits = 3, 4096, 64, 8
    N = 64 if then_plain else 14336   # 8 blocks, which leave the other SMs to the second product
    w, w2 = quantized(N, K, g, bits, 1), quantized(14336, K, g, bits, 2)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    r = OneRank(M, N)
    r.product(x, w, g, bits)
    ref, ref2 = r.y.clone(), mb.quantized_matmul(x, *w2, group_size=g, bits=bits)
    r.sync[32] += 2   # two signals more are expected
    late = (r.sync[:1] + 2).cpu().pin_memory()
    r.y.zero_()
    torch.cuda.synchronize()
    run, set_flag = torch.cuda.Stream(), torch.cuda.Stream()
    lib = _lib.load()
    lib.b200q_set_peer_wait_limit_ms(3000)
    lib.b200q_set_weights_constant(1)
    try:
        with torch.cuda.stream(run):
            r.product(x, w, g, bits, wait=True, wait_before_x=wait_before_x)
            y2 = mb.quantized_matmul(x, *w2, group_size=g, bits=bits) if then_plain else ref2
        time.sleep(1.2)
        early = not run.query()
        with torch.cuda.stream(set_flag):
            r.sync[:1].copy_(late, non_blocking=True)
        torch.cuda.synchronize()
    finally:
        lib.b200q_set_weights_constant(0)
        lib.b200q_set_peer_wait_limit_ms(0)
    assert early, "the product did not wait"
    r.check_status()
    ops.check_status()
    assert torch.equal(r.y, ref) and torch.equal(y2, ref2)


@pytest.mark.parametrize("bits,g", [(4, 64), (6, 32)])
@pytest.mark.parametrize("M", (1, 4))
def test_weights_requested_before_the_previous_kernel_has_ended(bits, g, M):
    """Under the promise of constant weights a product's weights are under way while the kernel that writes its x still runs: a chain
    of products, each the next one's x, and a buffer that another kernel fills right before."""
    import mlx_b200 as mb
    from mlx_b200 import _lib, ops

    K = 4096
    ws = [quantized(K, K, g, bits, s) for s in range(4)]
    xs = [torch.randn(M, K, device="cuda", dtype=torch.bfloat16) for _ in range(20)]
    buf = torch.empty_like(xs[0])

    def chain():
        out = []
        for x in xs:
            buf.copy_(x)
            h = buf
            for w in ws:
                h = mb.quantized_matmul(h, *w, group_size=g, bits=bits)
            out.append(h)
        return torch.stack(out)

    ref = chain()
    _lib.load().b200q_set_weights_constant(1)
    try:
        got = chain()
        torch.cuda.synchronize()
    finally:
        _lib.load().b200q_set_weights_constant(0)
    ops.check_status()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("bits,g,M,K", [(3, 64, 8, 1152), (5, 128, 16, 2304), (6, 32, 4, 640), (6, 64, 1, 4352), (2, 32, 3, 384), (4, 64, 5, 1152)])
def test_output_and_signal_of_every_form_of_the_decode_kernel(bits, g, M, K):
    """Columns of a wider output in three buffers at once, twice in a row with the wait for the step before inside the second launch (whose
    flag is there): every buffer, nothing beside the columns, one signal per launch and buffer."""
    import mlx_b200 as mb

    N, N_total, col0 = 200, 328, 96
    assert mb.qmm_kernel_name(torch.bfloat16, M, N, K, g, bits) == "qmv_rows"
    w = quantized(N, K, g, bits, bits)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    r = OneRank(M, N_total, copies=3)
    r.y.fill_(7)
    ref = mb.quantized_matmul(x, *w, group_size=g, bits=bits)
    r.product(x, w, g, bits, col0=col0)
    r.product(x, w, g, bits, col0=col0, wait=True, wait_before_x=1)
    r.check_status()
    for y in r.y:
        assert torch.equal(y[:, col0:col0 + N], ref)
        assert (y[:, :col0] == 7).all() and (y[:, col0 + N:] == 7).all()
    assert int(r.sync[0]) == 6 and int(r.sync[32]) == 6 and int(r.sync[64]) == 0
