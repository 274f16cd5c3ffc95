"""GPU parity of the batched K-quant GEMM (prefill) against the oracle and the reference's own
golden vectors (tests/golden/q4k_int8.npz, q6k_int8.npz)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import oracle as orc
from gpu_util import pkg, dev, close, close_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,M,N,K", [(12, 128, 16, 512), (12, 130, 7, 1024), (12, 64, 65, 2560), (14, 128, 16, 512), (14, 33, 9, 2560),
                                      (14, 20, 3, 9728), (13, 16, 3, 512),
                                      # several output tiles per persistent CTA, ragged last row / token tile, every token-tile width
                                      (12, 300, 300, 2560), (14, 260, 270, 1024), (12, 1, 2, 256), (14, 129, 33, 256), (12, 257, 129, 768),
                                      (12, 40000, 40, 256), (14, 19000, 70, 512),
                                      # more output tiles than SMs: whole rounds, then the leftover tiles cut into K ranges (ragged edges)
                                      (12, 2500, 2000, 2048), (14, 2500, 1999, 1024)])
def test_gemm_quant_batched_matches_oracle(t, M, N, K):
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1003 + M + N))
    W = orc.gen_weight(rng, t, M, K)
    X = orc.gen_act(rng, N * K)
    y = torch.zeros(N * M, dtype=torch.float16, device="cuda")
    jb.gemm_quant_batched(y, dev(W), t, dev(X), M, N, K)
    want = orc.entry_gemm_quant_batched(W, t, X, M, N, K).astype(np.float32).reshape(-1)
    ok, md = close_gemm(y.float().cpu().numpy(), want, N, M)
    assert ok, md


# weights expanded once for many tokens: the first size that takes that way and its neighbours, ragged rows (groups of four, and not), K ranges of tail tiles,
# a last row tile that is mostly beyond the matrix, a matrix in two pieces
WIDE = [(12, 300, 383, 512), (12, 300, 384, 768), (14, 300, 384, 512), (12, 515, 385, 512), (14, 513, 400, 768), (12, 256, 511, 2560), (14, 772, 390, 4096), (12, 66000, 384, 512),
        # fewer than 2048 rows: from 448 tokens on
        (12, 300, 447, 768), (12, 300, 448, 768), (12, 515, 449, 512), (14, 513, 450, 768), (14, 772, 460, 4096), (14, 2047, 448, 512), (14, 2048, 384, 512)]
# few tokens: every number of token tiles, one row, rows that do not fill a tile, one super-block, more super-blocks than ranges
FEW = [(t, M, N, K) for t in (12, 14) for M, N, K in ((40, 8, 512), (16, 9, 256), (2500, 17, 2560), (100, 25, 768), (33, 33, 9728), (1000, 41, 1024), (18, 48, 5120), (70, 49, 512), (64, 64, 2560), (17, 2, 4096),
                                              # token tiles dealt to two and to four CTAs, and not
                                              (1024, 12, 2560), (1024, 40, 2560), (1024, 57, 2560), (512, 31, 256), (2360, 32, 256), (2384, 32, 2560), (4096, 48, 2560))]


@pytest.mark.parametrize("t,M,N,K", WIDE + FEW)
def test_gemm_of_many_and_of_few_tokens(t, M, N, K):
    test_gemm_quant_batched_matches_oracle(t, M, N, K)


@pytest.mark.parametrize("t,M,N,K", [(12, 40, 5, 768), (14, 24, 6, 512)])
def test_gemm_integer_accumulators_bit_exact(t, M, N, K):
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1004 + M))
    W = orc.gen_weight(rng, t, M, K)
    X = orc.gen_act(rng, N * K)
    G = K // 32 if t == 12 else K // 16
    dots = torch.zeros((N, M, G), dtype=torch.int32, device="cuda")
    y = torch.zeros(N * M, dtype=torch.float16, device="cuda")
    jb.gemm_quant_batched_int_dots(y, dots, dev(W), t, dev(X), M, N, K)
    assert np.array_equal(dots.cpu().numpy(), orc.mmq_int_dots(W, t, X, M, N, K))


@pytest.mark.parametrize("name,t", [("q4k_int8.npz", 12), ("q6k_int8.npz", 14)])
def test_reference_golden_vectors(golden_dir, name, t):
    """The reference's own acceptance bar for its int8 GEMM: every |Δ| <= 0.5 against its int8 host model
    (tests/test_mmq_q4k_int8.cu:533-541, tests/test_mmq_q6k_int8.cu:298-310)."""
    import torch
    jb = pkg()
    g = np.load(os.path.join(golden_dir, name))
    M, N, K = map(int, g["shape"])
    y = torch.zeros(N * M, dtype=torch.float16, device="cuda")
    jb.gemm_quant_batched(y, dev(g["W"]), t, dev(g["X"].view(np.float16)), M, N, K)
    ref = g["Y_int8"].view(np.float16).astype(np.float32)
    assert np.max(np.abs(y.float().cpu().numpy() - ref)) <= 0.5


@pytest.mark.parametrize("t,M,N,K", [(12, 9728, 48, 2560), (14, 2560, 48, 9728), (12, 9728, 64, 2560), (14, 2560, 64, 9728), (12, 4096, 64, 2560),
                                      (12, 4096, 8, 2560), (14, 1024, 24, 2560), (12, 2560, 2, 4096), (14, 151, 57, 768)])
def test_few_tokens_stream_the_weights_once(t, M, N, K):
    """2..64 tokens go through the weight-streaming kernel (csrc/mmq_stream.cu): the decoder's own shapes at 48 and 64 streams
    (the two largest matrices at 64 streams are handed to the tensor-core kernel, which is faster there), every token-tile
    count, ragged row and token edges, and K ranges split over CTAs (few rows, long K)."""
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1007 + M + N))
    W = orc.gen_weight(rng, t, M, K)
    X = orc.gen_act(rng, N * K)
    y = torch.full((N * M,), float("nan"), dtype=torch.float16, device="cuda")
    jb.gemm_quant_batched(y, dev(W), t, dev(X), M, N, K)
    want = orc.entry_gemm_quant_batched(W, t, X, M, N, K).astype(np.float32).reshape(-1)
    ok, md = close_gemm(y.float().cpu().numpy(), want, N, M)
    assert ok, md
    assert jb.device_status() == 0


@pytest.mark.parametrize("t,M0,M1,N,K", [(12, 300, 200, 100, 1024), (14, 130, 257, 70, 512), (12, 2500, 2300, 1000, 1024), (12, 9728, 9728, 64, 2560),
                                          (12, 96, 64, 8, 512)])
def test_two_products_over_the_same_activations(t, M0, M1, N, K):
    """gemm_quant_batched_pair (the gate and up projections of a batched layer): both outputs against the oracle.  The shapes
    cover the shared launch of the tensor-core kernel with ragged row tiles of both matrices, more tiles than SMs (whole
    rounds plus split tail tiles that belong to either matrix), the decoder's own pair at 64 streams, and the few-token
    path (two launches)."""
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1010 + M0 + N))
    W0 = orc.gen_weight(rng, t, M0, K); W1 = orc.gen_weight(rng, t, M1, K)
    X = orc.gen_act(rng, N * K)
    y0 = torch.full((N * M0,), float("nan"), dtype=torch.float16, device="cuda")
    y1 = torch.full((N * M1,), float("nan"), dtype=torch.float16, device="cuda")
    jb.gemm_quant_batched_pair(y0, dev(W0), t, M0, y1, dev(W1), t, M1, dev(X), N, K)
    for y, W, M in ((y0, W0, M0), (y1, W1, M1)):
        want = orc.entry_gemm_quant_batched(W, t, X, M, N, K).astype(np.float32).reshape(-1)
        ok, md = close_gemm(y.float().cpu().numpy(), want, N, M)
        assert ok, md
    assert jb.device_status() == 0


@pytest.mark.parametrize("t", [12, 14])
def test_tensor_core_and_cuda_core_paths_agree(t):
    """The tcgen05 kernel and the CUDA-core kernel (the one that exports the integer accumulators) compute the same
    quantised product; they differ by the fp16 rounding of the operand products only."""
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1006 + t))
    M, N, K = 200, 48, 1536
    W = dev(orc.gen_weight(rng, t, M, K)); X = dev(orc.gen_act(rng, N * K))
    G = K // 32 if t == 12 else K // 16
    dots = torch.zeros((N, M, G), dtype=torch.int32, device="cuda")
    a = torch.zeros(N * M, dtype=torch.float16, device="cuda"); b = torch.zeros_like(a)
    jb.gemm_quant_batched(a, W, t, X, M, N, K)
    jb.gemm_quant_batched_int_dots(b, dots, W, t, X, M, N, K)
    ok, md = close_gemm(a.float().cpu().numpy(), b.float().cpu().numpy(), N, M)
    assert ok, md
    assert jb.device_status() == 0


def test_n_equal_one_routes_to_gemv():
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1005))
    M, K = 77, 1024
    W = dev(orc.gen_weight(rng, 12, M, K)); x = dev(orc.gen_act(rng, K))
    a = torch.zeros(M, dtype=torch.float16, device="cuda"); b = torch.zeros_like(a)
    jb.gemm_quant_batched(a, W, 12, x, M, 1, K)
    jb.gemv_quant(b, W, 12, x, M, K)
    assert torch.equal(a, b)


def test_captured_product_replays_after_larger_calls():
    """A caller's own graph holds the address of the product's scratch: replayed after calls that ask for more of it, it gives what it gave before."""
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1011))
    M, K = 1024, 1024
    W = dev(orc.gen_weight(rng, 12, M, K))
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    for N in (8, 100, 400):
        with torch.cuda.stream(st):
            X = dev(orc.gen_act(rng, N * K))
            y = torch.zeros(N * M, dtype=torch.float16, device="cuda")
            jb.gemm_quant_batched(y, W, 12, X, M, N, K, stream=st)
            torch.cuda.synchronize()
            want = y.clone()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                jb.gemm_quant_batched(y, W, 12, X, M, N, K, stream=st)
            for n in (800 + N, 2000 + N):
                big = torch.zeros(n * M, dtype=torch.float16, device="cuda")
                jb.gemm_quant_batched(big, W, 12, torch.ones(n * K, dtype=torch.float16, device="cuda"), M, n, K, stream=st)
            keep = [torch.full((1 << i,), 0x5A, dtype=torch.uint8, device="cuda") for i in range(18, 27)]
            y.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, want), N
            del keep, g
    assert jb.device_status() == 0


def _stream_products(jb, seed, sizes, W, M, K, st):
    """(launch, outputs): launch() enqueues one product per size on st."""
    import torch
    rng = np.random.Generator(np.random.PCG64(seed))
    with torch.cuda.stream(st):
        xs = [dev(orc.gen_act(rng, n * K)) for n in sizes]
        ys = [torch.zeros(n * M, dtype=torch.float16, device="cuda") for n in sizes]
    def launch():
        for n, x, y in zip(sizes, xs, ys):
            jb.gemm_quant_batched(y, W, 12, x, M, n, K, stream=st)
    return launch, ys


@pytest.mark.parametrize("count,threads", [(2, False), (40, False), (4, True)])
def test_products_on_several_streams_at_once(count, threads):
    """Products of every path (few tokens, fused, expanded) on several streams at the same time, more of them than the library keeps scratch for, and from
    several threads: the bits of each stream's products run alone."""
    import threading
    import torch
    jb = pkg()
    M, K, sizes = 4096, 2560, (512, 8, 100, 400, 30)
    W = dev(orc.gen_weight(np.random.Generator(np.random.PCG64(1012)), 12, M, K))
    torch.cuda.synchronize()
    # not torch.cuda.Stream: it hands out 32 streams in turn
    import ctypes
    rt = ctypes.CDLL("libcudart.so")
    handles = []
    for _ in range(count):
        h = ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(h), 1) == 0
        handles.append(h)
    work = [_stream_products(jb, 1013 + i, sizes, W, M, K, torch.cuda.ExternalStream(h.value)) for i, h in enumerate(handles)]
    want = []
    for launch, ys in work:
        launch()
        torch.cuda.synchronize()
        want.append([y.clone() for y in ys])
        for y in ys:
            y.zero_()
    torch.cuda.synchronize()
    for _ in range(3):
        if threads:
            ts = [threading.Thread(target=launch) for launch, _ in work]
            for t in ts: t.start()
            for t in ts: t.join()
        else:
            for launch, _ in work:
                launch()
        torch.cuda.synchronize()
        for (_, ys), w in zip(work, want):
            assert all(torch.equal(a, b) for a, b in zip(ys, w))
    assert jb.device_status() == 0


def test_two_sessions_prompt_at_once():
    """Prompts of two decoder sessions on two streams, long enough for the expanded weights, give what they give one after the other."""
    import torch
    jb = pkg()
    m = orc.gen_model(81, n_layers=2, hidden=1024, n_heads=8, n_kv=2, hd=128, ffn=2048, vocab=512)
    w = jb.decoder.upload(m)
    st = [torch.cuda.Stream() for _ in range(2)]
    d = [jb.decoder.Decoder(m["cfg"], w, 1600, jb.decoder.FUSED | jb.decoder.PREFILL) for _ in range(2)]
    prompts = [np.random.Generator(np.random.PCG64(1300 + i)).integers(0, 512, n) for i, n in enumerate((1500, 700))]
    torch.cuda.synchronize()
    want = []
    for i in range(2):
        d[i].prefill(prompts[i], 0, st[i])
        want.append(d[i].logits().clone())
    for _ in range(4):
        for i in range(2):
            d[i].prefill(prompts[i], 0, st[i])
        assert all(torch.equal(d[i].logits(), want[i]) for i in range(2))
    for x in d:
        x.close()
    assert jb.device_status() == 0


def test_a_second_session_takes_over_the_expanded_weights():
    """Two buffers of expanded weights and the sums of split products are the stream's, not a session's: 147 MB more for each session otherwise."""
    import torch
    jb = pkg()
    m = orc.gen_model(83, n_layers=1, hidden=512, n_heads=4, n_kv=1, hd=128, ffn=1024, vocab=512)
    w = jb.decoder.upload(m)
    prompt = np.random.Generator(np.random.PCG64(83)).integers(0, 512, 600)
    sessions, taken, logits = [], [], []
    for _ in range(4):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        d = jb.decoder.Decoder(m["cfg"], w, 700, jb.decoder.FUSED | jb.decoder.PREFILL)
        d.prefill(prompt, 0, torch.cuda.Stream())
        logits.append(d.logits())
        taken.append(free - torch.cuda.mem_get_info()[0])
        sessions.append(d)
    # caches of 700 positions and buffers of 600 tokens: a few MB, in whole 2 MB pieces of the driver's
    assert all(t < 32 << 20 for t in taken[1:]), taken
    assert all(torch.equal(l, logits[0]) for l in logits)
    for d in sessions:
        d.close()
    assert jb.device_status() == 0


def test_a_second_session_takes_over_the_scratch_of_short_prompts():
    """Operands and partial sums of a prompt of few tokens are the stream's too (10 MB at these widths)."""
    import torch
    jb = pkg()
    m = orc.gen_model(85, n_layers=1, hidden=512, n_heads=4, n_kv=1, hd=128, ffn=8192, vocab=512)
    w = jb.decoder.upload(m)
    prompt = np.random.Generator(np.random.PCG64(85)).integers(0, 512, 100)
    sessions, taken, logits = [], [], []
    for _ in range(4):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        d = jb.decoder.Decoder(m["cfg"], w, 128, jb.decoder.FUSED | jb.decoder.PREFILL)
        d.prefill(prompt, 0, torch.cuda.Stream())
        logits.append(d.logits())
        taken.append(free - torch.cuda.mem_get_info()[0])
        sessions.append(d)
    assert all(t < 6 << 20 for t in taken[1:]), taken
    assert all(torch.equal(l, logits[0]) for l in logits)
    for d in sessions:
        d.close()
    assert jb.device_status() == 0


@pytest.mark.parametrize("lengths", [(640, 500), (640, 60), (60, 100)])
def test_two_sessions_prompt_on_one_stream_from_two_threads(lengths):
    """A chunk has its expansions, operands and partial sums in buffers of the stream: a session on the same stream in another thread waits its turn."""
    import threading
    import torch
    jb = pkg()
    m = orc.gen_model(84, n_layers=3, hidden=1024, n_heads=8, n_kv=2, hd=128, ffn=2048, vocab=512)
    w = jb.decoder.upload(m)
    st = torch.cuda.Stream()
    d = [jb.decoder.Decoder(m["cfg"], w, 700, jb.decoder.FUSED | jb.decoder.PREFILL) for _ in range(2)]
    prompts = [np.random.Generator(np.random.PCG64(1400 + i)).integers(0, 512, n) for i, n in enumerate(lengths)]
    want = []
    for i in range(2):
        d[i].prefill(prompts[i], 0, st)
        want.append(d[i].logits().clone())
    for _ in range(10):
        ts = [threading.Thread(target=lambda i=i: [d[i].prefill(prompts[i], 0, st) for _ in range(5)]) for i in range(2)]
        for t in ts: t.start()
        for t in ts: t.join()
        assert all(torch.equal(d[i].logits(), want[i]) for i in range(2))
    for x in d:
        x.close()
    assert jb.device_status(st) == 0


def test_capture_on_another_stream_than_the_warm_up():
    """A product captured on a stream that has no scratch yet: refused while the device has not seen a call that asked for as much (in a process of its own),
    else the graph gives the uncaptured result, by the expanded path too."""
    code = """
import numpy as np, torch
from oracle import oracle as orc
from gpu_util import pkg, dev
jb = pkg()
jb.lib.jllm_b200_init(-1)
M, K = 1024, 512
W = dev(orc.gen_weight(np.random.Generator(np.random.PCG64(9)), 14, M, K))
def graph(N, x, y):
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    rc = 0
    with torch.cuda.graph(g, stream=st):
        try:
            jb.gemm_quant_batched(y, W, 14, x, M, N, K, stream=st)
        except jb.JllmError as e:
            rc = e.code
    return g, rc
for N in (40, 200, 500):
    x, y = dev(orc.gen_act(np.random.Generator(np.random.PCG64(N)), N * K)), torch.zeros(N * M, dtype=torch.float16, device="cuda")
    g, rc = graph(N, x, y)
    assert rc == 5, (N, rc)
    jb.gemm_quant_batched(y, W, 14, x, M, N, K)
    torch.cuda.synchronize()
    want = y.clone()
    y.zero_()
    g, rc = graph(N, x, y)
    assert rc == 0, (N, rc, jb.last_error())
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want), N
assert jb.device_status() == 0
"""
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here])))
    assert r.returncode == 0, r.stderr[-2000:]


def test_products_beside_another_threads_capture():
    """Products on new streams, one of which needs more scratch than there is, while another thread captures: both are as they are alone."""
    import ctypes
    import threading
    import torch
    jb = pkg()
    M, K = 1024, 1024
    rng = np.random.Generator(np.random.PCG64(1014))
    W = dev(orc.gen_weight(rng, 12, M, K))
    rt, sizes = ctypes.CDLL("libcudart.so"), (30, 500, 6000)
    xs, ys = [dev(orc.gen_act(rng, n * K)) for n in sizes], [torch.zeros(n * M, dtype=torch.float16, device="cuda") for n in sizes]
    x, y = dev(orc.gen_act(rng, 40 * K)), torch.zeros(40 * M, dtype=torch.float16, device="cuda")
    jb.gemm_quant_batched(y, W, 12, x, M, 40, K)
    torch.cuda.synchronize()
    want, failed, handles = y.clone(), [], [ctypes.c_void_p() for _ in sizes]
    assert all(rt.cudaStreamCreateWithFlags(ctypes.byref(h), 1) == 0 for h in handles)
    torch.cuda.synchronize()
    def other():
        try:
            for n, a, b, h in zip(sizes, xs, ys, handles):
                jb.gemm_quant_batched(b, W, 12, a, M, n, K, stream=h.value)
        except Exception as e:
            failed.append(e)
    g, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=st):
        t = threading.Thread(target=other)
        t.start()
        t.join()
        jb.gemm_quant_batched(y, W, 12, x, M, 40, K, stream=st)
    assert not failed, failed
    torch.cuda.synchronize()
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    for n, a, b in zip(sizes, xs, ys):
        again = torch.zeros_like(b)
        jb.gemm_quant_batched(again, W, 12, a, M, n, K)
        torch.cuda.synchronize()
        assert torch.equal(again, b), n
    assert jb.device_status() == 0
