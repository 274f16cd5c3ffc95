"""Products of a few tokens (2..128: prompt chunks and lock-step streams) on the split-by-units tensor-core kernel, and longer chunks whose
kernels between the products write the next product's operand, against the kernels that serve weights these do not take (a Q6_K matrix that
starts at an odd multiple of two bytes).

Both sides build the same fp16 operands and sum them in fp32 in another order.  What that may do: a key, formed by one product from
identical operands, differs by the last fp16 bit of a few values, which moves a cache code by one at most and its head's scale by 2^-10
of itself.  Further on, one such bit re-rounds the codes of a group of activations (tests/test_gpu_batch_decoder.py: error RMS 0.05 and
maximum 0.43 of the logit RMS against the oracle over the streams of a model of this size), so their logits are held to that file's
bounds; the logits of one token, where a flipped group weighs more than in the mean over streams, to the error RMS of 0.15 that
tests/test_gpu_decoder.py derives for them."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import oracle as orc
from gpu_util import pkg, ulp16

pytestmark = pytest.mark.gpu

ERR_RMS, ERR_MAX, ONE_TOKEN_RMS = 0.08, 0.6, 0.15
# super-blocks of a row, in the order hidden, heads' outputs, MLP: Q6_K rows of 1, 2, 4 and 8 to a multiple of 16 bytes; tiles cut off at their last rows
SHAPES = {
    "even": dict(n_layers=2, hidden=512, n_heads=4, n_kv=2, hd=128, ffn=1024, vocab=2048),
    "odd": dict(n_layers=2, hidden=768, n_heads=6, n_kv=2, hd=128, ffn=1280, vocab=1000),
    "whole": dict(n_layers=1, hidden=2048, n_heads=2, n_kv=1, hd=128, ffn=2048, vocab=2056),
    # the norms' forms: up to 32, 64 and 128 tiles of a token, up to 32 and 64 super-blocks, the last warps with fewer
    "w4096": dict(n_layers=1, hidden=4096, n_heads=2, n_kv=1, hd=128, ffn=512, vocab=512),
    "w4352": dict(n_layers=1, hidden=4352, n_heads=2, n_kv=1, hd=128, ffn=512, vocab=512),
    "w8448": dict(n_layers=1, hidden=8448, n_heads=2, n_kv=1, hd=128, ffn=512, vocab=512),
}


def weights(shape, swap):
    """The model's weights on the device; swap: Q6_K where the benchmark's mix has Q4_K and the other way round."""
    c = dict(SHAPES[shape])
    m = orc.gen_model(5, **c)
    if swap:
        r = np.random.Generator(np.random.PCG64(6))
        four = lambda rows, K: (orc.gen_q4k(r, rows, K, orc.model_sigma(orc.Q4_K, K), orc.MODEL_MIN_RATIO), orc.Q4_K)
        six = lambda rows, K: (orc.gen_q6k(r, rows, K, orc.model_sigma(orc.Q6_K, K)), orc.Q6_K)
        H, Q, KV, I = c["hidden"], c["n_heads"] * 128, c["n_kv"] * 128, c["ffn"]
        for lw in m["layers"]:
            lw.update(wq=six(Q, H), wk=six(KV, H), wv=four(KV, H), wo=six(H, Q), gate=six(I, H), up=four(I, H), down=four(H, I))
    return m["cfg"], pkg().decoder.upload(m)


def elsewhere(w):
    """The same weights with one Q6_K matrix two bytes further on: taken by the general kernels alone."""
    import torch
    w = dict(w, layers=[dict(l) for l in w["layers"]])
    name = next(n for n in ("wv", "wq") if w["layers"][0][n][1] == orc.Q6_K)
    for l in w["layers"]:
        t = l[name][0].reshape(-1)
        buf = torch.empty(t.numel() + 16, dtype=torch.uint8, device="cuda")
        buf[2:2 + t.numel()] = t
        l[name] = (buf[2:2 + t.numel()], l[name][1])
    return w


def shifted(v):
    """The vector one element further on than a 16-byte boundary."""
    import torch
    buf = torch.empty(v.numel() + 4, dtype=v.dtype, device="cuda")
    buf[1:1 + v.numel()] = v
    return buf[1:1 + v.numel()]


def device_bytes(ptr, n):
    import torch
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    C.CDLL("libcudart.so").cudaMemcpy(C.c_void_p(out.data_ptr()), C.c_void_p(ptr), C.c_size_t(n), 3)
    return out.cpu().numpy()


def first_keys(d, n, kv):
    """Key codes [n][kv][128] and scales [n][kv] of the first layer."""
    buf = pkg().lib.jllm_b200_decoder_buffer
    buf.restype = C.c_void_p
    return (device_bytes(buf(C.c_void_p(d._h), 7), n * kv * 128).view(np.int8).reshape(n, kv, 128).astype(np.int32),
            device_bytes(buf(C.c_void_p(d._h), 8), n * kv * 4).view(np.float32).reshape(n, kv))


def check_logits(got, want, bound):
    rms = float(np.sqrt(np.mean(want ** 2)))
    err = np.abs(got - want)
    print("logit error: max %.4f, rms %.4f of the logit RMS" % (float(err.max()) / rms, float(np.sqrt(np.mean(err ** 2))) / rms))
    assert np.isfinite(got).all() and np.sqrt(np.mean(err ** 2)) <= bound * rms and err.max() <= ERR_MAX * rms


def chunk_as_the_general_kernels(cfg, w, n):
    """A prompt of n tokens by both sides: key codes and scales of the first layer, logits."""
    import torch
    jb = pkg()
    prompt = np.random.Generator(np.random.PCG64(n)).integers(0, cfg["vocab"], n)
    kv = cfg["n_kv_heads"]
    sides = []
    for ws in (w, elsewhere(w)):
        d = jb.decoder.Decoder(cfg, ws, 512, jb.decoder.FUSED | jb.decoder.PREFILL)
        st = torch.cuda.Stream()
        n0 = jb.launch_count()
        d.prefill(prompt, 0, st)
        launches = jb.launch_count() - n0
        codes, scales = first_keys(d, n, kv)
        sides.append((codes, scales, d.logits().cpu().numpy().astype(np.float64), launches))
        assert jb.device_status(st) == 0
        d.close()
    (codes, scales, logits, few), (codes0, scales0, logits0, many) = sides
    assert few < many                                      # the general kernels need a launch for every quantiser, sum and residual
    assert np.all(np.abs(scales - scales0) <= 2.0 ** -10 * np.abs(scales0))
    assert np.abs(codes - codes0).max() <= 1 and np.mean(codes != codes0) <= 0.05
    check_logits(logits, logits0, ONE_TOKEN_RMS)


# padded to 16 tokens; two accumulators up to 48, three super-blocks of weights in tensor memory up to 96, two above, two accumulators again up to 112
@pytest.mark.parametrize("shape,swap", [("even", False), ("odd", False), ("odd", True), ("whole", False)])
# beyond 128: rows of many tokens, tiles of 32..256 tokens with and without K ranges, and from 384 or 448 on the expanded weights
@pytest.mark.parametrize("n", [2, 16, 17, 48, 49, 96, 97, 112, 113, 128, 129, 257, 450])
def test_prompt_chunk_as_the_general_kernels(shape, swap, n):
    chunk_as_the_general_kernels(*weights(shape, swap), n)


@pytest.mark.parametrize("shape", ["w4096", "w4352", "w8448"])
@pytest.mark.parametrize("n", [17, 129])
def test_wide_models(shape, n):
    chunk_as_the_general_kernels(*weights(shape, False), n)


@pytest.mark.parametrize("n", [17, 129])
@pytest.mark.parametrize("neox,norms", [(0, True), (0, False), (1, False)])
def test_adjacent_pairs_and_heads_without_norms(monkeypatch, neox, norms, n):
    """rope_neox = 0 turns adjacent elements; models without head norms give null vectors."""
    jb = pkg()

    class Desc(jb.decoder.ModelDesc):
        def __setattr__(self, name, value):
            super().__setattr__(name, neox if name == "rope_neox" else value)

    monkeypatch.setattr(jb.decoder, "ModelDesc", Desc)
    cfg, w = weights("odd", False)
    if not norms:
        w["layers"] = [{k: v for k, v in l.items() if k not in ("q_norm", "k_norm")} for l in w["layers"]]
    chunk_as_the_general_kernels(cfg, w, n)
    if n == 17:
        prompts = np.random.Generator(np.random.PCG64(3)).integers(0, cfg["vocab"], (5, 3)).astype(np.int32)
        streams_as_the_general_kernels(cfg, w, prompts)


@pytest.mark.parametrize("n,at", [(20, 7), (150, 100)])
def test_an_infinite_token_reaches_no_other_tokens_row(n, at):
    """Token `at` of a prompt is infinite: every other key of the first layer has the codes and the scale that it has without it."""
    import torch
    jb = pkg()
    cfg, w = weights("odd", False)
    bad = dict(w, tok_embd=(w["tok_embd"][0].clone(), w["tok_embd"][1]))
    bad["tok_embd"][0].reshape(cfg["vocab"], -1, 144)[3, 1, 0:2] = torch.tensor([0x00, 0x7C], dtype=torch.uint8, device="cuda")      # an infinite block scale of token 3
    prompt = np.random.Generator(np.random.PCG64(n)).integers(4, cfg["vocab"], n)
    prompt[at] = 3
    st = torch.cuda.Stream()
    sides = []
    for ws in (w, bad):
        d = jb.decoder.Decoder(cfg, ws, 512, jb.decoder.FUSED | jb.decoder.PREFILL)
        d.prefill(prompt, 0, st)
        sides.append(first_keys(d, n, cfg["n_kv_heads"]))
        assert jb.device_status(st) == 0
        d.close()
    others = np.arange(n) != at
    assert all(np.array_equal(a[others], b[others]) for a, b in zip(*sides))
    assert not np.array_equal(sides[0][0][at], sides[1][0][at])


def test_an_infinite_stream_reaches_no_other_stream():
    import torch
    jb = pkg()
    cfg, w = weights("odd", False)
    bad = dict(w, tok_embd=(w["tok_embd"][0].clone(), w["tok_embd"][1]))
    bad["tok_embd"][0].reshape(cfg["vocab"], -1, 144)[3, 1, 0:2] = torch.tensor([0x00, 0x7C], dtype=torch.uint8, device="cuda")
    prompts = np.random.Generator(np.random.PCG64(9)).integers(4, cfg["vocab"], (19, 3)).astype(np.int32)
    prompts[5, 1] = 3
    st = torch.cuda.Stream()
    sides = []
    for ws in (w, bad):
        d = jb.decoder.BatchDecoder(cfg, ws, 16, 19)
        tokens = d.generate(prompts, 1, st)
        sides.append((d.logits(), tokens))
        assert jb.device_status(st) == 0
        d.close()
    others = torch.arange(19, device="cuda") != 5
    assert torch.equal(sides[0][0][others], sides[1][0][others])
    assert not torch.isfinite(sides[1][0][5]).any() and sides[1][1][0, 5] == 0      # no logit is a candidate: token 0


# output matrices of Q6_K rows of 2, 3 and 8 super-blocks and of Q4_K ones; fewer units than SMs, and tiles that two and three CTAs share
@pytest.mark.parametrize("hidden,vocab,q4", [(512, 2048, False), (768, 24000, False), (768, 1000, True), (2048, 2056, False), (1024, 20000, True)])
@pytest.mark.parametrize("streams", [2, 17, 128])
def test_logits_product_over_known_activations(hidden, vocab, q4, streams):
    """Layers that add nothing and tokens of small whole numbers, whose norm is the same in any order of summation: the logits are the output product over
    activations that the stand-alone product can be given bit for bit."""
    import torch
    jb = pkg()
    m = orc.gen_model(11, n_layers=1, hidden=hidden, n_heads=2, n_kv=1, hd=128, ffn=256, vocab=vocab)
    w = jb.decoder.upload(m)
    r = np.random.Generator(np.random.PCG64(12))
    if q4:
        w["output"] = (torch.from_numpy(orc.gen_q4k(r, vocab, hidden, orc.model_sigma(orc.Q4_K, hidden), orc.MODEL_MIN_RATIO)).cuda(), orc.Q4_K)
    for name in ("wo", "down"):
        w["layers"][0][name][0].zero_()
    embed = torch.randint(0, 256, (vocab * hidden // 256, 144), dtype=torch.uint8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(13))
    embed[:, :16] = torch.tensor([0x00, 0x3C, 0, 0] + [1] * 4 + [0] * 4 + [1] * 4, dtype=torch.uint8, device="cuda")      # d = 1, dmin = 0, scales 1: a weight is its code
    w["tok_embd"] = (embed.reshape(-1), orc.Q4_K)
    prompts = r.integers(0, vocab, (streams, 1)).astype(np.int32)
    st = torch.cuda.Stream()
    d = jb.decoder.BatchDecoder(m["cfg"], w, 8, streams)
    d.generate(prompts, 1, st)
    got = d.logits().double().cpu().numpy()
    assert jb.device_status(st) == 0
    d.close()
    codes = embed.reshape(vocab, -1, 144)[torch.from_numpy(prompts[:, 0].astype(np.int64)).cuda()][..., 16:].reshape(streams, -1, 4, 32)
    x = torch.cat([codes & 15, codes >> 4], -1).reshape(streams, hidden).half()
    normed, y = torch.empty_like(x), torch.zeros((streams, vocab), dtype=torch.float16, device="cuda")
    jb.fused_rmsnorm_residual(normed, x, None, w["out_norm"], streams, hidden, m["cfg"]["eps"], 1)
    jb.gemm_quant_batched(y, w["output"][0], w["output"][1], normed, vocab, streams, hidden)
    torch.cuda.synchronize()
    want = y.double().cpu().numpy()
    # the same fp16 operands, summed in fp32 in another order: hidden 2^-24 of the sum of magnitudes, which is sqrt(hidden) of an output's size or so
    # (2.4e-3 of the RMS at 2048), and each side rounds to fp16; a super-block too many or too few is 0.3 of it at least
    rms = np.sqrt(np.mean(want ** 2))
    assert (np.abs(got - want) <= 2 * ulp16(want) + hidden ** 1.5 * 2.0 ** -24 * rms).all(), np.abs(got - want).max() / rms


def test_a_chunk_of_one_token_keeps_its_integer_products():
    """Three tokens in chunks of two: the last one alone.  Its key codes of the first layer are those of the general kernels, bit for bit."""
    import torch
    jb = pkg()
    cfg, w = weights("odd", False)
    st = torch.cuda.Stream()
    kv, sides = cfg["n_kv_heads"], []
    for ws in (w, elsewhere(w)):
        d = jb.decoder.Decoder(cfg, ws, 64, jb.decoder.FUSED | jb.decoder.PREFILL)
        d.prefill(np.array([5, 6, 7]), 0, st, chunk=2)
        sides.append([a[2] for a in first_keys(d, 3, kv)])
        assert jb.device_status(st) == 0
        d.close()
    assert all(np.array_equal(a, b) for a, b in zip(*sides))


def streams_as_the_general_kernels(cfg, w, prompts):
    import torch
    jb = pkg()
    sides, kernels = [], []
    for ws in (w, elsewhere(w)):
        d = jb.decoder.BatchDecoder(cfg, ws, 16, len(prompts))
        st = torch.cuda.Stream()
        d.generate(prompts, 1, st)
        first = d.logits()
        d.generate(prompts, 1, st)
        assert torch.equal(first, d.logits())              # a session can be used again, and sums in a fixed order
        sides.append(first.double().cpu().numpy())
        kernels.append(d.kernels_per_step())
        assert jb.device_status(st) == 0
        d.close()
    assert kernels[0] < kernels[1]                         # the two sides are two ways
    check_logits(*sides, ERR_RMS)


@pytest.mark.parametrize("shape,swap,streams", [("even", False, 2), ("odd", True, 33), ("odd", False, 96), ("whole", False, 128), ("even", True, 113), ("w4352", False, 9)])
def test_streams_as_the_general_kernels(shape, swap, streams):
    cfg, w = weights(shape, swap)
    streams_as_the_general_kernels(cfg, w, np.random.Generator(np.random.PCG64(streams)).integers(0, cfg["vocab"], (streams, 3)).astype(np.int32))


@pytest.mark.parametrize("name", ["rms_attn", "rms_ffn", "q_norm", "k_norm", "out_norm"])
def test_norm_vectors_may_start_at_any_element(name):
    """The kernels between the products read norm vectors 16 bytes at a time: a model whose vectors start elsewhere stays with the general ones."""
    import torch
    jb = pkg()
    cfg, w = weights("even", False)
    moved = dict(w, layers=[dict(l, **({name: shifted(l[name])} if name in l else {})) for l in w["layers"]])
    if name == "out_norm":
        moved["out_norm"] = shifted(w["out_norm"])
    st = torch.cuda.Stream()
    for n in (20, 150):
        prompt = np.random.Generator(np.random.PCG64(n)).integers(0, cfg["vocab"], n)
        got = []
        for ws in (moved, elsewhere(w)):
            d = jb.decoder.Decoder(cfg, ws, 256, jb.decoder.FUSED | jb.decoder.PREFILL)
            d.prefill(prompt, 0, st)
            got.append(d.logits().cpu().numpy().astype(np.float64))
            assert jb.device_status(st) == 0
            d.close()
        check_logits(*got, ONE_TOKEN_RMS)
    prompts = np.random.Generator(np.random.PCG64(7)).integers(0, cfg["vocab"], (5, 3)).astype(np.int32)
    got = []
    for ws in (moved, elsewhere(w)):
        d = jb.decoder.BatchDecoder(cfg, ws, 16, 5)
        d.generate(prompts, 1, st)
        got.append(d.logits().double().cpu().numpy())
        assert jb.device_status(st) == 0
        d.close()
    check_logits(*got, ERR_RMS)


@pytest.mark.parametrize("name", ["rms_attn", "rms_ffn"])
def test_a_missing_norm_vector_is_refused(name):
    jb = pkg()
    cfg, w = weights("even", False)
    w = dict(w, layers=[dict(l) for l in w["layers"]])
    w["layers"][1][name] = None
    d = jb.decoder.Decoder(cfg, w, 256, jb.decoder.FUSED | jb.decoder.PREFILL)
    for n in (20, 150):
        with pytest.raises(jb.JllmError):
            d.prefill(np.zeros(n, np.int32), 0)
    d.close()
    d = jb.decoder.BatchDecoder(cfg, w, 16, 5)
    with pytest.raises(jb.JllmError):
        d.generate(np.zeros((5, 3), np.int32), 1)
    d.close()


@pytest.mark.parametrize("switch", ["JLLM_B200_MMQ_STREAM=0", "JLLM_B200_MMQ_PAIR=0", "JLLM_B200_MMQ=cuda", "JLLM_B200_MMQ_DEBUG=1"])
def test_switches_of_the_products_hold_for_sessions(switch):
    """A switch that chooses among the general kernels makes sessions run them, whatever the weights; the one that prints prints here too."""
    code = """
import numpy as np, torch
import test_gpu_mmq_few as t
jb = t.pkg()
cfg, w = t.weights("even", False)
st = torch.cuda.Stream()
for n in (20, 150):
    counts = []
    for ws in (w, t.elsewhere(w)):
        d = jb.decoder.Decoder(cfg, ws, 256, jb.decoder.FUSED | jb.decoder.PREFILL)
        n0 = jb.launch_count()
        d.prefill(np.arange(n, dtype=np.int32), 0, st)
        counts.append(jb.launch_count() - n0)
        d.close()
    b = []
    for ws in (w, t.elsewhere(w)):
        d = jb.decoder.BatchDecoder(cfg, ws, 8, 5)
        d.generate(np.zeros((5, 2), np.int32), 1, st)
        b.append(d.kernels_per_step())
        d.close()
    print("counts", *counts, *b)
assert jb.device_status(st) == 0
"""
    here = os.path.dirname(os.path.abspath(__file__))
    name, value = switch.split("=")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here]), **{name: value}))
    assert r.returncode == 0, r.stderr[-2000:]
    counts = [[int(x) for x in l.split()[1:]] for l in r.stdout.splitlines() if l.startswith("counts")]
    assert len(counts) == 2
    if name == "JLLM_B200_MMQ_DEBUG":
        assert "[mmq_few]" in r.stderr and all(c[0] < c[1] and c[2] < c[3] for c in counts)
    else:
        assert all(c[0] == c[1] and c[2] == c[3] for c in counts), counts
