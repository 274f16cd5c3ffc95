"""GPU parity of decode / prefill attention over INT8 and FP16 KV against the CPU oracle (C ABI).
Bar: 1e-3 relative plus 2e-3 of the largest output magnitude of the head (fp16 outputs)."""
import numpy as np
import pytest

from oracle import oracle as orc
from gpu_util import pkg, dev

pytestmark = pytest.mark.gpu


def _check(got, want):
    got = np.asarray(got, np.float32).reshape(want.shape)
    want = np.asarray(want, np.float32)
    tol = 1e-3 * np.abs(want) + 2e-3 * np.abs(want).max(axis=-1, keepdims=True) + 1e-6
    assert np.all(np.abs(got - want) <= tol), float(np.abs(got - want).max())


@pytest.mark.parametrize("L", [1, 2, 63, 64, 65, 127, 128, 129, 255, 256, 1024, 4096])
def test_decode_int8_gqa(L):
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(1002 + L))
    nh, nkv, hd = 32, 8, 128
    q = orc.gen_act(rng, nh * hd)
    k, ks = orc.gen_kv(rng, L, nkv, hd)
    v, vs = orc.gen_kv(rng, L, nkv, hd)
    out = torch.zeros(nh * hd, dtype=torch.float16, device="cuda")
    jb.flash_attention_decode(out, dev(q), dev(k), dev(v), nh, nkv, hd, hd, L, float(1 / np.sqrt(hd)), True, dev(ks), dev(vs), 0)
    _check(out.cpu().numpy(), orc.attention_decode(q, k, v, nh, nkv, hd, L, 1 / np.sqrt(hd), True, ks, vs))
    assert jb.device_status() == 0


@pytest.mark.parametrize("nh,nkv,hd,L,window,int8", [(8, 8, 64, 300, 0, False), (16, 2, 128, 500, 0, False), (8, 1, 256, 200, 64, True),
                                                      (4, 4, 128, 700, 128, False), (32, 8, 128, 2000, 0, True)])
def test_decode_general_shapes(nh, nkv, hd, L, window, int8):
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(nh * hd + L))
    q = orc.gen_act(rng, nh * hd)
    if int8:
        k, ks = orc.gen_kv(rng, L, nkv, hd); v, vs = orc.gen_kv(rng, L, nkv, hd)
        args = (dev(k), dev(v)); sc = (dev(ks), dev(vs))
    else:
        k = (rng.standard_normal((L, nkv, hd)) * 0.5).astype(np.float16); v = (rng.standard_normal((L, nkv, hd)) * 0.5).astype(np.float16)
        ks = vs = None
        args = (dev(k), dev(v)); sc = (None, None)
    out = torch.zeros(nh * hd, dtype=torch.float16, device="cuda")
    jb.flash_attention_decode(out, dev(q), args[0], args[1], nh, nkv, hd, hd, L, float(1 / np.sqrt(hd)), int8, sc[0], sc[1], window)
    _check(out.cpu().numpy(), orc.attention_decode(q, k, v, nh, nkv, hd, L, 1 / np.sqrt(hd), int8, ks, vs, window))


def test_decode_dyn_and_prefill_and_batched():
    import torch
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(77))
    nh, nkv, hd, L = 32, 8, 128, 333
    scale = float(1 / np.sqrt(hd))
    q = orc.gen_act(rng, nh * hd)
    k, ks = orc.gen_kv(rng, L, nkv, hd); v, vs = orc.gen_kv(rng, L, nkv, hd)
    kd, vd, ksd, vsd = dev(k), dev(v), dev(ks), dev(vs)
    want = orc.attention_decode(q, k, v, nh, nkv, hd, L, scale, True, ks, vs)
    out = torch.zeros(nh * hd, dtype=torch.float16, device="cuda")
    d_pos = torch.tensor([L - 1], dtype=torch.int32, device="cuda")
    # the _dyn variant takes ONE scale pointer used for K and V (attention.cu:1024); check with vs == ks
    want_dyn = orc.attention_decode(q, k, v, nh, nkv, hd, L, scale, True, ks, ks)
    for ns in (1, 4):
        jb.get_splitk_partials(nh, ns, hd)
        jb.flash_attention_decode_dyn(out, dev(q), kd, vd, nh, nkv, hd, hd, d_pos, scale, True, ksd, 0, ns)
        _check(out.cpu().numpy(), want_dyn)
    # prefill: N queries, causal
    N, start = 7, L - 7
    qs = orc.gen_act(rng, N * nh * hd)
    outp = torch.zeros(N * nh * hd, dtype=torch.float16, device="cuda")
    jb.flash_attention_prefill_batched(outp, dev(qs), kd, vd, nh, nkv, hd, hd, N, start, scale, True, ksd, vsd, 0)
    _check(outp.cpu().numpy(), orc.attention_prefill(qs, k, v, nh, nkv, hd, N, start, scale, True, ks, vs).reshape(N * nh, hd))
    # ragged batch == loop over the single-sequence entry point
    B = 5
    lens = rng.integers(1, 600, B).astype(np.int32)
    seqs = [(orc.gen_kv(rng, int(l), nkv, hd), orc.gen_kv(rng, int(l), nkv, hd)) for l in lens]
    qb = orc.gen_act(rng, B * nh * hd)
    kt = [dev(s[0][0]) for s in seqs]; vt = [dev(s[1][0]) for s in seqs]; kst = [dev(s[0][1]) for s in seqs]; vst = [dev(s[1][1]) for s in seqs]
    mk = lambda ts: torch.tensor([t.data_ptr() for t in ts], dtype=torch.int64, device="cuda")
    outb = torch.zeros(B * nh * hd, dtype=torch.float16, device="cuda")
    jb.flash_attention_decode_batched(outb, dev(qb), mk(kt), mk(vt), mk(kst), mk(vst), dev(lens), B, int(lens.max()), nh, nkv, hd, scale, True)
    qbd = dev(qb)
    for b in range(B):
        one = torch.zeros(nh * hd, dtype=torch.float16, device="cuda")
        jb.flash_attention_decode(one, qbd[b * nh * hd:(b + 1) * nh * hd], kt[b], vt[b], nh, nkv, hd, hd, int(lens[b]), scale, True, kst[b], vst[b], 0)
        _check(outb[b * nh * hd:(b + 1) * nh * hd].cpu().numpy(), one.float().cpu().numpy().reshape(nh, hd))
        (kk, kks), (vv, vvs) = seqs[b]
        _check(one.cpu().numpy(), orc.attention_decode(qb[b * nh * hd:(b + 1) * nh * hd], kk, vv, nh, nkv, hd, int(lens[b]), scale, True, kks, vvs))


def test_attention_argument_errors():
    import torch
    jb = pkg()
    out = torch.zeros(128, dtype=torch.float16, device="cuda")
    with pytest.raises(jb.JllmError):
        jb.flash_attention_decode(out, out, out, out, 3, 2, 64, 64, 4, 1.0, False, None, None, 0)     # heads not a multiple of kv heads
    with pytest.raises(jb.JllmError):
        jb.flash_attention_decode(out, out, None, out, 2, 2, 64, 64, 4, 1.0, False, None, None, 0)    # null cache


@pytest.mark.parametrize("N,start,nh,nkv", [(1, 0, 32, 8), (5, 0, 32, 8), (33, 0, 32, 8), (64, 17, 32, 8), (130, 300, 32, 8), (37, 5, 16, 8), (9, 2, 8, 8)])
def test_prefill_int8_query_tiled(N, start, nh, nkv):
    """Causal prefill over an INT8 cache with 128-wide heads (the query-tiled tensor-core kernel): token t at position
    start + t attends keys [0, start + t]; ragged token counts, non-zero start, GQA groups of 4, 2 and 1."""
    import torch
    jb = pkg()
    hd = 128
    rng = np.random.Generator(np.random.PCG64(5000 + N + start + nh))
    L = start + N
    scale = float(1 / np.sqrt(hd))
    q = orc.gen_act(rng, N * nh * hd)
    k, ks = orc.gen_kv(rng, L, nkv, hd); v, vs = orc.gen_kv(rng, L, nkv, hd)
    out = torch.full((N * nh * hd + 64,), 7.0, dtype=torch.float16, device="cuda")
    jb.flash_attention_prefill_batched(out, dev(q), dev(k), dev(v), nh, nkv, hd, hd, N, start, scale, True, dev(ks), dev(vs), 0)
    got = out.float().cpu().numpy()
    assert np.all(got[N * nh * hd:] == 7.0), "wrote past the output"
    _check(got[:N * nh * hd], orc.attention_prefill(q, k, v, nh, nkv, hd, N, start, scale, True, ks, vs).reshape(N * nh, hd))
    assert jb.device_status() == 0


@pytest.mark.parametrize("N", [33, 512])
def test_prefill_int8_matches_reference_gpu_record(N):
    """The same kernel against what the reference's own prefill attention returned on a B200 (tests/golden/ref_gpu.npz)."""
    import os
    import torch
    from golden import gpu_cases as gc
    jb = pkg()
    ref = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "ref_gpu.npz"))
    c = gc.attention_prefill(N)
    out = torch.zeros(N * gc.NH * gc.HD, dtype=torch.float16, device="cuda")
    jb.flash_attention_prefill_batched(out, dev(c["q"]), dev(c["k"]), dev(c["v"]), gc.NH, gc.NKV, gc.HD, gc.HD, N, 0, gc.SCALE, True, dev(c["ks"]), dev(c["vs"]), 0)
    sel = gc.prefill_sample(N)
    got = out.float().cpu().numpy().reshape(N, gc.NH, gc.HD)[sel].reshape(-1, gc.HD)
    want = ref[f"prefill_attn_N{N}_out"].view(np.float16).astype(np.float32).reshape(-1, gc.HD)
    _check(got, want)


def _prompt_on_a_workspace(jb, q, k, ks, v, vs, nh, nkv, N, start):
    import torch
    out = torch.full((N * nh * 128 + 64,), 7.0, dtype=torch.float16, device="cuda")
    ws = torch.full((jb.flash_attention_prefill_workspace_bytes(nkv, start + N),), 0x7F, dtype=torch.uint8, device="cuda")      # 0x7F7F: NaN in fp16
    n0 = jb.launch_count()
    jb.flash_attention_prefill_workspace(out, dev(q), dev(k), dev(v), nh, nkv, 128, 128, N, start, float(1 / np.sqrt(128)), True, dev(ks), dev(vs), 0, ws)
    widened = N >= 64 if nh // nkv > 4 else N >= 64 and N * nkv >= 2048  # elsewhere the kernel over the codes is the faster one
    assert jb.launch_count() - n0 == (2 if widened else 1)
    got = out.float().cpu().numpy()
    assert np.all(got[N * nh * 128:] == 7.0), "wrote past the output"
    return got[:N * nh * 128].reshape(N, nh, 128)


# groups of 1 .. 128 query heads, row tiles of 128 / group tokens and their neighbours, a start inside a key tile, counts around 64, several turns of the
# five-stage key ring
@pytest.mark.parametrize("N,start,nh,nkv", [(63, 0, 32, 32), (64, 130, 32, 32), (65, 0, 32, 32), (129, 300, 16, 16), (512, 0, 4, 4), (255, 0, 32, 8), (256, 0, 32, 8), (257, 63, 32, 8),
                                            (300, 1000, 32, 8), (256, 100, 16, 8), (130, 63, 32, 16), (2048, 0, 2, 1), (64, 0, 16, 2), (127, 37, 16, 2), (100, 2000, 16, 2),
                                            (70, 500, 16, 1), (66, 64, 64, 2), (64, 130, 128, 1), (65, 1, 128, 1)])
def test_prefill_int8_on_a_workspace(N, start, nh, nkv):
    """Causal prefill over an INT8 cache whose codes are widened into a workspace (the tcgen05 kernel where it gains), to the tolerance of the other kernels.
    The keys of the last quarter are long: scores rise late and by far more than the 2^8 up to which a maximum is kept."""
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(6000 + 7 * N + start + nh))
    L = start + N
    q = orc.gen_act(rng, N * nh * 128)
    k, ks = orc.gen_kv(rng, L, nkv, 128); v, vs = orc.gen_kv(rng, L, nkv, 128)
    ks[3 * L // 4:] *= 12
    got = _prompt_on_a_workspace(jb, q, k, ks, v, vs, nh, nkv, N, start)
    _check(got, orc.attention_prefill(q, k, v, nh, nkv, 128, N, start, 1 / np.sqrt(128), True, ks, vs))
    assert jb.device_status() == 0


def test_prefill_workspace_arguments():
    import torch
    jb = pkg()
    t, f = torch.zeros(64 * 4 * 128, dtype=torch.float16, device="cuda"), torch.zeros(64 * 4, dtype=torch.float32, device="cuda")
    c = torch.zeros(64 * 4 * 128, dtype=torch.int8, device="cuda")
    need = jb.flash_attention_prefill_workspace_bytes(4, 64)
    for ws in (torch.zeros(need - 1, dtype=torch.uint8, device="cuda"), torch.zeros(need + 1, dtype=torch.uint8, device="cuda")[1:]):
        with pytest.raises(jb.JllmError) as e:
            jb.flash_attention_prefill_workspace(t, t, c, c, 4, 4, 128, 128, 64, 0, 1.0, True, f, f, 0, ws)
        assert e.value.code == 1
    a, b = torch.ones_like(t), torch.ones_like(t)                        # no workspace: the call without one
    q = dev(orc.gen_act(np.random.Generator(np.random.PCG64(1)), 64 * 4 * 128))
    jb.flash_attention_prefill_workspace(a, q, c, c, 4, 4, 128, 128, 64, 0, 1.0, True, f, f, 0, None)
    jb.flash_attention_prefill_batched(b, q, c, c, 4, 4, 128, 128, 64, 0, 1.0, True, f, f, 0)
    assert torch.equal(a, b)


@pytest.mark.parametrize("late,nh,nkv", [(1, 32, 8), (70, 8, 8), (299, 16, 2)])
def test_prefill_int8_is_not_spoiled_by_later_tokens(late, nh, nkv):
    """A token whose values overflowed (an infinite scale) leaves the tokens before it as they were, bit for bit, and is not hidden from those that see it."""
    jb = pkg()
    rng = np.random.Generator(np.random.PCG64(6500 + late))
    N = 300
    q = orc.gen_act(rng, N * nh * 128)
    k, ks = orc.gen_kv(rng, N, nkv, 128); v, vs = orc.gen_kv(rng, N, nkv, 128)
    clean = _prompt_on_a_workspace(jb, q, k, ks, v, vs, nh, nkv, N, 0)
    for a in (vs, ks):
        keep = a[late, nkv - 1]
        a[late, nkv - 1] = np.inf
        got = _prompt_on_a_workspace(jb, q, k, ks, v, vs, nh, nkv, N, 0)
        a[late, nkv - 1] = keep
        assert np.array_equal(got[:late], clean[:late])
        hit = got[late:, nh - nh // nkv:]
        assert not np.isfinite(hit).all() and np.array_equal(got[late:, :nh - nh // nkv], clean[late:, :nh - nh // nkv])
    assert jb.device_status() == 0
