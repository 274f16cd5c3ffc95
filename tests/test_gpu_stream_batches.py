"""Edges of a batch of streams: the groups in which the tensor maps of a ragged attention call travel (14, 64 or 120 sequences a launch), and
the slices in which a row of logits is searched for its greedy token (16, 4 or 1 CTAs a row)."""
import numpy as np
import pytest

from oracle import oracle as orc
from gpu_util import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [14, 15, 64, 65, 120, 121])
def test_ragged_attention_across_launch_groups(batch):
    import torch
    jb = pkg()
    g = torch.Generator(device="cuda")
    g.manual_seed(batch)
    L, kv, heads = 96, 2, 8
    codes = lambda: [torch.randint(-127, 128, (L, kv, 128), dtype=torch.int8, device="cuda", generator=g) for _ in range(batch)]
    scales = lambda: [torch.rand((L, kv), device="cuda", generator=g) * 0.02 for _ in range(batch)]
    k, v, ks, vs = codes(), codes(), scales(), scales()
    q = torch.randn((batch, heads, 128), device="cuda", generator=g).half()
    lengths = torch.from_numpy(np.random.Generator(np.random.PCG64(batch)).integers(1, L + 1, batch).astype(np.int32)).cuda()
    out = torch.zeros_like(q)
    plan = jb.AttnPlan(k, v, ks, vs, L, kv)
    plan.decode(out, q, lengths, heads, 128 ** -0.5, torch.cuda.current_stream())
    torch.cuda.synchronize()
    plan.close()
    for i, n in enumerate(lengths.tolist()):
        keys, values = ((c[i][:n].double() * s[i][:n, :, None].double()).transpose(0, 1).repeat_interleave(heads // kv, 0) for c, s in ((k, ks), (v, vs)))
        want = (torch.softmax(q[i][:, None].double() @ keys.transpose(1, 2) * 128 ** -0.5, -1) @ values)[:, 0]
        # integer dots over 16-bit fixed point: 2^-15 of the largest weight per key, then one fp16 rounding
        bound = 2.0 ** -10 * want.abs() + 2.0 ** -11 * values.abs().amax(1)
        assert ((out[i].double() - want).abs() <= bound).all(), (i, n, float(((out[i].double() - want).abs() - bound).max()))


@pytest.mark.parametrize("streams,vocab", [(2, 2048), (31, 2050), (32, 2048), (147, 3000), (148, 2048)])
def test_greedy_token_of_every_stream(streams, vocab):
    import torch
    jb = pkg()
    m = orc.gen_model(81, n_layers=1, hidden=256, n_heads=2, n_kv=1, hd=128, ffn=512, vocab=vocab)
    d = jb.decoder.BatchDecoder(m["cfg"], jb.decoder.upload(m), 16, streams)
    prompts = np.random.Generator(np.random.PCG64(streams)).integers(0, vocab, (streams, 3)).astype(np.int32)
    st = torch.cuda.Stream()
    for n_new in (1, 3):                                   # the last token asked for is the argmax of the logits that are left
        got = d.generate(prompts, n_new, st)
        assert got.shape == (n_new, streams) and np.array_equal(got[-1], np.argmax(d.logits().float().cpu().numpy(), 1))
    d.step_device(st)                                      # and a step goes on from there
    after = d.logits().float().cpu().numpy()
    full = d.generate(prompts, 4, st)
    assert np.array_equal(full[:3], got) and np.array_equal(full[3], np.argmax(after, 1))
    assert jb.device_status(st) == 0
    d.close()
