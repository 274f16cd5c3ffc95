"""Single precision: products over many tokens at the edges of their tiles (64 rows, 16 / 32 / 64 tokens, K tiles of 32 and 64, unaligned rows), and
attention at the edges of the runs of keys that a warp requests together (4 warps, 8 keys up to heads of 128, 4 up to 256, one beyond)."""
import numpy as np
import pytest

from gpu_util import pkg

pytestmark = pytest.mark.gpu


def pad8(n):
    return (n + 7) // 8 * 8


@pytest.mark.parametrize("M,N,K", [(64, 2, 64), (63, 15, 8), (65, 16, 31), (130, 17, 65), (66, 33, 130), (9600, 32, 33), (9602, 63, 40), (19200, 64, 36), (19201, 130, 100)])
@pytest.mark.parametrize("glu", [False, True])
@pytest.mark.parametrize("aligned", [True, False])
def test_products(M, N, K, glu, aligned):
    import torch
    jb = pkg()
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N)
    def rows(n):                                          # [n][pad8(K)], zero beyond K; not aligned: one element further on than a 16-byte boundary
        t = torch.zeros(n * pad8(K) + 4, device="cuda")[(0 if aligned else 1):][:n * pad8(K)].reshape(n, pad8(K))
        t[:, :K] = torch.randn((n, K), device="cuda", generator=g)
        return t
    W, V, x = rows(M), rows(M), rows(N)
    y = torch.full((N + 1, M), 7.0, device="cuda")
    jb.dense_matmul(y, W, x, M, N, K, W_up=V if glu else None)
    a, size = x.double() @ W.double().T, x.double().abs() @ W.double().abs().T
    # K roundings of at most 2^-24 of the sum of magnitudes, in whatever order the terms are added
    bound = K * 2.0 ** -24 * size
    if glu:
        b, sb = x.double() @ V.double().T, x.double().abs() @ V.double().abs().T
        silu = a * torch.sigmoid(a)
        # |silu'| < 1.1, and a few roundings of expf, the division and the products
        bound = 1.1 * bound * b.abs() + silu.abs() * K * 2.0 ** -24 * sb + 2.0 ** -20 * (silu * b).abs() + 1e-30
        a = silu * b
    assert ((y[:N].double() - a).abs() <= bound).all()
    assert (y[N] == 7).all()


@pytest.mark.parametrize("counts", [[0, 16, 17, 0, 33, 1], [300, 0, 0, 0], [5] * 20, [0] * 31 + [40] + [0] * 32 + [17, 0, 3], [1] * 33, [3] * 31 + [500, 2] + [0] * 64 + [16],
                                    [0] * 63 + [900]])
def test_grouped_products(counts):
    import torch
    jb = pkg()
    M, K, N, G = 70, 72, sum(counts), len(counts)
    g = torch.Generator(device="cuda")
    g.manual_seed(G)
    W, x = torch.randn((G * M, K), device="cuda", generator=g), torch.randn((N, K), device="cuda", generator=g)
    off = torch.from_numpy(np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)).cuda()
    y = torch.zeros((N, M), device="cuda")
    jb.dense_matmul(y, W, x, M, N, K, group_offsets=off, n_groups=G)
    for i in range(G):
        s, w = slice(int(off[i]), int(off[i + 1])), W[i * M:(i + 1) * M].double()
        assert ((y[s].double() - x[s].double() @ w.T).abs() <= K * 2.0 ** -24 * (x[s].double().abs() @ w.abs().T)).all()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (127, 128), (136, 128), (256, 250), (264, 264)])
def test_attention_of_few_keys(dim, vdim, dtype):
    import torch
    jb = pkg()
    H, G, most = 4, 2, 70
    g = torch.Generator(device="cuda")
    g.manual_seed(dim)
    t = getattr(torch, dtype)
    k, v = (torch.randn((most, G, d), device="cuda", generator=g).to(t) for d in (dim, vdim))
    q = torch.randn((1, H * dim), device="cuda", generator=g).to(t)
    for n in (1, 3, 4, 5, 15, 16, 17, 31, 32, 33, 64, 65, 70):
        out = torch.zeros((1, pad8(H * vdim)), dtype=t, device="cuda")
        jb.sink_attention(out, q, k, v, H, G, dim, vdim, dim ** -0.5, seq_len=n, n_splits=1)
        keys, values = (c[:n].double().transpose(0, 1).repeat_interleave(H // G, 0) for c in (k, v))
        want = (torch.softmax(q.double().reshape(H, 1, dim) @ keys.transpose(1, 2) * dim ** -0.5, -1) @ values).reshape(-1)
        assert (out[0, :H * vdim].double() - want).abs().max() < (3e-6 if dtype == "float32" else 1.5e-2) * max(1.0, float(want.abs().max())), n
