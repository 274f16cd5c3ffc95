"""The memory's prompt kernels at the edges of their chunks (16 to 64 tokens in one, 128 in a row), their 64 dimensions and 32 value columns, and with values
that are not finite."""
import numpy as np
import pytest

from gpu_util import pkg
from oracle import delizen as orc
from test_gpu_delizen import f32, memory_case, zeros
from test_gpu_layered import as_np, pad8, rng, up

pytestmark = pytest.mark.gpu


def shifted(t, by):
    """The tensor `by` elements further on than a 16-byte boundary."""
    import torch
    buf = torch.empty(t.numel() + by, dtype=t.dtype, device="cuda")
    buf[by:] = t.reshape(-1)
    return buf[by:].reshape(t.shape)


def run(jb, q, k, v, zi, zf, cuts, shift=None):
    """raw outputs [T][H][V] and the state left behind; shift: elements by which raw, out and the norm's weights start off a 16-byte boundary"""
    T, H, D = q.shape
    V = v.shape[2]
    a, b = pad8(H * D), pad8(H * V)
    proj = np.zeros((T, 2 * a + 2 * b))
    proj[:, :H * D], proj[:, a:a + H * D], proj[:, 2 * a:2 * a + H * V] = q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)
    gates = np.zeros((T, pad8(2 * H)))
    gates[:, :H], gates[:, H:2 * H] = zi, zf
    pd, gd, bd, wd, state = up(proj, "bfloat16"), f32(gates), f32(np.zeros(2 * H), False), f32(np.ones(H * V), False), zeros(jb.mlstm_state_floats(H, D, V))
    got, at = [], 0
    for c in cuts:
        out, raw = zeros((c, b), "bfloat16"), zeros((c, H * V))
        if shift:
            raw, out, wd = shifted(raw, shift[0]), shifted(out, shift[1]), shifted(wd, shift[2])
        jb.mlstm(out, raw, state, pd[at:at + c].contiguous(), gd[at:at + c].contiguous(), bd, wd, H, D, V, 13.0, 1e-4, c, at)
        got.append(as_np(raw).reshape(c, H, V))
        if np.abs(got[-1]).max() < 1e15:                    # the kernel behind: head norms, and gates of a half
            x = got[-1] / np.sqrt((got[-1] ** 2).mean(2, keepdims=True) + 1e-4)
            assert np.abs(as_np(out).reshape(c, -1)[:, :H * V].reshape(c, H, V) - x / 2).max() <= 2.0 ** -8 * np.abs(x).max()
        at += c
    assert at == T
    return np.concatenate(got), as_np(state)


@pytest.mark.parametrize("H,D,V", [(1, 8, 8), (2, 64, 32), (1, 72, 40), (3, 128, 64), (2, 136, 24), (1, 192, 96), (1, 256, 72)])
@pytest.mark.parametrize("kind", ["plain", "drop", "far"])
@pytest.mark.parametrize("cuts", [[16], [17], [33], [64], [65], [127], [128], [129], [256, 16], [257, 383, 17], [64, 48, 100, 20]])
def test_edges(H, D, V, kind, cuts):
    jb, T = pkg(), sum(cuts)
    q, k, v, _, zi, zf = memory_case(rng(D + T), H, D, V, T, kind, "bfloat16")
    want = np.stack([orc.mlstm_memory(q[:, h] * D ** -0.5, k[:, h], v[:, h], orc.capped(zi[:, h], 13.0), orc.log_sigmoid(orc.capped(zf[:, h], 13.0)))[0] for h in range(H)], 1)
    got, _ = run(jb, q, k, v, zi, zf, cuts)
    assert (np.abs(got - want) / np.abs(want).max(axis=(0, 2))[None, :, None]).max() < 2e-4      # as in the general test: two bf16 parts, and n . q may cancel


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("T,at", [(300, 0), (300, 31), (300, 100), (300, 127), (300, 128), (300, 200), (50, 0), (50, 20), (50, 49), (64, 63), (16, 5)])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(T, at, value):
    jb = pkg()
    q, k, v, _, zi, zf = memory_case(rng(at), 2, 64, 40, T, "plain", "bfloat16")
    clean, _ = run(jb, q, k, v, zi, zf, [T])
    v = v.copy()
    v[at, 1, 33] = value
    got, _ = run(jb, q, k, v, zi, zf, [T])
    other = np.arange(40) != 33
    # the chunk's part is then added up in fp32 one token after the other: 2^-24 of up to 128 terms
    for a, b in ((got[:at], clean[:at]), (got[:, 0], clean[:, 0]), (got[:, 1, other], clean[:, 1, other])):
        assert np.isfinite(a).all() and np.abs(a - b).max(initial=0) <= 1e-4 * np.abs(clean).max()
    assert not np.isfinite(got[at:, 1, 33]).any()


@pytest.mark.parametrize("T", [30, 100, 200])
def test_weights_below_the_normal_numbers(T):
    """The first token alone meets every query, so much later that its weight is a subnormal number, and its values are large enough to show it."""
    jb, D, V = pkg(), 64, 32
    q, k, v = np.zeros((T, 1, D)), np.zeros((T, 1, D)), np.zeros((T, 1, V))
    q[:, 0, 0], k[0, 0, 0], k[1:, 0, 1], v[0] = 4.0, 1.0, 1.0, 2.0 ** 100
    # what the next eight tokens forget takes it to 2^-128.5
    zi, zf = np.zeros((T, 1)), np.full((T, 1), 60.0)
    zf[1:9, 0] = -16.63
    want = orc.mlstm_memory(q[:, 0] * D ** -0.5, k[:, 0], v[:, 0], orc.capped(zi[:, 0], 13.0), orc.log_sigmoid(orc.capped(zf[:, 0], 13.0)))[0]
    got, _ = run(jb, q, k, v, zi, zf, [T])
    low = np.abs(want[8:]) / 2.0 ** 100
    assert ((low > 2.0 ** -133) & (low < 2.0 ** -126)).all()                   # what is looked at is where it should be
    # the weighted score of 2^-129.5 goes into the product as a bf16 number, a multiple of 2^-133: half of that is 2^-4.5 of it
    assert (np.abs(got[8:, 0] - want[8:]) <= 2.0 ** -4 * np.abs(want[8:])).all(), (got[8:12, 0, 0], want[8:12, 0])


@pytest.mark.parametrize("shift", [(2, 0, 0), (1, 0, 0), (0, 1, 0), (0, 2, 0), (0, 0, 1), (2, 4, 4)])
@pytest.mark.parametrize("T", [8, 40, 200])
def test_outputs_may_start_at_any_element(T, shift):
    """`raw` at 8-byte boundaries is for the prompt kernels, elsewhere for the one that takes token by token; the kernel behind them reads it either way."""
    jb, (H, D, V) = pkg(), (2, 64, 40)
    q, k, v, _, zi, zf = memory_case(rng(T), H, D, V, T, "plain", "bfloat16")
    want, _ = run(jb, q, k, v, zi, zf, [T])
    got, _ = run(jb, q, k, v, zi, zf, [T], shift)
    if shift[0] % 2 == 0:
        assert np.array_equal(got, want)
    else:
        assert np.abs(got - want).max() <= 4e-4 * np.abs(want).max()      # both within the 2e-4 of test_edges
