"""The tiled attention of 32-bit prompts (csrc/attention_prompt_f32.cu) against 64-bit: edges of its tiles of
rows and keys, every grouping, head sizes, masks, a sink, infinities."""

import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _run(qkv, lens, nh, nkv, hd, scale, cap, window, chunk, keep, sink):
    from strata_inference_b200.kernels import native
    native.library()
    assert native.attention_prompt_f32_supports(nh, nkv, hd)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = SimpleNamespace(max_count=max(lens), n_seqs=len(lens), seq_start=i32([0] * len(lens)), seq_end=i32(lens),
                          seq_row0=i32([sum(lens[:i]) for i in range(len(lens))]))
    out = torch.full((qkv.shape[0], nh * hd), float("nan"), device=DEV)
    native.attention_prompt_f32(qkv.to(DEV), out, ctx, nh, nkv, hd, scale, cap, window, chunk=chunk, keep=keep,
                                sink=None if sink is None else sink.to(DEV))
    return out.cpu()


def _plain(x, nh, nkv, hd, scale, cap, window, chunk, keep, sink):
    T = x.shape[0]
    x = x.double()
    q = x[:, :nh * hd].view(T, nh, hd)
    k, v = (x[:, (nh + i * nkv) * hd:(nh + (i + 1) * nkv) * hd].reshape(T, nkv, hd).repeat_interleave(nh // nkv, 1)
            for i in (0, 1))
    s = torch.einsum("thd,jhd->htj", q, k) * scale
    s = cap * torch.tanh(s / cap) if cap else s
    i = torch.arange(T)
    far = i[:, None] - i[None, :]
    seen = far >= 0
    if window:
        seen &= (far < window) | (i[None, :] < keep)
    if chunk:
        seen &= i[None, :] >= i[:, None] - i[:, None] % chunk
    s = s.masked_fill(~seen, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(nh, T, 1)], 2)
    w = torch.softmax(s, -1)[..., :T]
    return torch.einsum("htj,jhd->thd", w, v).reshape(T, nh * hd)


@pytest.mark.parametrize("lens,nh,nkv,hd,cap,window,chunk,keep,with_sink", [
    ([1], 1, 1, 4, 0.0, 0, 0, 0, False), ([15, 16, 17], 8, 4, 256, 50.0, 0, 0, 0, False),
    ([31, 32, 33, 64, 65], 4, 4, 64, 0.0, 0, 0, 0, True), ([130, 3], 3, 1, 48, 20.0, 0, 0, 0, False),
    ([97], 32, 1, 100, 0.0, 0, 0, 0, False), ([200], 16, 2, 128, 0.0, 33, 0, 0, True),
    ([150, 40], 10, 2, 252, 0.0, 32, 0, 31, False), ([150], 4, 2, 16, 0.0, 1, 0, 70, False),
    ([160, 64], 4, 2, 128, 0.0, 0, 64, 0, True), ([99], 2, 2, 68, 30.0, 0, 7, 0, False)])
def test_prompts_against_64_bit(lens, nh, nkv, hd, cap, window, chunk, keep, with_sink):
    g = torch.Generator().manual_seed(3)
    wide = 8                                    # columns behind q | k | v that the kernel must not read
    qkv = torch.randn(sum(lens), (nh + 2 * nkv) * hd + wide, generator=g)
    qkv[:, (nh + 2 * nkv) * hd:] = float("nan")
    sink = torch.randn(nh, generator=g) + 1.0 if with_sink else None
    scale = 2.0 / math.sqrt(hd)
    got = _run(qkv, lens, nh, nkv, hd, scale, cap, window, chunk, keep, sink)
    row0 = 0
    for n in lens:
        want = _plain(qkv[row0:row0 + n], nh, nkv, hd, scale, cap, window, chunk, keep, sink)
        # scores of up to ~10, each a sum of head_dim products: an error of hd 2^-24 of its terms' size (at
        # most |q| |k| scale ~ 2 sqrt(hd)) moves a weight by as much, and the output by that of the largest value
        tol = 2 * math.sqrt(hd) * hd * 2.0 ** -24 + 64 * 2.0 ** -24
        assert (got[row0:row0 + n].double() - want).abs().max() <= tol * want.abs().max(), f"{n} rows"
        row0 += n


@pytest.mark.parametrize("where", ["k", "v"])
def test_an_infinity_stays_behind_its_row(where):
    g = torch.Generator().manual_seed(4)
    T, nh, nkv, hd, at = 120, 4, 2, 64, 75
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, generator=g)
    clean = _run(qkv, [T], nh, nkv, hd, 0.1, 0.0, 0, 0, 0, None)
    qkv[at, (nh if where == "k" else nh + nkv) * hd:(nh + nkv if where == "k" else nh + 2 * nkv) * hd] = math.inf
    got = _run(qkv, [T], nh, nkv, hd, 0.1, 0.0, 0, 0, 0, None)
    assert torch.equal(got[:at], clean[:at])
    assert not torch.isfinite(got[at]).all()


@pytest.mark.parametrize("lens,nh,nkv,hd,cap,spread", [
    ([64] * 16, 8, 4, 256, 50.0, 3.0), ([16] * 16, 8, 4, 256, 50.0, 1.0), ([301, 700], 8, 4, 256, 50.0, 2.0),
    ([300], 16, 8, 256, 50.0, 4.0), ([40] * 8, 4, 2, 16, 0.0, 2.0), ([200, 90], 16, 8, 128, 0.0, 2.0)])
def test_no_further_from_64_bits_than_the_general_kernel(lens, nh, nkv, hd, cap, spread):
    """The tiles' error against 64 bits (2-norm over all outputs) is that of a warp per row and head, at most.  Over
    some 10^5 elements two equally exact orders of the sums come within 2 % of one another; 5 % are allowed."""
    from strata_inference_b200.kernels import native
    native.library()
    g = torch.Generator().manual_seed(0)
    qkv = torch.randn(sum(lens), (nh + 2 * nkv) * hd, generator=g)
    qkv[:, :(nh + nkv) * hd] *= spread
    scale = torch.tensor(hd ** -0.5, dtype=torch.float32).item()
    tiled = _run(qkv, lens, nh, nkv, hd, scale, cap, 0, 0, 0, None)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    row0 = [sum(lens[:i]) for i in range(len(lens))]
    x, out = qkv.to(DEV), torch.empty(sum(lens), nh * hd, device=DEV)
    native.attention_rows(x, x.shape[1], x[:, nh * hd:], x[:, (nh + nkv) * hd:], x.shape[1], None, None, None, 64, 0,
                          i32([i for n in lens for i in range(n)]), i32([b for b, n in enumerate(lens) for _ in range(n)]),
                          i32(list(range(len(lens)))), i32([0] * len(lens)), i32(row0), out, None, nh, nkv, hd, scale,
                          cap, 0, 1)
    want = torch.cat([_plain(qkv[r:r + n], nh, nkv, hd, scale, cap, 0, 0, 0, None) for r, n in zip(row0, lens)])
    off = [(y.double() - want).norm().item() for y in (tiled, out.cpu())]
    assert off[0] <= 1.05 * off[1], f"{off[0] / off[1]:.3f} of the general kernel's error"


@pytest.mark.parametrize("lengths,tiled", [([3, 8], False), ([2, 16], True)])
def test_the_shortest_prompts_stay_with_the_general_kernel(lengths, tiled, monkeypatch):
    from helpers import TINY_A
    from strata_inference_b200 import Engine
    from strata_inference_b200.kernels import native
    native.library()
    calls, plain = [], native.attention_prompt_f32
    monkeypatch.setattr(native, "attention_prompt_f32", lambda *a, **kw: (calls.append(1), plain(*a, **kw))[1])
    eng = Engine.from_random(TINY_A, 1, dtype="float32", max_tokens=256)
    eng.step([(eng.new_sequence(), [5 + i for i in range(n)]) for n in lengths])
    assert bool(calls) == tiled
