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
