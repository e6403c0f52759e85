"""Row-wise kernels in their wide forms against 64-bit: widths at and off the 16-byte groups, more pairs than are
asked for at once."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
# one rounding to bfloat16 of a value that is 2^-20 or so off in 32-bit
BF16 = 2.0 ** -8


def _native():
    from strata_inference_b200.kernels import native
    native.library()
    return native


@pytest.mark.parametrize("rows, heads, vd, pad, gated", [
    (1, 1, 8, 8, True), (37, 3, 24, 32, True), (5, 2, 7, 16, True), (300, 8, 256, 256, True), (9, 4, 40, 48, False)])
def test_head_gate(rows, heads, vd, pad, gated):
    n = _native()
    g = torch.Generator().manual_seed(vd)
    o = torch.randn(rows, heads * pad, generator=g).to(torch.bfloat16)
    z = torch.randn(rows, heads + 3, generator=g).to(torch.bfloat16)
    y = torch.empty(rows, heads * vd, dtype=torch.bfloat16, device=DEV)
    n.head_gate(o.to(DEV), z.to(DEV)[:, 3:] if gated else None, y, heads, vd, pad)
    want = o.double().view(rows, heads, pad)[:, :, :vd]
    if gated:
        want = want * torch.sigmoid(z.double()[:, 3:, None])
    assert bool(((y.double().cpu() - want.reshape(rows, -1)).abs() <= BF16 * want.reshape(rows, -1).abs() + 1e-9).all())


@pytest.mark.parametrize("rows, width, top", [(1, 8, 1), (70, 104, 7), (70, 104, 8), (33, 64, 9), (5, 77, 3), (700, 512, 17)])
@pytest.mark.parametrize("plain", [False, True])
def test_routed_combine(rows, width, top, plain):
    n = _native()
    g = torch.Generator().manual_seed(width + top)
    ys = torch.randn(rows * top, width, generator=g).to(torch.bfloat16)
    where = torch.randperm(rows * top, generator=g).to(torch.int32).view(rows, top)
    w, bw = torch.rand(rows, top, generator=g), torch.rand(rows, generator=g)
    base = torch.randn(rows, width, generator=g).to(torch.bfloat16)
    out = torch.empty(rows, width, dtype=torch.bfloat16, device=DEV)
    n.routed_combine(ys.to(DEV), where.to(DEV), None if plain else w.to(DEV), None if plain else base.to(DEV), out,
                     None if plain else bw.to(DEV))
    terms = ys.double()[where.long()] * (1.0 if plain else w.double()[:, :, None])
    want, size = terms.sum(1), terms.abs().sum(1)
    if not plain:
        want, size = want + base.double() * bw.double()[:, None], size + base.double().abs()
    assert bool(((out.double().cpu() - want).abs() <= BF16 * want.abs() + (top + 1) * 2.0 ** -24 * size).all())


@pytest.mark.parametrize("rows, heads, vd, memory, act", [
    (3, 2, 1, False, 0), (33, 5, 77, True, 1), (20, 3, 128, True, 0), (20, 3, 129, False, 1), (50, 4, 256, True, 0),
    (7, 2, 257, True, 1)])
def test_head_norm_gate(rows, heads, vd, memory, act):
    n = _native()
    g = torch.Generator().manual_seed(vd)
    cols = vd + 1 if memory else vd
    o = torch.randn(rows, heads * cols, generator=g)
    m = torch.randn(rows, heads, generator=g) if memory else None
    w = torch.rand(heads * vd, generator=g) + 0.5
    z = torch.randn(rows, heads * vd + 5, generator=g)
    y = torch.empty(rows, heads * vd, device=DEV)
    n.head_norm_gate(o.to(DEV), None if m is None else m.to(DEV), w.to(DEV), z.to(DEV)[:, 5:], y, heads, vd, 1e-5, act)
    x = o.double().view(rows, heads, cols)
    if memory:
        x = x[:, :, :vd] / (torch.maximum(x[:, :, vd].abs(), torch.exp(-m.double())) + 1e-6)[:, :, None]
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double().view(heads, vd)
    a = z.double()[:, 5:].view(rows, heads, vd)
    want = (x * (torch.sigmoid(a) if act else a * torch.sigmoid(a))).reshape(rows, -1)
    # (a sum of vd squares, two divisions, a root and an exponential)
    assert bool(((y.double().cpu() - want).abs() <= (vd + 16) * 2.0 ** -24 * want.abs() + 1e-9).all())
