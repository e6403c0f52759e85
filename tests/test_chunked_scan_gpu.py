"""The recurrences in chunks of 64 tokens (csrc/chunked_scan.cu) against the recurrence token by token in
64-bit: chunk edges, widths that are no multiples of anything, grouped key heads, a state to begin with,
a sequence without a slot, factors of zero, infinities."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
# The longest sums of 32-bit terms are a product with the matrix (up to 128 keys) and one over a chunk
# (64 tokens), whose factors are such sums themselves: 4 x 192 roundings of 2^-24 bound the error relative
# to the largest output.
TOL = 4 * 192 * 2.0 ** -24


def _native():
    from strata_inference_b200.kernels import native
    native.library()
    return native


def _context(lens, slots, starts):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    row0 = [sum(lens[:i]) for i in range(len(lens))]
    return SimpleNamespace(max_count=max(lens), n_seqs=len(lens), seq_slot=i32(slots), seq_start=i32(starts),
                           seq_end=i32([s + n for s, n in zip(starts, lens)]), seq_row0=i32(row0)), row0


def _walk(q, k, v, keep, take, S, delta):
    """q, k [T, H, kd], v [T, H, cols], keep, take [T, H], S [H, kd, cols], all 64-bit."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * keep[t][:, None, None]
        u = v[t] - (S * k[t][:, :, None]).sum(1) if delta else v[t]
        S = S + k[t][:, :, None] * (take[t][:, None] * u)[:, None, :]
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out, S


def _unit(x):
    return x / x.norm(dim=-1, keepdim=True)


SHAPES = [
    # lengths, heads, key heads, key width, value width
    ([64], 2, 1, 16, 16), ([65, 1, 63], 3, 3, 50, 7), ([128, 129], 4, 2, 64, 65), ([200], 2, 2, 65, 17),
    ([1], 1, 1, 1, 1), ([300, 2, 64, 191], 4, 1, 128, 128), ([77], 2, 2, 128, 200), ([257], 1, 1, 3, 64)]


@pytest.mark.parametrize("mode", ["delta", "gated", "retention", "memory"])
@pytest.mark.parametrize("lens,H,G,kd,vd", SHAPES)
def test_chunks_against_token_by_token(mode, lens, H, G, kd, vd, monkeypatch):
    n = _native()
    monkeypatch.setattr(n, "CHUNKED_SCAN_MIN_ROWS", 1)
    if mode in ("memory", "retention"):
        G = H
    g = torch.Generator().manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    R, B = sum(lens), len(lens)
    slots = [2 * i + 1 for i in range(B)]
    if B > 1:
        slots[1] = -1                               # a sequence that holds no slot begins with zeros
    ctx, row0 = _context(lens, slots, [3 * i for i in range(B)])
    cols = vd + 1 if mode == "memory" else vd
    size = -(-(H * cols * kd + H) // 4) * 4
    state = rnd(2 * B + 1, size)
    q, k, v = rnd(R, G, kd), rnd(R, G, kd), rnd(R, H, vd)
    keep = torch.exp(-torch.exp(rnd(R, H)))
    take = torch.sigmoid(rnd(R, H))
    keep[R // 2] = 0.0                              # everything before this token is forgotten
    if mode == "delta":
        q, k = _unit(q) * kd ** -0.5, _unit(k)
    elif mode == "retention":
        decay = torch.sigmoid(rnd(H) + 2)
        keep, take = decay.expand(R, H), torch.ones(R, H)
    elif mode == "memory":
        cap, bias_i, bias_f = 9.0, rnd(H), rnd(H) + 2
        gi, gf = 3 * rnd(R, H), 3 * rnd(R, H)
    dev = state.clone().to(DEV)
    flat = lambda x: x.reshape(R, -1).contiguous().to(DEV)  # noqa: E731
    out = torch.empty(R, H * cols, device=DEV)
    if mode == "delta":
        n.delta_scan(flat(q), flat(k), flat(v), flat(keep), flat(take), dev, out, ctx, H, G, kd, vd)
    elif mode == "gated":
        n.gated_scan(flat(q), flat(k), flat(v), flat(keep), flat(take), dev, out, ctx, H, G, kd, vd)
    elif mode == "retention":
        n.retention_scan(flat(q), flat(k), flat(v), decay.to(DEV), dev, out, ctx, H, kd, vd)
    else:
        m_out = torch.empty(R, H, device=DEV)
        proj = torch.cat([flat(q), flat(k), flat(v), flat(v), flat(gi), flat(gf)], 1)
        n.memory_scan(proj, bias_i.to(DEV), bias_f.to(DEV), cap, dev, out, m_out, ctx, H, kd, vd)
    torch.cuda.synchronize()
    for b in range(B):
        rows = slice(row0[b], row0[b] + lens[b])
        first = state[slots[b]].double() if slots[b] >= 0 else torch.zeros(size, dtype=torch.float64)
        S = first[:H * cols * kd].view(H, cols, kd).transpose(1, 2)
        heads = lambda x: x[rows].double().repeat_interleave(H // G, 1)  # noqa: E731
        vv, a, c = v[rows].double(), keep[rows].double(), take[rows].double()
        scale = 1.0
        if mode == "memory":
            scale = kd ** -0.5
            vv = torch.cat([vv, torch.ones(lens[b], H, 1, dtype=torch.float64)], 2)
            i = cap * torch.tanh((gi[rows].double() + bias_i.double()) / cap)
            f = torch.nn.functional.logsigmoid(cap * torch.tanh((gf[rows].double() + bias_f.double()) / cap))
            m = first[H * cols * kd:H * cols * kd + H]
            a, c, ms = torch.empty_like(i), torch.empty_like(i), torch.empty_like(i)
            for t in range(lens[b]):
                new = torch.maximum(f[t] + m, i[t])
                a[t], c[t], ms[t], m = torch.exp(f[t] + m - new), torch.exp(i[t] - new), new, new
            assert torch.allclose(m_out[rows].double().cpu(), ms, rtol=1e-5, atol=1e-5)
            if slots[b] >= 0:
                assert torch.allclose(dev[slots[b], H * cols * kd:H * cols * kd + H].double().cpu(), m, rtol=1e-5, atol=1e-5)
        want, S = _walk(heads(q) * scale, heads(k), vv, a, c, S, mode == "delta")
        got = out[rows].view(lens[b], H, cols).double().cpu()
        # (the memory's factors are exponentials of 32-bit differences: a few roundings of values up to ~10)
        tol = TOL * (4 if mode == "memory" else 1)
        assert (got - want).abs().max() <= tol * want.abs().max(), f"outputs of sequence {b}"
        if slots[b] >= 0:
            after = dev[slots[b], :H * cols * kd].view(H, cols, kd).transpose(1, 2).double().cpu()
            assert (after - S).abs().max() <= tol * S.abs().max(), f"state of sequence {b}"
    untouched = [s for s in range(2 * B + 1) if s not in slots]
    assert torch.equal(dev[untouched].cpu(), state[untouched]), "other slots' states"


@pytest.mark.parametrize("mode", ["delta", "gated"])
@pytest.mark.parametrize("where", ["k", "v", "q", "keep"])
def test_an_infinity_stays_behind_its_token(mode, where, monkeypatch):
    n = _native()
    monkeypatch.setattr(n, "CHUNKED_SCAN_MIN_ROWS", 1)
    g = torch.Generator().manual_seed(5)
    T, H, kd, vd, at = 150, 2, 32, 20, 90
    x = {"q": _unit(torch.randn(T, H, kd, generator=g)), "k": _unit(torch.randn(T, H, kd, generator=g)),
         "v": torch.randn(T, H, vd, generator=g), "keep": torch.rand(T, H, generator=g),
         "take": torch.rand(T, H, generator=g)}
    ctx, _ = _context([T], [0], [0])
    outs = []
    for value in (1.0, float("inf")):
        x[where][at] = value
        dev = {name: t.reshape(T, -1).contiguous().to(DEV) for name, t in x.items()}
        out = torch.empty(T, H * vd, device=DEV)
        scan = n.delta_scan if mode == "delta" else n.gated_scan
        scan(dev["q"], dev["k"], dev["v"], dev["keep"], dev["take"], torch.zeros(1, H * kd * vd, device=DEV), out,
             ctx, H, H, kd, vd)
        outs.append(out.cpu())
    assert torch.equal(outs[0][:at], outs[1][:at]), "rows before the infinity"
    assert not torch.isfinite(outs[1][at]).all(), "its own row"
