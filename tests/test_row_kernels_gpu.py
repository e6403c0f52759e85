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


@pytest.mark.parametrize("lens, starts, G, H, kd, vd, dtype", [
    ([256], [0], 1, 1, 1, 1, torch.float32), ([250, 3, 1, 9], [0, 7, 0, 2], 2, 4, 50, 33, torch.float32),
    ([133, 300], [5, 0], 4, 8, 128, 256, torch.bfloat16), ([400], [1], 2, 2, 256, 300, torch.bfloat16),
    ([2, 255], [3, 4], 3, 3, 257, 16, torch.float32),
    # (enough rows and heads for the runs)
    ([24000], [0], 1, 1, 1, 1, torch.float32), ([690, 3, 1, 34], [0, 7, 0, 2], 8, 16, 50, 33, torch.float32),
    ([1133, 300], [5, 0], 4, 8, 128, 256, torch.bfloat16), ([1001], [1], 8, 8, 256, 300, torch.bfloat16)])
def test_delta_prepare_of_many_rows(lens, starts, G, H, kd, vd, dtype):
    """Runs of 8 rows that share their channels' inputs: sequences that begin and end inside a run, inputs from
    the slots' histories, a sequence without a slot, key heads wider than the runs take."""
    from types import SimpleNamespace
    n = _native()
    g = torch.Generator().manual_seed(kd)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    R, B, taps = sum(lens), len(lens), 4
    ch, mats = 2 * G * kd + H * vd, H * vd * kd
    slots = [2 * b for b in range(B)]
    if B > 2:
        slots[1] = -1
    row0 = [sum(lens[:b]) for b in range(B)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = SimpleNamespace(
        row_pos=i32([s + i for s, m in zip(starts, lens) for i in range(m)]), n_seqs=B, seq_slot=i32(slots),
        row_seq=i32([b for b, m in enumerate(lens) for _ in range(m)]), seq_start=i32(starts),
        seq_end=i32([s + m for s, m in zip(starts, lens)]), seq_row0=i32(row0))
    proj = rnd(R, ch + H * vd + 2 * H).to(dtype)
    conv, a_log, bias = rnd(ch, taps), rnd(H), rnd(H)
    state = rnd(2 * B, -(-(mats + (taps - 1) * ch) // 4) * 4)
    outs = [torch.empty(R, m, device=DEV) for m in (G * kd, G * kd, H * vd, H, H)]
    dev = state.clone().to(DEV)
    n.delta_prepare(proj.to(DEV), conv.to(DEV), a_log.to(DEV), bias.to(DEV), dev, mats, *outs, ctx, H, G, kd, vd, taps)
    q, k, v, beta, decay = (t.double().cpu() for t in outs)
    x = proj.double()
    for b in range(B):
        rows = slice(row0[b], row0[b] + lens[b])
        past = torch.zeros(taps - 1, ch, dtype=torch.float64)
        if slots[b] >= 0:
            past = state[slots[b], mats:mats + (taps - 1) * ch].double().view(taps - 1, ch)
        full = torch.cat([past, x[rows, :ch]])
        y = sum(full[j:j + lens[b]] * conv[:, j].double() for j in range(taps))
        y = y * torch.sigmoid(y)
        heads = y[:, :2 * G * kd].view(lens[b], 2 * G, kd)
        size = torch.sqrt((heads * heads).sum(-1, keepdim=True) + 1e-6)
        heads = heads / size
        # (an activated sum is off by its terms' rounding, whatever it comes to; a unit norm divides that by
        # the head's length, which is small where the sums cancel)
        terms = sum(full[j:j + lens[b]].abs() * conv[:, j].double().abs() for j in range(taps))[:, :2 * G * kd]
        off = 8 * 2.0 ** -24 * terms.view(lens[b], 2 * G, kd).amax(-1, keepdim=True) * kd ** 0.5 / size
        want = (heads[:, :G].reshape(lens[b], -1) * kd ** -0.5, heads[:, G:].reshape(lens[b], -1), y[:, 2 * G * kd:],
                torch.sigmoid(x[rows, ch + H * vd:ch + H * vd + H]),
                torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(x[rows, ch + H * vd + H:] + bias.double())))
        # (four products, an exponential and, for q and k, a sum of kd squares, a root and two divisions; the
        # decay's exponent is of the size of ten)
        for name, got, ref in zip("q k v beta decay".split(), (q, k, v, beta, decay), want):
            room = (kd + 64) * 2.0 ** -24 * ref.abs().max()
            if name in "qk":
                room = room + (off[:, :G] * kd ** -0.5 if name == "q" else off[:, G:]).expand(-1, -1, kd).reshape(lens[b], -1)
            assert bool(((got[rows] - ref).abs() <= room).all()), f"{name} of sequence {b}"
        if slots[b] >= 0:
            kept = dev[slots[b], mats:mats + (taps - 1) * ch].double().cpu().view(taps - 1, ch)
            assert torch.equal(kept, full[lens[b]:])


def test_delta_prepare_does_not_depend_on_what_is_beside_a_sequence():
    """Runs of 8 rows give the same bits as rows one by one: ten sequences in one call against each alone."""
    from types import SimpleNamespace
    n = _native()
    g = torch.Generator().manual_seed(12)
    G, H, kd, vd, taps, lens = 4, 8, 100, 72, 4, [205 + 3 * b for b in range(10)]
    ch, mats = 2 * G * kd + H * vd, 16
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    proj = torch.randn(sum(lens), ch + H * vd + 2 * H, generator=g).to(torch.bfloat16).to(DEV)
    conv, a_log, bias = (torch.randn(*s, generator=g).to(DEV) for s in ((ch, taps), (H,), (H,)))
    first = torch.randn(10, mats + (taps - 1) * ch, generator=g).to(DEV)

    def prepare(seqs, rows, state):
        m = [lens[b] for b in seqs]
        ctx = SimpleNamespace(
            row_pos=i32([9 + i for k in m for i in range(k)]), n_seqs=len(m), seq_slot=i32(seqs),
            row_seq=i32([b for b, k in enumerate(m) for _ in range(k)]), seq_start=i32([9] * len(m)),
            seq_end=i32([9 + k for k in m]), seq_row0=i32([sum(m[:b]) for b in range(len(m))]))
        outs = [torch.empty(sum(m), w, device=DEV) for w in (G * kd, G * kd, H * vd, H, H)]
        n.delta_prepare(proj[rows], conv, a_log, bias, state, mats, *outs, ctx, H, G, kd, vd, taps)
        return outs

    together, alone = first.clone(), first.clone()
    got, at = prepare(list(range(10)), slice(0, sum(lens)), together), 0
    for b, k in enumerate(lens):
        for name, x, y in zip("q k v beta decay".split(), got, prepare([b], slice(at, at + k), alone)):
            assert torch.equal(x[at:at + k], y), f"{name} of sequence {b}"
        at += k
    assert torch.equal(together, alone)
