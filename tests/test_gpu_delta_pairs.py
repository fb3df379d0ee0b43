"""Delta-rule prompts, taken two tokens at a time through stages of eight, against the single-token kernel over the same
rows: lengths at the edges of pairs and stages, decays that make a pair apply its decays to the state at once, and what
follows a sequence in the pass must not matter to it."""
import numpy as np
import pytest
import torch

import b200nn
from b200nn import ops

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 7, 8, 9, 15, 16, 17, 24, 31, 40]


def _ints(*parts):
    return torch.from_numpy(np.concatenate([np.asarray(p, np.int32).ravel() for p in parts])).cuda()


@pytest.mark.parametrize("H,KH,dim,vdim", [(2, 1, 32, 16), (2, 2, 128, 48), (1, 1, 256, 32), (24, 8, 128, 128)])
@pytest.mark.parametrize("channel", [False, True])
def test_prompts_agree_with_single_tokens(reg, H, KH, dim, vdim, channel):
    g = torch.Generator(device="cuda").manual_seed(dim + H)
    E, N, taps = len(LENGTHS), sum(LENGTHS), 4
    cw = 2 * KH * dim + H * vdim
    pw = -(-(cw + H) // 16) * 16 if channel else -(-(cw + H * vdim + 2 * H) // 4) * 4
    ext = H * max(dim, vdim)
    decays = H * dim if channel else H
    proj, exts = torch.randn(N, pw, generator=g, device="cuda"), torch.randn(N, 2 * ext, generator=g, device="cuda")
    conv, norm = torch.randn(taps, cw, generator=g, device="cuda") * 0.5, torch.rand(vdim, generator=g, device="cuda") + 0.5
    a_exp = torch.exp(torch.linspace(-4.0, 4.5, H, device="cuda"))  # from hardly a decay to about e^-90 a token
    dt = torch.randn(decays, generator=g, device="cuda")
    shape, ptrs = (H, KH, dim, vdim, taps, 1e-5), tuple(t.data_ptr() for t in (conv, a_exp, dt, norm))
    row0 = np.concatenate([[0], np.cumsum(LENGTHS)[:-1]])
    slots = np.arange(E)[::-1].copy()

    def run(rows, at, pos, slot, cs, st, n_seq=0, meta=None):
        out = torch.zeros(len(rows), H, vdim, device="cuda")
        x, e, tp, ts = proj[rows].contiguous(), exts[rows].contiguous(), _ints(pos), _ints(slot)
        scratch = torch.full((len(rows) * (cw + decays + H + KH + 4 + H * vdim),), float("nan"), device="cuda")
        torch.cuda.synchronize()
        tail = (cs.data_ptr(), st.data_ptr(), tp.data_ptr(), ts.data_ptr(), len(rows), out.data_ptr(), reg)
        kw = dict(n_seq=n_seq, max_n=max(LENGTHS) if n_seq else 0, seq_ptr=meta.data_ptr() if n_seq else None, scratch_ptr=scratch.data_ptr(), flags=b200nn.LM_F32)
        if channel:
            ops.channel_delta_rule(shape, ptrs, x.data_ptr(), e.data_ptr(), *tail, **kw)
        else:
            ops.delta_rule(shape, ptrs, x.data_ptr(), *tail, **kw)
        reg.synchronize()
        return out

    states = [(torch.zeros(E, taps, cw, device="cuda"), torch.zeros(E, H, dim, vdim, device="cuda")) for _ in range(2)]
    meta = _ints(slots, row0, LENGTHS, np.zeros(E), np.repeat(np.arange(E), LENGTHS))
    pos = np.concatenate([np.arange(n) for n in LENGTHS])
    got = run(list(range(N)), row0, pos, np.repeat(slots, LENGTHS), *states[0], n_seq=E, meta=meta)
    want = torch.zeros_like(got)
    for t in range(max(LENGTHS)):
        live = [i for i, n in enumerate(LENGTHS) if t < n]
        rows = [int(row0[i]) + t for i in live]
        want[rows] = run(rows, None, [t] * len(live), slots[live], *states[1])
    # f32 on both sides: 3e-5 of the norm is what each may differ from the float64 recurrence
    for i, n in enumerate(LENGTHS):
        a, b = got[row0[i]:row0[i] + n], want[row0[i]:row0[i] + n]
        assert torch.linalg.norm(a - b) <= 6e-5 * torch.linalg.norm(b), f"sequence of {n}"
        a, b = states[0][1][slots[i]], states[1][1][slots[i]]
        assert torch.linalg.norm(a - b) <= 6e-5 * torch.linalg.norm(b) + 1e-30, f"state of {n}"
        assert torch.equal(states[0][0][slots[i]], states[1][0][slots[i]]), f"convolution inputs of {n}"
    assert reg.device_error() == 0


@pytest.mark.parametrize("channel", [False, True])
def test_sequences_of_no_rows_change_nothing(reg, channel):
    """Entries of no rows first, last and between others, one of them behind the last row of the pass."""
    g = torch.Generator(device="cuda").manual_seed(3)
    H, KH, dim, vdim, taps = 3, 1, 64, 32, 4
    lengths = [0, 5, 0, 0, 9, 0]
    E, N = len(lengths), sum(lengths)
    cw = 2 * KH * dim + H * vdim
    pw = -(-(cw + H) // 16) * 16 if channel else -(-(cw + H * vdim + 2 * H) // 4) * 4
    decays, ext = (H * dim if channel else H), H * max(dim, vdim)
    proj, exts = torch.randn(N, pw, generator=g, device="cuda"), torch.randn(N, 2 * ext, generator=g, device="cuda")
    conv, norm = torch.randn(taps, cw, generator=g, device="cuda"), torch.rand(vdim, generator=g, device="cuda") + 0.5
    a_exp, dt = torch.ones(H, device="cuda"), torch.randn(decays, generator=g, device="cuda")
    first = (torch.randn(E, taps, cw, generator=g, device="cuda"), torch.randn(E, H, dim, vdim, generator=g, device="cuda"))

    def run(entries):
        cs, st, out = first[0].clone(), first[1].clone(), torch.zeros(N, H, vdim, device="cuda")
        scratch = torch.zeros(N * (cw + decays + H + KH + 4 + H * vdim), device="cuda")
        ns = [lengths[i] for i in entries]
        row0 = np.concatenate([[0], np.cumsum(ns)[:-1]])
        meta = _ints(entries, row0, ns, [4] * len(ns), np.repeat(np.arange(len(ns)), ns))
        pos, slot = _ints(np.concatenate([4 + np.arange(n) for n in ns])), _ints(np.repeat(entries, ns))
        torch.cuda.synchronize()
        shape, ptrs = (H, KH, dim, vdim, taps, 1e-5), tuple(t.data_ptr() for t in (conv, a_exp, dt, norm))
        tail = (cs.data_ptr(), st.data_ptr(), pos.data_ptr(), slot.data_ptr(), N, out.data_ptr(), reg)
        kw = dict(n_seq=len(ns), max_n=max(ns), seq_ptr=meta.data_ptr(), scratch_ptr=scratch.data_ptr(), flags=b200nn.LM_F32)
        if channel:
            ops.channel_delta_rule(shape, ptrs, proj.data_ptr(), exts.data_ptr(), *tail, **kw)
        else:
            ops.delta_rule(shape, ptrs, proj.data_ptr(), *tail, **kw)
        reg.synchronize()
        return out, cs, st
    got, want = run(list(range(E))), run([1, 4])
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    for i in (0, 2, 3, 5):
        assert torch.equal(got[1][i], first[0][i]) and torch.equal(got[2][i], first[1][i])
    assert not torch.equal(got[2][1], first[1][1]) and reg.device_error() == 0


# passes of at most three tokens a sequence take them one at a time where the decays are per channel (one and two columns a lane,
# every share of dim per lane); one of four does not
@pytest.mark.parametrize("longest", [3, 4])
@pytest.mark.parametrize("H,KH,dim,vdim", [(8, 4, 32, 128), (16, 4, 64, 64), (8, 8, 96, 96), (6, 2, 128, 128), (2, 1, 128, 16)])
def test_short_prompts_agree_with_single_tokens(reg, monkeypatch, H, KH, dim, vdim, longest):
    monkeypatch.setitem(globals(), "LENGTHS", [1, 2, longest, 3, 1, 2])
    test_prompts_agree_with_single_tokens(reg, H, KH, dim, vdim, True)
