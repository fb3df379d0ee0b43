"""Prefill attention on the tensor cores against a plain float64 statement, where its blocks take several items each and
where the running maxima move."""
import numpy as np
import pytest
import torch

from b200nn import ops

pytestmark = pytest.mark.gpu


def _exact(q, k, v, B, H, S, past):
    q = q.double().reshape(B, S, H, 64).transpose(1, 2)
    s = q @ k.double()[:, :, :past + S].transpose(-1, -2) * 0.125
    at = torch.arange(past + S, device="cuda")
    s = s.masked_fill(at[None, :] > past + torch.arange(S, device="cuda")[:, None], -float("inf"))
    return (torch.softmax(s, -1) @ v.double()[:, :, :past + S]).transpose(1, 2).reshape(B * S, H * 64)


# one item; a block more items than the GPU holds blocks; several items a block, the last ones short; rows past the end of a
# sequence inside its last tile; a whole warp of them; keys of a past that ends inside a tile; a cache longer than what is written
@pytest.mark.parametrize("B,H,S,past,cap", [(1, 1, 1, 0, 1), (3, 99, 100, 0, 128), (13, 12, 300, 0, 300), (9, 25, 257, 127, 400),
                                            (40, 12, 130, 3, 140), (2, 12, 33, 900, 1024)])
@pytest.mark.parametrize("growth", [0.0, 6.0, -6.0])
def test_prefill_attention_items_and_moving_maxima(reg, B, H, S, past, cap, growth):
    g = torch.Generator(device="cuda").manual_seed(B + S)
    n = past + S
    q = torch.randn(B * S, H * 64, generator=g, device="cuda").half()
    k, v = (torch.randn(B, H, cap, 64, generator=g, device="cuda").half() for _ in range(2))
    # scores that grow (or shrink) along the keys by `growth` spreads from end to end: every tile moves the maxima, or none
    k *= torch.exp2(torch.linspace(-abs(growth) / 2, abs(growth) / 2, cap, device="cuda") * (1 if growth >= 0 else -1))[None, None, :, None].half()
    k[:, :, n:] = float("nan")  # never read: not written yet
    v[:, :, n:] = float("nan")
    out = torch.full((B * S + 8, H * 64), 7.0, device="cuda", dtype=torch.float16)
    torch.cuda.synchronize()
    ops.prefill_attention_f16(q.data_ptr(), k.data_ptr(), v.data_ptr(), B, H, cap, S, past, out.data_ptr(), reg)
    reg.synchronize()
    assert (out[B * S:] == 7.0).all()
    ref = _exact(q, k, v, B, H, S, past)
    # probabilities and outputs rounded to fp16: 2^-11 at most of each, half that on average, twice
    assert (torch.linalg.norm(out[:B * S].double() - ref) / torch.linalg.norm(ref)).item() < 6e-4
    assert reg.device_error() == 0


def test_prefill_attention_keeps_what_is_not_finite_to_its_own_rows(reg):
    B, H, S = 3, 2, 200
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randn(B * S, H * 64, generator=g, device="cuda").half()
    k, v = (torch.randn(B, H, S, 64, generator=g, device="cuda").half() for _ in range(2))
    clean, out = (torch.zeros(B * S, H * 64, device="cuda", dtype=torch.float16) for _ in range(2))
    torch.cuda.synchronize()
    ops.prefill_attention_f16(q.data_ptr(), k.data_ptr(), v.data_ptr(), B, H, S, S, 0, clean.data_ptr(), reg)
    reg.synchronize()
    q[S + 3], q[2 * S - 1] = float("nan"), float("inf")
    torch.cuda.synchronize()
    ops.prefill_attention_f16(q.data_ptr(), k.data_ptr(), v.data_ptr(), B, H, S, S, 0, out.data_ptr(), reg)
    reg.synchronize()
    bad = np.zeros(B * S, dtype=bool)
    bad[[S + 3, 2 * S - 1]] = True
    assert not torch.isfinite(out[bad]).any() and torch.equal(out[~torch.from_numpy(bad).cuda()], clean[~torch.from_numpy(bad).cuda()])
