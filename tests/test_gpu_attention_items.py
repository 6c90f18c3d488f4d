"""The attention core over the ways its units of 128 queries are put together into items: one, two and four units per
item, an odd last query block, a remainder of rows in smaller items, rows of different lengths in one item."""

import pytest
import torch

from bionemo_inference_runtime_b200 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("B,R,S", [(1, 3, 300), (1, 20, 100), (1, 60, 64), (1, 201, 65), (10, 10, 256), (1, 77, 385), (2, 33, 129)])
def test_rows_of_different_lengths_in_one_item(B, R, S, masked):
    g = torch.Generator(device=DEV).manual_seed(B * 1000 + R + S)
    qkvg = torch.randn(4, B * R, 4, S, 32, generator=g, device=DEV).bfloat16()
    bias = torch.randn(B, 4, S, ops.pad8(S), generator=g, device=DEV).bfloat16()
    bias[..., S:] = float("nan")  # the key padding never reaches a result
    lens = torch.randint(0, S + 1, (B, R), dtype=torch.int32, device=DEV, generator=g)
    lens[0, :3] = torch.tensor([S, 0, 1], dtype=torch.int32, device=DEV)
    valid = torch.arange(S, device=DEV) < lens[..., None]
    bits = None
    if masked:
        valid = valid & (torch.rand(B, R, S, generator=g, device=DEV) > 0.3)
        lens, bits = ops.key_mask_bits(valid)
    _lib.reset_device_status()
    got = ops.attention(qkvg, bias, lens, B, R, S, key_mask=bits).float()
    assert _lib.device_status() == 0
    q, k, v, gate = qkvg.float().view(4, B, R, 4, S, 32)
    logits = (q @ k.transpose(-1, -2) + bias[..., :S].float()[:, None]) * 32**-0.5
    logits = torch.where(valid[:, :, None, None, :], logits, torch.full_like(logits, -1e9))  # no valid key: uniform
    want = (logits.softmax(-1) @ v * gate).permute(0, 1, 3, 2, 4).reshape(B, R, S, 128)
    torch.testing.assert_close(got, want, rtol=2e-2, atol=2e-2)
