"""The contraction at the edges of its 256 x 256 tiles: one tile with and without its lower half, narrow column tiles, a
second tile of one row, several K steps with a remainder."""

import pytest
import torch

from bionemo_inference_runtime_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N", [(1, 1), (2, 32), (1, 65), (1, 127), (1, 128), (2, 129), (1, 255), (1, 256), (1, 257), (1, 385), (1, 513)])
def test_contraction_at_tile_edges(B, N):
    g = torch.Generator(device="cuda").manual_seed(N)
    pitch = (N + 15) // 16 * 16
    ab = torch.zeros(B, 256, N, pitch, dtype=torch.bfloat16, device="cuda")
    ab[..., :N] = torch.randn(B, 256, N, N, generator=g, device="cuda").bfloat16()
    _lib.reset_device_status()
    x = ops.trimul_contract(ab, N)
    assert _lib.device_status() == 0
    a, b = ab[:, :128, :, :N].float(), ab[:, 128:, :, :N].float()
    torch.testing.assert_close(x[..., :N].float(), a @ b.transpose(-1, -2), rtol=1e-2, atol=1e-2 * N**0.5)


@pytest.mark.parametrize("N", [8, 32, 70, 96, 330])
def test_many_tiles_with_an_odd_number_of_stores(N):
    """Tiles of 1, 1, 3, 3 and 6 + 5 column groups, a dozen tiles a block: the two slabs of a warp have to take turns over
    the tiles as well."""
    g = torch.Generator(device="cuda").manual_seed(N)
    B, pitch = 16, (N + 15) // 16 * 16
    ab = torch.randn(B, 256, N, pitch, generator=g, device="cuda").bfloat16()
    a, b = ab[:, :128, :, :N].float(), ab[:, 128:, :, :N].float()
    want = a @ b.transpose(-1, -2)
    for _ in range(5):
        torch.testing.assert_close(ops.trimul_contract(ab, N)[..., :N].float(), want, rtol=1e-2, atol=1e-2 * N**0.5)
    assert _lib.device_status() == 0
