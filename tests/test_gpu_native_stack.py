"""The native form of a stack (one call, single track on a second stream) against the same layers called one by one."""

import pytest
import torch

import bionemo_inference_runtime_b200 as b200
from bionemo_inference_runtime_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _randomise(module):
    g = torch.Generator(device=DEV).manual_seed(1)
    for name, p in module.named_parameters():
        p.data.copy_(torch.randn(p.shape, generator=g, device=DEV) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1)
                     + (1.0 if p.dim() == 1 and not name.endswith("bias") else 0.0))
    return module


@pytest.mark.parametrize("version,f32,backend", [("v1", False, "Heuristic"), ("v1", True, "VANILLA"), ("v2", False, "Heuristic")])
@pytest.mark.parametrize("B,N", [(1, 33), (3, 72)])
def test_native_stack_equals_the_layers(version, f32, backend, B, N):
    stack = _randomise(b200.PairformerModule(num_blocks=3, dtype=torch.bfloat16, version=version, trimul_high_precision=f32,
                                             triangle_attn_backend=backend, attention_initial_norm=version == "v1").to(DEV))
    g = torch.Generator(device=DEV).manual_seed(2)
    s = torch.randn(B, N, 384, generator=g, device=DEV).bfloat16()
    z = torch.randn(B, N, N, 128, generator=g, device=DEV).bfloat16()
    mask = (torch.arange(N, device=DEV)[None] < torch.tensor([N, N - 5, 7][:B], device=DEV)[:, None]).float()
    pair = mask[:, :, None] * mask[:, None, :]
    z0 = z.clone()
    got = stack(s, z, mask, pair)
    assert stack._native.stack is not None and torch.equal(z, z0)
    again = stack(s, z, mask, pair)
    handle = stack.layers[1].register_forward_hook(lambda *args: None)  # a hooked layer is called itself
    want = stack(s, z, mask, pair)
    handle.remove()
    for a, b, c in zip(got, again, want):
        assert torch.equal(a, b) and torch.equal(a, c)
    # an edited option takes effect: the ending node's bias written transposed has no native form
    stack.layers[0].tri_attn_end.transposed_bias = True
    stack(s, z, mask, pair)
    assert stack._native.stack is None
    stack.layers[0].tri_attn_end.transposed_bias = False
    # ... and so does an edited weight
    with torch.no_grad():
        stack.layers[2].transition_s.fc3.weight.mul_(2.0)
    assert not torch.equal(stack(s, z, mask, pair)[0], got[0])
    assert _lib.device_status() == 0


def test_masks_in_one_launch_equal_the_torch_operations():
    g = torch.Generator(device=DEV).manual_seed(3)
    from bionemo_inference_runtime_b200 import _host, ops

    for B, N in ((1, 1), (2, 31), (1, 96), (3, 130)):
        mask = (torch.rand(B, N, N, generator=g, device=DEV) > 0.4).float()
        rows, columns = _host.mask_lengths(mask)
        assert torch.equal(rows, (mask > 0.5).sum(-1).int()) and torch.equal(columns, (mask > 0.5).sum(-2).int())
        for source, additive in ((mask.transpose(1, 2), False), ((mask - 1) * 1e9, True)):
            valid = source >= 0 if additive else source > 0.5
            for a, b in zip(_host.mask_bits(source, additive), ops.key_mask_bits(valid)):
                assert torch.equal(a, b)


def test_an_error_inside_the_single_track_joins_the_side_stream(monkeypatch):
    """The last block's single transition is refused on the host when the blocks before it are enqueued already.  Streams
    that are not joined again would make the capture of such a call fail at its end."""
    from bionemo_inference_runtime_b200.layers import pairformer

    class Broken(pairformer._host.Stack):
        singles = 0

        def add_single(self, *args):
            self.singles += 1
            args = list(args)
            if self.singles == 2:
                args[9] = args[9][:, :256].contiguous()  # w1 for another width
            super().add_single(*args)

    stack = _randomise(b200.PairformerModule(num_blocks=2, dtype=torch.bfloat16, triangle_attn_backend="Heuristic").to(DEV))
    inputs = (torch.randn(1, 48, 384, device=DEV).bfloat16(), torch.randn(1, 48, 48, 128, device=DEV).bfloat16(),
              torch.ones(1, 48, device=DEV), torch.ones(1, 48, 48, device=DEV))
    with monkeypatch.context() as m:
        m.setattr(pairformer._host, "Stack", Broken)
        stream = torch.cuda.current_stream()
        with pytest.raises(ValueError, match="last dimension"):
            stack(*inputs)
        assert torch.cuda.current_stream() == stream
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            with pytest.raises(ValueError, match="last dimension"):
                stack(*inputs)
    torch.cuda.synchronize()
    stack._native = None
    assert all(torch.isfinite(t).all() for t in stack(*inputs)) and _lib.device_status() == 0


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("seq", [False, True])
def test_weights_refolded_by_their_layer_reach_the_stack(seq, graph):
    """Linear.load_weights writes parameters without counting as an edit; post_load_weights() of the layer that folds them
    is what makes it take effect, in the layer, in the native stack and in a recorded graph."""
    cls = b200.PairformerModule if seq else b200.PairformerNoSeqModule
    stack = _randomise(cls(num_blocks=2, dtype=torch.bfloat16, triangle_attn_backend="Heuristic", use_cuda_graph=graph).to(DEV))
    inputs = (torch.randn(1, 40, 40, 128, device=DEV).bfloat16(), torch.ones(1, 40, 40, device=DEV))
    if seq:
        inputs = (torch.randn(1, 40, 384, device=DEV).bfloat16(), inputs[0], torch.ones(1, 40, device=DEV), inputs[1])
    before = stack(*inputs)
    transition = stack.layers[1].transition_z
    transition.fc3.load_weights([{"weight": -transition.fc3.weight.clone()}])
    transition.post_load_weights()
    after = stack(*inputs)
    handle = stack.layers[0].register_forward_hook(lambda *args: None)  # a hooked layer is called itself
    stack.use_cuda_graph = False
    want = stack(*inputs)
    handle.remove()
    z = (lambda out: out[1]) if seq else (lambda out: out)
    assert not torch.equal(z(before), z(after)) and torch.equal(z(after), z(want))


def test_single_track_inputs_that_do_not_fit_are_refused():
    """Another width of s, or a residual that would have to be broadcast, is an error on the host and not a read outside
    the weights or the residual."""
    stack = b200.PairformerModule(num_blocks=1, dtype=torch.bfloat16, triangle_attn_backend="Heuristic").to(DEV)
    z, mask, pair = torch.randn(2, 24, 24, 128, device=DEV).bfloat16(), torch.ones(2, 24, device=DEV), torch.ones(2, 24, 24, device=DEV)
    for shape in ((2, 24, 512), (2, 24, 256), (1, 24, 384), (2, 23, 384)):
        with pytest.raises(ValueError):
            stack(torch.zeros(shape, device=DEV).bfloat16(), z, mask, pair)
    s = torch.zeros(2, 24, 384, device=DEV).bfloat16()
    for residual in (s[:1], s[:, :1], s[..., :128]):
        with pytest.raises(ValueError):
            stack.layers[0].attention(s, z, mask, residual=residual)


def test_row_lengths_of_another_shape_mean_their_values_in_order():
    """[B * N] and any other shape of B * N values are read as [B, N], also where that takes a copy."""
    node = _randomise(b200.TriangleAttentionStartingNode(128, 32, 4, dtype=torch.bfloat16).to(DEV))
    z = torch.randn(3, 20, 20, 128, device=DEV).bfloat16()
    lengths = torch.randint(1, 21, (3, 20), device=DEV, dtype=torch.int32)
    want = node(z, mask_bias=lengths)
    strided = torch.zeros(20, 3, 2, device=DEV, dtype=torch.int32)
    strided[..., 0] = lengths.reshape(20, 3)
    for other in (lengths.reshape(-1), lengths.reshape(20, 3), strided[..., 0], lengths.t().contiguous().t()):
        assert torch.equal(node(z, mask_bias=other), want)


def test_a_buffer_that_is_not_contiguous_is_replaced():
    node = _randomise(b200.TriangleAttentionStartingNode(128, 32, 4, dtype=torch.bfloat16).to(DEV))
    z = torch.randn(1, 40, 40, 128, device=DEV).bfloat16()
    buffers = {}
    want = node(z, buffers=buffers)
    workspace = buffers["tri_attn_workspace"]
    buffers["tri_attn_workspace"] = torch.zeros(1, dtype=torch.uint8, device=DEV).expand(workspace.shape)
    assert torch.equal(node(z, buffers=buffers), want) and buffers["tri_attn_workspace"].is_contiguous()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_masks_are_reduced_on_their_own_device():
    mask = (torch.rand(2, 40, 40) > 0.4).float()
    payload = b200.precompute_pair_masks("Heuristic", mask.to("cuda:1"))  # the current device is cuda:0
    assert payload.mask_bias.device.index == 1 and torch.equal(payload.mask_bias.cpu(), (mask > 0.5).sum(-1).int())
    assert torch.equal(payload.mask_bias_transposed.cpu(), (mask > 0.5).sum(-2).int())


def test_native_stack_on_many_streams_and_threads():
    """More caller's streams than side tracks are kept, and two threads on the same stream."""
    from concurrent.futures import ThreadPoolExecutor

    from bionemo_inference_runtime_b200.layers import pairformer

    stack = _randomise(b200.PairformerModule(num_blocks=3, dtype=torch.bfloat16, triangle_attn_backend="Heuristic").to(DEV))
    g = torch.Generator(device=DEV).manual_seed(5)
    mask, pair = torch.ones(1, 56, device=DEV), torch.ones(1, 56, 56, device=DEV)
    inputs = [(torch.randn(1, 56, 384, generator=g, device=DEV).bfloat16(),
               torch.randn(1, 56, 56, 128, generator=g, device=DEV).bfloat16(), mask, pair) for _ in range(10)]
    want = [stack(*i) for i in inputs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in inputs]

    def call(k, repeats=3):
        with torch.cuda.stream(streams[k]):
            for _ in range(repeats):
                out = stack(*inputs[k])
        streams[k].synchronize()
        return out

    for _ in range(2):
        for k, out in enumerate([call(k) for k in range(len(inputs))]):
            assert all(torch.equal(a, b) for a, b in zip(out, want[k]))
    assert len(pairformer._side_tracks) <= 8
    streams[1] = streams[0]  # two threads, one stream
    with ThreadPoolExecutor(2) as pool:
        for k, out in enumerate(pool.map(lambda k: call(k, 20), (0, 1))):
            assert all(torch.equal(a, b) for a, b in zip(out, want[k]))
    assert _lib.device_status() == 0
