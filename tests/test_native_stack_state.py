"""What the native form of a stack depends on, without a GPU: the kernels' side is replaced by recorders."""

import copy
import pickle
from types import SimpleNamespace

import pytest
import torch

import bionemo_inference_runtime_b200 as b200
from bionemo_inference_runtime_b200.layers import pairformer


def _stack(**options):
    return b200.PairformerModule(num_blocks=2, dtype=torch.bfloat16, triangle_attn_backend="Heuristic", **options)


def _inputs(device, n=8):
    return (torch.zeros(1, n, 384, device=device), torch.zeros(1, n, n, 128, device=device, dtype=torch.bfloat16),
            torch.ones(1, n), torch.ones(1, n, n))


def test_side_track_belongs_to_the_device_and_the_stream(monkeypatch):
    """Two devices ("cpu" and "meta" stand for them) whose current stream has the same handle take different tracks; a
    second call on a device takes the track of the first."""
    used = []

    def run_both(s, z, *args):
        used.append((z.device, args[-1]))
        return s, z

    monkeypatch.setattr(pairformer, "_native_stack", lambda module, z: SimpleNamespace(stack=SimpleNamespace(run_both=run_both)))
    monkeypatch.setattr(pairformer, "_side_tracks", {})
    monkeypatch.setattr(pairformer._host, "current_stream", lambda: 0)
    monkeypatch.setattr(pairformer._host, "SideTrack", object)
    stack = _stack()
    for device in ("cpu", "meta", "cpu", "meta"):
        stack._run(*_inputs(device), None, None)
    tracks = [track for _, track in used]
    assert tracks[0] is not tracks[1] and tracks[0] is tracks[2] and tracks[1] is tracks[3]


def test_packed_weights_of_one_device_are_not_used_on_another(monkeypatch):
    built = []
    monkeypatch.setattr(pairformer, "_build_native_stack", lambda layers, device: built.append(device) or object())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    stack = _stack()
    for device in ("cpu", "cpu", "meta", "meta"):
        pairformer._native_stack(stack, _inputs(device)[1])
    assert [d.type for d in built] == ["cpu", "meta"]


def test_an_option_replaced_at_its_old_address_is_seen(monkeypatch):
    """Two replacements between two calls: the second object may get the address of the one that was looked at."""
    built = []
    monkeypatch.setattr(pairformer, "_build_native_stack", lambda layers, device: built.append(1) or object())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    stack, z = _stack(), _inputs("cpu")[1]
    node = stack.layers[1].tri_mul_in
    node.eps = float("2e-5")
    pairformer._native_stack(stack, z)
    address = id(node.eps)
    node.eps = None
    others = []
    while len(others) < 1000 and (not others or id(others[-1]) != address):
        others.append(float("3e-5"))
    node.eps = others[-1]
    pairformer._native_stack(stack, z)
    pairformer._native_stack(stack, z)
    assert len(built) == 2


def test_a_parameter_replaced_at_its_old_address_is_seen():
    layer = b200.Transition(128, 512, dtype=torch.bfloat16).cpu()
    weight = layer.fc3.weight
    state, address = pairformer._host.weight_state(layer), weight.data_ptr()
    assert pairformer._host.same_weights(state, layer) and not pairformer._host.same_weights(None, layer)
    weight.data = torch.empty(0, dtype=torch.bfloat16)
    others = []
    while len(others) < 100 and (not others or others[-1].data_ptr() != address):
        others.append(torch.zeros(128, 512, dtype=torch.bfloat16))
    weight.data = others[-1]
    assert not pairformer._host.same_weights(state, layer)


def test_state_is_not_copied_with_a_layer():
    layer = b200.Transition(128, 512, dtype=torch.bfloat16).cpu()
    layer._pack_state = pairformer._host.weight_state(layer)
    stack = _stack()
    stack._native = pairformer._NativeStack(stack.layers, torch.device("cpu"), None, [])
    assert copy.deepcopy(layer)._pack_state is None and copy.deepcopy(stack)._native is None
    assert pickle.loads(pickle.dumps(layer))._pack_state is None and pickle.loads(pickle.dumps(stack))._native is None


def _patch_forward(layers):
    layers[1].tri_attn_end.forward = lambda *args, **kwargs: None


def _compile(layers):
    layers[1].transition_z._compiled_call_impl = lambda *args, **kwargs: None


def _one_without_single_track(layers):
    layers[1].no_update_s = True


def _one_without_masked_output(layers):
    layers[1].tri_mul_in.pair_mask_left_aligned = False


def _foreign_norm(layers):
    layers[1].attention.set_input_norm(torch.nn.LayerNorm(384))


@pytest.mark.parametrize("change", [_patch_forward, _compile, _one_without_single_track, _one_without_masked_output, _foreign_norm])
def test_layers_that_differ_from_the_native_form_are_called_themselves(monkeypatch, change):
    pack = torch.zeros(1)
    for cls in (b200.TriangleMultiplicationNode, b200.TriangleAttentionStartingNode, b200.TriangleAttentionEndingNode):
        monkeypatch.setattr(cls, "_packed", lambda self, device: pack)
    monkeypatch.setattr(b200.Transition, "_packed", lambda self, device: pack if self._fused else dict.fromkeys(("w1", "sc1", "w2", "sc2"), pack))
    monkeypatch.setattr(b200.AttentionPairBias, "_weights", lambda self, device: dict.fromkeys(("w_in", "sc_in", "w_o", "sc_o", "packed_z"), pack))
    layers = _stack().layers
    assert pairformer._build_native_stack(layers, "cpu") is not None
    change(layers)
    assert pairformer._build_native_stack(layers, "cpu") is None


@pytest.mark.parametrize("kind", ["parameter", "buffer", "attribute"])
def test_an_edited_weight_is_seen_whatever_it_is(kind):
    layer = b200.Transition(128, 512, dtype=torch.bfloat16).cpu()
    value = layer.fc3.weight.detach().clone()
    if kind != "parameter":
        del layer.fc3.weight
        if kind == "buffer":
            layer.fc3.register_buffer("weight", value)
        else:
            layer.fc3.weight = value
    state = pairformer._host.weight_state(layer)
    objects, weights = pairformer._host.module_state(layer)
    assert pairformer._host.same_weights(state, layer) and pairformer._host.same_state(objects, weights, layer)
    with torch.no_grad():
        layer.fc3.weight.zero_()
    assert not pairformer._host.same_weights(state, layer) and not pairformer._host.same_state(objects, weights, layer)
