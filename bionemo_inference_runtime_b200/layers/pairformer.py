"""Pairformer blocks on the sm_100a kernels.

Counterparts of ``PairformerLayerV1``, ``PairformerLayerV2``, ``PairformerNoSeqLayer``, ``PairformerNoSeqModule`` and
``PairformerModule`` (``bionemo_ir/_torch/layers/transformers/pairformer.py:44-510``).  Per block the pair track runs
triangle multiplication outgoing and incoming, triangle attention starting and ending node and the pair
transition, every update added to ``z`` (``_transform_z``, lines 174-216 of the same file); the single track
(``PairformerLayerV1.forward``, lines 218-252) then adds the attention with pair bias and the single transition to
``s``.  Submodule names (``attention``, ``tri_mul_out``, ``tri_mul_in``, ``tri_attn_start``, ``tri_attn_end``,
``transition_s``, ``transition_z``) and therefore the ``state_dict`` keys are the reference's, so a Pairformer
checkpoint loads unchanged.

The module can replay its whole stack from one CUDA graph (``use_cuda_graph=True``): at 15 kernel launches per block
the launch overhead is what the reference removes with graph capture at small token counts
(``bionemo_ir/_torch/graph_optimization/region.py``).
"""

from __future__ import annotations

import torch
import torch.nn as nn

from .. import _host
from .attention_backend import (AttentionMetadata, PrecomputedPairMasks, mask_to_lengths, precompute_pair_masks,
                                precompute_single_masks)
from .attention_pair_bias import AttentionPairBias
from .auto_chunk import CHUNK_REGISTRY, PAIR_TRANSITION
from .buffers import PreallocatedBuffers
from .transition import Transition
from .triangle_multiplication import (TriangleMultiplicationMetadata, TriangleMultiplicationNode,
                                      TriangleMultiplicationNodeType, precompute_trimul_metadata)
from .triangle_nodes import _EMPTY_ROW_MODES, TriangleAttentionEndingNode, TriangleAttentionStartingNode

# (device, caller's stream) -> the stream and events of the single track beside it; taken out while a call uses it.  The
# device is part of the key because stream handles are per device: the default stream's is 0 on every one.
_side_tracks: dict[tuple[torch.device, int], "_host.SideTrack"] = {}


class _LayersState:
    """The state of a stack's layers: their options, hooks and packed weights, and the parameters these were folded from.
    The objects are held, so that one replaced by another at its address does not look unchanged, and packed weights
    whose addresses a native stack or a graph has recorded stay allocated.  Not copied or pickled with the module."""

    def __init__(self, layers):
        self.objects, self.weights = _host.module_state(layers)

    def holds(self, layers) -> bool:
        return _host.same_state(self.objects, self.weights, layers)

    def __deepcopy__(self, memo):
        return None

    def __reduce__(self):
        return type(None), ()


class _NativeStack(_LayersState):
    """The packed weights of a stack in the form of ``_host.Stack`` (None: the stack has no such form), valid on one device
    and for the state that the layers are in now, with their weights packed."""

    def __init__(self, layers, device: torch.device, stack, chunk_policies):
        super().__init__(layers)
        self.device, self.stack, self.chunk_policies = device, stack, chunk_policies


def _native_stack(module: nn.Module, z: torch.Tensor) -> "_NativeStack | None":
    """The native form of ``module.layers`` for this call, or None when a layer has to be called itself: it is hooked or
    of another class, its options need the general path, or its rows are chunked at this size."""
    if nn.modules.module._has_any_global_hook():
        return None
    native = module.__dict__.get("_native")
    if native is None or native.device != z.device or not native.holds(module.layers):
        if torch.cuda.is_current_stream_capturing():
            return None  # folding weights now would only fill them at replay
        stack = _build_native_stack(module.layers, z.device)
        policies = {} if stack is None else {
            id(p): p for layer in module.layers
            for p in (layer.tri_attn_start.mha.chunk_policy, layer.tri_attn_end.mha.chunk_policy) if p is not None}
        # a stack that has no native form is remembered as well
        native = module._native = _NativeStack(module.layers, z.device, stack, list(policies.values()))
    if native.stack is None:
        return None
    chunked = any(p.chunk_size < z.shape[1] and p.should_chunk(z) for p in native.chunk_policies)
    return None if chunked else native


def _build_native_stack(layers, device):
    if _host.more_than_its_class(layers):  # hooked, compiled or patched
        return None
    bf16 = torch.bfloat16
    stack, first = _host.Stack(), layers[0]
    for layer in layers:
        if layer.no_update_s != first.no_update_s:
            return None  # one call walks both tracks of all blocks, or the pair track alone
        if type(layer) not in (PairformerLayerV1, PairformerLayerV2, PairformerNoSeqLayer) or layer.dtype != bf16:
            return None
        tri, nodes, trans = (layer.tri_mul_out, layer.tri_mul_in), (layer.tri_attn_start, layer.tri_attn_end), layer.transition_z
        if (any(type(t) is not TriangleMultiplicationNode or t.mean_normalization
                or t.pair_mask_left_aligned != first.tri_mul_out.pair_mask_left_aligned for t in tri)  # masked output: all or none
                or [int(t.multiplication_type) for t in tri] != [0, 1]
                or [type(n) for n in nodes] != [TriangleAttentionStartingNode, TriangleAttentionEndingNode]
                or [int(n.node_type) for n in nodes] != [0, 1]
                or any(n.dtype != bf16 or n.transposed_bias or not n.pair_mask_left_aligned for n in nodes)
                or type(trans) is not Transition or trans.dtype != bf16 or not trans._fused):
            return None
        args = []
        for t in tri:
            args += [t._packed(device), t.eps]
        for n in nodes:
            args += [n._packed(device), n.layer_norm.eps, _EMPTY_ROW_MODES[n.empty_row_mode]]
        stack.add(*args, trans._packed(device), trans._norm_eps())
        if layer.no_update_s:
            continue
        attn, trans = layer.attention, layer.transition_s
        if (type(attn) is not AttentionPairBias or type(trans) is not Transition or trans.dtype != bf16 or trans._fused
                or (isinstance(layer, PairformerLayerV2) and (not layer._pre_norm_folded or layer.post_norm_s is not None))
                or any(norm is not getattr(layer, "pre_norm_s", None) for norm in attn._input_norm)):  # (not in the state)
            return None
        w, t, norm = attn._weights(device), trans._packed(device), attn._norm_of_s()
        stack.add_single(w["w_in"], w["sc_in"], w["w_o"], w["sc_o"], w["packed_z"], norm is not None,
                         attn.eps if norm is None else norm.eps, attn.eps, attn.head_dim**-0.5, t["w1"], t["sc1"], t["w2"],
                         t["sc2"], trans.norm is not None, trans._norm_eps())
    return stack


def _native_pair_inputs(first, z: torch.Tensor, pair_mask: torch.Tensor, precomputed: PrecomputedPairMasks,
                        metadata: TriangleMultiplicationMetadata) -> tuple:
    """The pair track's inputs as the native stack takes them; the same conversions and rules as in the layers."""
    if tuple(pair_mask.shape) != tuple(z.shape[:3]):
        raise ValueError(f"mask must have shape {tuple(z.shape[:3])}, got {tuple(pair_mask.shape)}")
    z = z.to(torch.bfloat16)
    lengths = [m if m.dtype == torch.int32 else mask_to_lengths(m, z.shape[0], z.shape[1]).contiguous()
               for m in (precomputed.mask_bias, precomputed.mask_bias_transposed)]
    mask_output = metadata.outgoing_actual_seqlen is not None and first.tri_mul_out.can_fuse_residual(z)
    return z, pair_mask.to(torch.float32), *lengths, mask_output


class PairformerLayerV1(nn.Module):
    def __init__(self, layer_idx: int = 0, token_s: int = 384, token_z: int = 128, num_heads: int = 16,
                 pairwise_head_width: int = 32, pairwise_num_heads: int = 4, no_update_s: bool = False,
                 no_update_z: bool = False, dtype: torch.dtype = None, eps: float = 1e-5, inf: float = 1e9,
                 triangle_attn_backend: str = "VANILLA", pairwise_attn_backend: str = "VANILLA",
                 skip_create_weights: bool = False, attention_initial_norm: bool = False,
                 s_path_dtype: str | torch.dtype | None = None, trimul_high_precision: bool = True,
                 trimul_mean_normalization: bool = False, pair_mask_left_aligned: bool = True,
                 pair_transition_factor: int = 4, tri_attn_transposed_bias: bool = False, **kwargs):
        """Arguments as the reference layer takes them (pairformer.py:45-67).  ``s_path_dtype`` other than bfloat16
        is accepted and the single track still computes in bfloat16 (fp32 accumulation), returning ``s`` in the
        dtype it came in."""
        super().__init__()
        if no_update_z:
            raise ValueError("no_update_z is not supported: the pair track is the purpose of these kernels")
        self.dtype = dtype
        self.no_update_s, self.no_update_z = no_update_s, False
        self.token_s, self.token_z = token_s, token_z
        self.triangle_attn_backend = triangle_attn_backend
        self.pairwise_attn_backend = pairwise_attn_backend
        self.pair_mask_left_aligned = pair_mask_left_aligned
        self.s_path_dtype = s_path_dtype if s_path_dtype is not None else dtype
        if not no_update_s:
            self.attention = AttentionPairBias(layer_idx=layer_idx, c_s=token_s, c_z=token_z, num_heads=num_heads,
                                               dtype=torch.bfloat16, bias_proj=True, eps=eps, inf=inf,
                                               skip_create_weights=skip_create_weights,
                                               attn_backend=pairwise_attn_backend, initial_norm=attention_initial_norm)

        def trimul(kind):
            return TriangleMultiplicationNode(layer_idx=layer_idx, dim=token_z, eps=eps, multiplication_type=kind,
                                              dtype=dtype, skip_create_weights=skip_create_weights,
                                              high_precision=trimul_high_precision,
                                              mean_normalization=trimul_mean_normalization,
                                              pair_mask_left_aligned=pair_mask_left_aligned)

        self.tri_mul_out = trimul(TriangleMultiplicationNodeType.OUTGOING)
        self.tri_mul_in = trimul(TriangleMultiplicationNodeType.INCOMING)
        node_kw = dict(inf=inf, layer_idx=layer_idx, dtype=dtype, skip_create_weights=skip_create_weights,
                       attn_backend=triangle_attn_backend, pair_mask_left_aligned=pair_mask_left_aligned)
        self.tri_attn_start = TriangleAttentionStartingNode(token_z, pairwise_head_width, pairwise_num_heads, **node_kw)
        self.tri_attn_end = TriangleAttentionEndingNode(token_z, pairwise_head_width, pairwise_num_heads,
                                                        transposed_bias=tri_attn_transposed_bias, **node_kw)
        if not no_update_s:
            self.transition_s = Transition(token_s, token_s * 4, layer_idx=layer_idx, eps=eps, dtype=torch.bfloat16,
                                           skip_create_weights=skip_create_weights)
        self.transition_z = Transition(token_z, token_z * pair_transition_factor, layer_idx=layer_idx, eps=eps,
                                       dtype=dtype, skip_create_weights=skip_create_weights,
                                       auto_chunk_policy=CHUNK_REGISTRY.get(PAIR_TRANSITION))

    def _transform_z(self, z: torch.Tensor, pair_mask: torch.Tensor, trimul_metadata: TriangleMultiplicationMetadata,
                     attn_metadatas: dict[str, AttentionMetadata] | None = None,
                     precomputed_masks: PrecomputedPairMasks | None = None,
                     buffers: PreallocatedBuffers | None = None, inplace_safe: bool = False) -> torch.Tensor:
        can_update_inplace = inplace_safe and not torch.cuda.is_current_stream_capturing()
        # every step reads bfloat16: fp32 results of the triangle multiplications would only be converted back
        keep = self.dtype == torch.bfloat16
        z = self.tri_mul_out(z, mask=pair_mask, trimul_metadata=trimul_metadata, residual=True, buffers=buffers, _keep_bf16=keep)
        z = self.tri_mul_in(z, mask=pair_mask, trimul_metadata=trimul_metadata, residual=True, buffers=buffers, _keep_bf16=keep)
        if self.dtype is not None and z.dtype != self.dtype:
            z = z.to(self.dtype)
        tri_attn_metadata = (attn_metadatas or {}).get("triangle_attn")
        if precomputed_masks is not None:
            mb_start, mb_end = precomputed_masks.mask_bias, precomputed_masks.mask_bias_transposed
        else:
            mb_start = mb_end = None
        for node, node_mask_bias in ((self.tri_attn_start, mb_start), (self.tri_attn_end, mb_end)):
            z = node(z, mask=pair_mask, mask_bias=node_mask_bias, attn_metadata=tri_attn_metadata, buffers=buffers,
                     residual=True, inplace_residual=can_update_inplace)
        return self.transition_z(z, residual=True, inplace=True)

    def forward(self, s: torch.Tensor, z: torch.Tensor, mask: torch.Tensor, pair_mask: torch.Tensor,
                trimul_metadata: TriangleMultiplicationMetadata,
                attn_metadatas: dict[str, AttentionMetadata] | None = None,
                precomputed_masks: PrecomputedPairMasks | None = None, precomputed_single_masks=None,
                buffers: PreallocatedBuffers | None = None, **kwargs) -> tuple[torch.Tensor, torch.Tensor]:
        z = self._transform_z(z, pair_mask, trimul_metadata, attn_metadatas, precomputed_masks=precomputed_masks,
                              buffers=buffers, inplace_safe=bool(kwargs.get("inplace_safe", False)))
        if not self.no_update_s:
            s = self._transform_s(s, z, mask, attn_metadatas, getattr(precomputed_single_masks, "mask_bias", None), buffers,
                                  _key_counts=kwargs.get("_key_counts"))
        return s, z

    def _transform_s(self, s: torch.Tensor, z: torch.Tensor | None, mask: torch.Tensor,
                     attn_metadatas: dict[str, AttentionMetadata] | None, mask_bias: torch.Tensor | None,
                     buffers: PreallocatedBuffers | None, **shared) -> torch.Tensor:
        """The block's single track on the updated pair tensor (``shared``: what a stack has computed already)."""
        s_dtype = s.dtype
        # attention(..., residual=s) is the reference's ``s + attention(s, z, mask)`` with the add in the
        # output-projection kernel; the result is a fresh tensor, so the transition updates it in place
        s = self.attention(s, z, mask, attn_metadata=(attn_metadatas or {}).get("pairwise_attn"),
                           mask_bias=mask_bias, buffers=buffers, residual=s, **shared)
        return self.transition_s(s.to(torch.bfloat16), residual=True, inplace=True).to(s_dtype)


class PairformerLayerV2(PairformerLayerV1):
    def __init__(self, post_layer_norm: bool = False, **kwargs):
        """The v2 layer (pairformer.py:356-416): ``s + attention(pre_norm_s(s), z)``, the single transition and an
        optional ``post_norm_s``.  ``pre_norm_s`` is folded into the attention's in-projection when the attention
        has no initial norm of its own, so the single track stays the same five launches."""
        super().__init__(**kwargs)
        if self.no_update_s:
            raise ValueError("the v2 layer updates the single representation; use PairformerNoSeqLayer otherwise")
        self.post_layer_norm = post_layer_norm
        self.pre_norm_s = nn.LayerNorm(self.token_s, dtype=torch.bfloat16)
        self.post_norm_s = nn.LayerNorm(self.token_s, dtype=torch.bfloat16) if post_layer_norm else None
        self._pre_norm_folded = self.attention.norm_s is None
        if self._pre_norm_folded:
            self.attention.set_input_norm(self.pre_norm_s)

    def _transform_s(self, s: torch.Tensor, z: torch.Tensor | None, mask: torch.Tensor,
                     attn_metadatas: dict[str, AttentionMetadata] | None, mask_bias: torch.Tensor | None,
                     buffers: PreallocatedBuffers | None, **shared) -> torch.Tensor:
        s_dtype = s.dtype
        s16 = s.to(torch.bfloat16)
        s_in = s16 if self._pre_norm_folded else self.pre_norm_s(s16)
        s16 = self.attention(s_in, z, mask, attn_metadata=(attn_metadatas or {}).get("pairwise_attn"),
                             mask_bias=mask_bias, buffers=buffers, residual=s16, **shared)
        s16 = self.transition_s(s16, residual=True, inplace=True)
        if self.post_norm_s is not None:
            s16 = self.post_norm_s(s16)
        return s16.to(s_dtype)


class PairformerNoSeqLayer(PairformerLayerV1):
    def __init__(self, *, layer_idx: int, **kwargs):
        """The layer without the single track (pairformer.py:255-306); arguments as :class:`PairformerLayerV1`."""
        kwargs.pop("no_update_s", None)
        super().__init__(layer_idx=layer_idx, no_update_s=True, **kwargs)

    def forward(self, z: torch.Tensor, pair_mask: torch.Tensor, trimul_metadata: TriangleMultiplicationMetadata,
                attn_metadatas: dict[str, AttentionMetadata] | None = None,
                precomputed_masks: PrecomputedPairMasks | None = None, precomputed_single_masks=None,
                buffers: PreallocatedBuffers | None = None, inplace_safe: bool = False, **kwargs) -> torch.Tensor:
        return self._transform_z(z, pair_mask, trimul_metadata, attn_metadatas, precomputed_masks=precomputed_masks,
                                 buffers=buffers, inplace_safe=inplace_safe)


class PairformerModule(nn.Module):
    """The stack with the single track (pairformer.py:418-510).  The reference builds it from a config object;
    here the same fields are keyword arguments (``num_blocks``, ``token_s``, ``token_z``, ``num_heads``, ...), or a
    ``config`` object carrying them under the reference's names."""

    _CONFIG_FIELDS = {"num_blocks": "num_blocks", "token_s": "token_s", "token_z": "token_z", "num_heads": "num_heads",
                      "pairwise_head_width": "pairwise_head_width", "pairwise_num_heads": "pairwise_num_heads",
                      "no_update_s": "no_update_s", "torch_dtype": "dtype", "norm_epsilon": "eps", "mask_inf": "inf",
                      "skip_create_weights": "skip_create_weights",
                      "triangle_attention_backend": "triangle_attn_backend",
                      "pairwise_attention_backend": "pairwise_attn_backend",
                      "attention_initial_norm": "attention_initial_norm",
                      "trimul_high_precision": "trimul_high_precision",
                      "trimul_mean_normalization": "trimul_mean_normalization", "s_path_dtype": "s_path_dtype",
                      "tri_attn_transposed_bias": "tri_attn_transposed_bias", "post_layer_norm": "post_layer_norm"}

    def __init__(self, config=None, use_cuda_graph: bool = False, version: str = "v1", **kwargs):
        """``use_cuda_graph`` (not in the reference, whose graph capture lives in its runtime) records one forward
        of the whole stack per input shape and replays it; inputs are copied into the graph's buffers."""
        super().__init__()
        self.use_cuda_graph = use_cuda_graph
        self._graph = None
        self._graph_key = None
        self._graph_state = None
        self._graph_io = None
        if config is not None:
            version = getattr(config, "version", version)
            for field, name in self._CONFIG_FIELDS.items():
                if hasattr(config, field):
                    kwargs.setdefault(name, getattr(config, field))
        num_blocks = kwargs.pop("num_blocks", 8)
        if version not in ("v1", "v2"):
            raise ValueError(f"unknown pairformer layer version {version!r}")
        if version == "v1":
            kwargs.pop("post_layer_norm", None)  # the reference passes it to both; only v2 reads it
        layer_cls = PairformerLayerV1 if version == "v1" else PairformerLayerV2
        self.config = config
        self.layers = nn.ModuleList([layer_cls(layer_idx=i, **kwargs) for i in range(num_blocks)])
        self.pair_mask_left_aligned = self.layers[0].pair_mask_left_aligned if self.layers else False

    def forward(self, s: torch.Tensor, z: torch.Tensor, mask: torch.Tensor, pair_mask: torch.Tensor,
                attn_metadatas: dict[str, AttentionMetadata] | None = None,
                buffers: PreallocatedBuffers | None = None, **kwargs) -> tuple[torch.Tensor, torch.Tensor]:
        if not self.layers:
            return s, z
        if not (self.use_cuda_graph and z.is_cuda) or torch.cuda.is_current_stream_capturing():
            return self._run(s, z, mask, pair_mask, attn_metadatas, buffers, **kwargs)
        inputs = (s, z, mask, pair_mask)
        # the recorded kernels hold the addresses of the layers' packed weights and the values of their options: a
        # reload, an in-place edit of a parameter or another option must record a new graph
        key = tuple((t.shape, t.dtype, t.device) for t in inputs)
        if self._graph is None or key != self._graph_key or not self._graph_state.holds(self.layers):
            static = [t.clone() for t in inputs]
            graph_buffers: dict = {}
            side = torch.cuda.Stream(z.device)
            side.wait_stream(torch.cuda.current_stream(z.device))
            with torch.cuda.stream(side):
                self._run(*static, attn_metadatas, graph_buffers, **kwargs)  # warm-up: folds the weights
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=side):
                    outs = self._run(*static, attn_metadatas, graph_buffers, **kwargs)
            torch.cuda.current_stream(z.device).wait_stream(side)
            self._graph, self._graph_key, self._graph_io = graph, key, (static, outs, graph_buffers)
            self._graph_state = _LayersState(self.layers)
        static, outs, _ = self._graph_io
        for dst, src in zip(static, inputs):
            dst.copy_(src)
        self._graph.replay()
        return outs[0].clone(), outs[1].clone()

    def _run(self, s, z, mask, pair_mask, attn_metadatas, buffers, **kwargs):
        first = self.layers[0]
        precomputed = precompute_pair_masks(first.triangle_attn_backend, pair_mask, inf=first.tri_attn_start.inf,
                                            dtype=first.dtype)
        if buffers is None:
            buffers = {}
        int_lengths = precomputed.mask_bias.dtype == torch.int32
        trimul_metadata = precompute_trimul_metadata(
            z, precomputed.mask_bias if int_lengths else None,
            precomputed.mask_bias_transposed if int_lengths else None, enabled=self.pair_mask_left_aligned)
        # the key mask of the single track, reduced once for all layers (reference: pairformer.py:472-476)
        precomputed_single = None if first.no_update_s else precompute_single_masks(
            first.pairwise_attn_backend, mask, inf=first.attention.inf)
        if precomputed_single is not None:
            kwargs["_key_counts"] = first.attention.key_counts(mask, precomputed_single.mask_bias, s.shape[0], s.shape[1],
                                                               s.device)
            native = None if attn_metadatas or first.no_update_s else _native_stack(self, z)
            if native is not None:
                key = z.device, _host.current_stream()
                track = _side_tracks.pop(key, None) or _host.SideTrack()
                s_out, z = native.stack.run_both(s.to(torch.bfloat16).contiguous(),
                                                 *_native_pair_inputs(first, z, pair_mask, precomputed, trimul_metadata),
                                                 kwargs["_key_counts"], buffers, track)
                while len(_side_tracks) >= 8:  # programs use a few streams; a bounded number is kept
                    _side_tracks.pop(next(iter(_side_tracks)), None)
                _side_tracks[key] = track
                return s_out.to(s.dtype), z
        for layer in self.layers:
            s, z = layer(s, z, mask, pair_mask, trimul_metadata, attn_metadatas, precomputed_masks=precomputed,
                         precomputed_single_masks=precomputed_single, buffers=buffers, **kwargs)
        return s, z


class PairformerNoSeqModule(nn.Module):
    def __init__(self, num_blocks: int = 8, token_z: int = 128, pairwise_head_width: int = 32,
                 pairwise_num_heads: int = 4, use_cuda_graph: bool = False, **kwargs):
        """``use_cuda_graph`` (not in the reference, whose graph capture lives in its runtime) records one forward
        of the whole stack per (shape, mask object) and replays it; inputs are copied into the graph's buffers."""
        super().__init__()
        self.layers = nn.ModuleList([
            PairformerNoSeqLayer(layer_idx=i, token_z=token_z, pairwise_head_width=pairwise_head_width,
                                 pairwise_num_heads=pairwise_num_heads, **kwargs) for i in range(num_blocks)])
        self.pair_mask_left_aligned = self.layers[0].pair_mask_left_aligned if self.layers else False
        self.use_cuda_graph = use_cuda_graph
        self._graph = None
        self._graph_key = None
        self._graph_state = None
        self._graph_in = self._graph_mask = self._graph_out = None

    def _run(self, z, pair_mask, attn_metadatas, buffers, **kwargs):
        first = self.layers[0]
        precomputed = precompute_pair_masks(first.triangle_attn_backend, pair_mask, inf=first.tri_attn_start.inf,
                                            dtype=first.dtype)
        if buffers is None:
            buffers = {}
        int_lengths = precomputed.mask_bias.dtype == torch.int32
        trimul_metadata = precompute_trimul_metadata(
            z, precomputed.mask_bias if int_lengths else None,
            precomputed.mask_bias_transposed if int_lengths else None, enabled=self.pair_mask_left_aligned)
        native = _native_stack(self, z)
        if native is not None:
            return native.stack.run_pair(*_native_pair_inputs(first, z, pair_mask, precomputed, trimul_metadata), buffers)
        for layer in self.layers:
            z = layer(z, pair_mask, trimul_metadata, attn_metadatas, precomputed_masks=precomputed, buffers=buffers,
                      **kwargs)
        return z

    def forward(self, z: torch.Tensor, pair_mask: torch.Tensor,
                attn_metadatas: dict[str, AttentionMetadata] | None = None,
                buffers: PreallocatedBuffers | None = None, **kwargs) -> torch.Tensor:
        if not self.layers:
            return z
        if not (self.use_cuda_graph and z.is_cuda) or torch.cuda.is_current_stream_capturing():
            return self._run(z, pair_mask, attn_metadatas, buffers, **kwargs)
        # as in PairformerModule.forward
        key = (z.shape, z.dtype, z.device, pair_mask.shape, pair_mask.dtype)
        if self._graph is None or key != self._graph_key or not self._graph_state.holds(self.layers):
            self._graph_in, self._graph_mask = z.clone(), pair_mask.clone()
            graph_buffers: dict = {}
            side = torch.cuda.Stream(z.device)
            side.wait_stream(torch.cuda.current_stream(z.device))
            with torch.cuda.stream(side):
                self._run(self._graph_in, self._graph_mask, attn_metadatas, graph_buffers, **kwargs)  # warm-up, folds
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=side):
                    self._graph_out = self._run(self._graph_in, self._graph_mask, attn_metadatas, graph_buffers, **kwargs)
            torch.cuda.current_stream(z.device).wait_stream(side)
            self._graph, self._graph_key, self._graph_buffers = graph, key, graph_buffers
            self._graph_state = _LayersState(self.layers)
        self._graph_in.copy_(z)
        self._graph_mask.copy_(pair_mask)
        self._graph.replay()
        return self._graph_out.clone()
