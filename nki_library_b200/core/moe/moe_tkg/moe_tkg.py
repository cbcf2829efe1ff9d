"""``moe_tkg``: MXFP8 expert MLP for token generation, with the reference's signature
(core/moe/moe_tkg/moe_tkg.py:43-70)."""

from __future__ import annotations

import math
from typing import Optional

import torch

from .... import _lib, pipeline
from ....weights import DenseExpertWeights, ExpertWeights, prepare_dense_cached, prepare_from_nki_cached
from ...utils.common_types import ActFnType, ExpertAffinityScaleMode
from ...utils.kernel_call import kernel_entry
from ..moe_cte.group_tokens import moe_group_tokens
from ..moe_cte.moe_cte_utils import get_n_blocks

_PREFIX = "[MoE TKG Kernel]"
_BLOCK = 128


@kernel_entry
def moe_tkg(
    hidden_input: torch.Tensor,
    expert_gate_up_weights,
    expert_down_weights,
    expert_affinities: torch.Tensor,
    expert_index: torch.Tensor,
    is_all_expert: bool,
    rank_id: Optional[torch.Tensor] = None,
    expert_gate_up_bias: Optional[torch.Tensor] = None,
    expert_down_bias: Optional[torch.Tensor] = None,
    expert_gate_up_weights_scale: Optional[torch.Tensor] = None,
    expert_down_weights_scale: Optional[torch.Tensor] = None,
    hidden_input_scale: Optional[torch.Tensor] = None,
    gate_up_input_scale: Optional[torch.Tensor] = None,
    down_input_scale: Optional[torch.Tensor] = None,
    mask_unselected_experts: bool = False,
    expert_affinities_eager: Optional[torch.Tensor] = None,
    expert_affinities_scaling_mode: ExpertAffinityScaleMode = ExpertAffinityScaleMode.NO_SCALE,
    activation_fn: ActFnType = ActFnType.SiLU,
    output_dtype=None,
    gate_clamp_upper_limit: Optional[float] = None,
    gate_clamp_lower_limit: Optional[float] = None,
    up_clamp_upper_limit: Optional[float] = None,
    up_clamp_lower_limit: Optional[float] = None,
    output_in_sbuf: bool = False,
    is_all_expert_dynamic: bool = False,
    block_size: int = None,
    _impl: int = 0,
    _check_status: bool = False,
    _prequantized=None,
) -> torch.Tensor:
    """Decode MoE expert layer, ``[T, H]`` in, ``[T, H]`` out.

    Selective mode (``is_all_expert=False``) runs each token through its
    ``expert_index[t, :]`` experts; every *active* expert's weights are streamed
    from HBM once, however many tokens picked it.  All-expert mode runs every
    token through the local experts ``[E_L * rank_id, E_L * (rank_id + 1))`` with
    the affinity columns sliced (and optionally masked by ``expert_index``) the
    way ``mask_expert_affinities`` does (core/moe/moe_tkg/moe_tkg_affinity_masking.py:31-117).
    ``is_all_expert_dynamic`` computes, per local expert, only the tokens whose masked affinity is non-zero.
    A rank whose columns lie past the table and a token whose mask names an expert outside it give NaN rows.
    Weights are the reference's x4-packed MXFP8 tensors with their scales, or a
    prepared :class:`~nki_library_b200.weights.ExpertWeights` passed as
    ``expert_gate_up_weights``.  Non-MX weights -- 4-D ``[E_L, H, 2, I]`` bf16, or fp8 with the per-row factors
    ``[E_L, 2, I]`` / ``[E_L, H]`` in the two scale arguments -- run on the dense bf16 kernels.  SBUF-resident
    tensors, pre-quantised hidden states and static (per-tensor input) quantisation are rejected.
    """
    A = _lib.kernel_assert
    A(not output_in_sbuf, f"{_PREFIX} output_in_sbuf has no meaning on a GPU")
    A(hidden_input_scale is None, f"{_PREFIX} pre-quantised hidden_input (hidden_input_scale) is not supported")
    A(gate_up_input_scale is None and down_input_scale is None,
      f"{_PREFIX} Static quantization is not supported in MoE TKG kernel")
    A(expert_affinities_scaling_mode != ExpertAffinityScaleMode.PRE_SCALE_DELAYED,
      f"{_PREFIX} PRE_SCALE_DELAYED option is only applicable in CTE expert_mlp case")
    A(expert_affinities_scaling_mode != ExpertAffinityScaleMode.PRE_SCALE,
      f"{_PREFIX} Kernel does not support pre-scale mode")
    if is_all_expert_dynamic:
        A(is_all_expert, f"{_PREFIX} is_all_expert_dynamic=True requires is_all_expert=True, but got {is_all_expert=}")
        A(block_size is not None,
          f"{_PREFIX} is_all_expert_dynamic=True requires block_size != None, but got {block_size=}")
    if is_all_expert:
        A(expert_affinities_eager is None,
          f"{_PREFIX} expert_affinities eager mode not supported with is_all_expert=True")
    _lib.require_cuda(hidden_input, expert_affinities, expert_index, rank_id)
    A(hidden_input.dim() == 2, f"{_PREFIX} hidden_input must be [T, H]")
    T, H = hidden_input.shape
    A(T <= 128 or is_all_expert,
      f"{_PREFIX} Currently only batch size * seq len <= 128 is supported (except for all-expert mode)")

    dense = isinstance(expert_gate_up_weights, DenseExpertWeights) or (
        isinstance(expert_gate_up_weights, torch.Tensor) and expert_gate_up_weights.dim() == 4)
    if dense:
        # non-MX weights: bf16 [E_L, H, 2, I] / [E_L, I, H], or fp8 with per-row factors [E_L, 2, I] / [E_L, H]
        # (core/moe/moe_tkg/all_expert_impl.py:65, selective_expert_impl.py:45; CPU definition moe_tkg_torch.py:226-290)
        weights = expert_gate_up_weights if isinstance(expert_gate_up_weights, DenseExpertWeights) else \
            prepare_dense_cached(expert_gate_up_weights, expert_down_weights, expert_gate_up_bias, expert_down_bias,
                                 expert_gate_up_weights_scale, expert_down_weights_scale)
    elif isinstance(expert_gate_up_weights, ExpertWeights):
        weights = expert_gate_up_weights
    else:
        A(expert_gate_up_weights_scale is not None and expert_down_weights_scale is not None,
          f"{_PREFIX} Scales must be set when using MX weights")
        weights = prepare_from_nki_cached(expert_gate_up_weights, expert_gate_up_weights_scale, expert_down_weights,
                                          expert_down_weights_scale, expert_gate_up_bias, expert_down_bias)
    A(weights.H == H, f"{_PREFIX} weight hidden size {weights.H} does not match hidden_input ({H})")
    E_L = weights.E
    post_scale = expert_affinities_scaling_mode == ExpertAffinityScaleMode.POST_SCALE
    hidden = hidden_input.to(torch.bfloat16).contiguous()
    dev = hidden.device
    out = torch.empty((T, H), dtype=torch.bfloat16, device=dev)
    clamps = ((gate_clamp_lower_limit, gate_clamp_upper_limit), (up_clamp_lower_limit, up_clamp_upper_limit))

    if not is_all_expert:
        idx = expert_index.to(torch.int32).contiguous()
        K = idx.shape[1]
        E = expert_affinities.shape[1]
        A(E == E_L, f"{_PREFIX} selective mode needs all {E} experts local, got {E_L}")
        n_blocks = get_n_blocks(T, K, E, _BLOCK)
        ws = (pipeline.get_dense_workspace if dense else pipeline.get_workspace)(n_blocks * _BLOCK, H, weights.I, dev)
        g = moe_group_tokens(idx, E, _BLOCK, n_blocks, skip_token=True, _tile_flags=ws.tile_flags)
        aff = None
        if post_scale:
            aff = expert_affinities.contiguous()
            if aff.dtype not in (torch.float32, torch.bfloat16):
                aff = aff.float()
        _run(weights, hidden, T, weights, g["token_position_to_id"], g["block_to_expert"], g["conditions"],
             _BLOCK, aff, g["inverse_map"], out, activation_fn.value, clamps[0], clamps[1], _impl, _check_status,
             workspace=ws, flags_ready=True)
    else:
        E = expert_affinities.shape[1]
        if post_scale:
            A(rank_id is not None, f"{_PREFIX} rank_id is required for all-expert mode with affinity scaling")
        # local expert columns [E_L * rank_id, E_L * (rank_id + 1)), taken with a device-side index so that the
        # rank tensor never has to travel to the host (moe_tkg_affinity_masking.py:31-117)
        want_aff = post_scale or is_all_expert_dynamic
        A(expert_affinities.device == dev, f"{_PREFIX} expert_affinities must be on the device of hidden_input")
        aff = local_affinities(expert_affinities, E_L, T, rank_id,
                               expert_index if mask_unselected_experts else None) if want_aff else None
        if is_all_expert_dynamic:
            # dynamic control flow: per expert only the tokens routed to it (non-zero masked affinity) are
            # gathered into blocks and computed (all_expert_mx_impl.py:276-350); the block bookkeeping is the
            # prefill grouping on the masked affinities, and the blocks of experts nobody chose never run
            A(block_size > 0 and T % block_size == 0, f"{_PREFIX} block_size must evenly divide T")
            n_blocks = E_L * math.ceil(T / _BLOCK)
            g = moe_group_tokens(aff, E_L, _BLOCK, n_blocks, skip_token=True, want_inverse=False)
            tpi, b2e, cond = g["token_position_to_id"], g["block_to_expert"], g["conditions"]
            table = torch.empty((T, E_L), dtype=torch.int32, device=dev)
            _lib.call("b200moe_build_position_table", _lib.ptr(tpi), _lib.ptr(b2e), _lib.ptr(cond), n_blocks, _BLOCK,
                      T, E_L, _lib.ptr(table), _lib.stream_ptr())
        else:
            cond = None
        kw = {}
        if not is_all_expert_dynamic:
            if _prequantized is not None and not dense:
                # the caller (moe_block_tkg) has run the fused RMSNorm + quantise kernel into this workspace
                ws, (tpi, b2e, table) = _prequantized
                kw = dict(workspace=ws, prequantized=True, flags_ready=True)
            else:
                tpi, b2e, table = all_expert_layout(T, E_L, dev)
        _run(weights, hidden, T, weights, tpi, b2e, cond, _BLOCK, aff if post_scale else None, table, out,
             activation_fn.value, clamps[0], clamps[1], _impl, _check_status, **kw)
    if output_dtype is not None and output_dtype != torch.bfloat16:
        return out.to(output_dtype)
    return out


def all_expert_layout(T: int, E_L: int, device):
    """Static block layout of the all-expert mode: every local expert owns ceil(T / 128) blocks that hold tokens
    0..T-1 in order.  Returns ``(token_position_to_id, block_to_expert, table [T, E_L])``."""
    Tpad = math.ceil(T / _BLOCK) * _BLOCK
    tpi = torch.empty(E_L * Tpad, dtype=torch.int32, device=device)
    b2e = torch.empty(E_L * Tpad // _BLOCK, dtype=torch.int32, device=device)
    table = torch.empty((T, E_L), dtype=torch.int32, device=device)
    _lib.call("b200moe_all_expert_setup", T, E_L, _BLOCK, _lib.ptr(tpi), _lib.ptr(b2e), _lib.ptr(table), None, _lib.F32, 0,
              None, 0, None, 0, None, _lib.stream_ptr())
    return tpi, b2e, table


def local_affinities(expert_affinities: torch.Tensor, E_L: int, T: int, rank_id, expert_index) -> torch.Tensor:
    """fp32 ``[T, E_L]``: this rank's columns of the affinity table, multiplied by 0 where ``expert_index`` (None = keep
    all) does not name the expert.  The rank is read on the device and never travels to the host, so what cannot be checked
    here shows in the result: columns past the table, and every column of a token with an expert id outside ``[0, E)``,
    are NaN."""
    E = expert_affinities.shape[1]
    dev = expert_affinities.device
    _lib.kernel_assert((rank_id is None or rank_id.device == dev) and (expert_index is None or expert_index.device == dev),
                       f"{_PREFIX} expert_affinities, expert_index and rank_id must be on one device")
    _lib.kernel_assert(rank_id is None or rank_id.numel() > 0, f"{_PREFIX} rank_id must hold the rank")
    aff = expert_affinities.expand(T, E) if expert_affinities.shape[0] == 1 else expert_affinities
    _lib.kernel_assert(aff.shape[0] == T or (expert_index is None and aff.shape[0] > T),
                       f"{_PREFIX} expert_affinities must hold one row per token")
    aff = aff.contiguous()
    if aff.dtype not in (torch.float32, torch.bfloat16):
        aff = aff.float()
    rank = None if rank_id is None else rank_id.reshape(-1)[:1]
    if rank is not None and rank.dtype not in (torch.int32, torch.int64):
        rank = rank.to(torch.int64)
    idx, K = None, 0
    if expert_index is not None:
        idx = expert_index
        if idx.dtype not in (torch.int32, torch.uint32):
            idx = (idx.clamp(-1, E) if idx.dtype == torch.int64 else idx).to(torch.int32)
        _lib.kernel_assert(idx.shape[0] <= T, f"{_PREFIX} expert_index must hold one row per token")
        if idx.shape[0] < T:  # a token without a row selects nothing
            idx = torch.nn.functional.pad(idx.view(torch.int32), (0, 0, 0, T - idx.shape[0]), value=-2 ** 31)
        idx, K = idx.contiguous(), idx.shape[1]
    out = torch.empty((T, E_L), dtype=torch.float32, device=aff.device)
    _lib.call("b200moe_all_expert_setup", T, E_L, _BLOCK, None, None, None, _lib.ptr(aff), _lib.dtype_code(aff), E,
              _lib.ptr(rank), 0 if rank is None else rank.element_size(), _lib.ptr(idx), K, _lib.ptr(out),
              _lib.stream_ptr())
    return out


def _run(weights, *args, **kw):
    """MX weights go through the block-scaled kernels, dense weights through the bf16 ones."""
    if isinstance(weights, DenseExpertWeights):
        return pipeline.run_blocks_dense(*args, **kw)
    return pipeline.run_blocks(*args, **kw)
