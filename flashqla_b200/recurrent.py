"""Recurrent GDN update: decode, spec-decode verify, tree verify, ragged sequences.

Host-side mirror of ``fused_sigmoid_gating_delta_rule_update``
(reference: flash_qla/ops/gated_delta_rule/recurrent_fused.py:6287-7537): same name, argument
order, defaults and error behaviour; the work is one launch of ``qla_recurrent_update`` in the
C-ABI library.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _cabi


def fused_sigmoid_gating_delta_rule_update(
    A_log: torch.Tensor,
    a: torch.Tensor,
    dt_bias: torch.Tensor,
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    b: torch.Tensor,
    initial_state_source: torch.Tensor,
    initial_state_indices: Optional[torch.Tensor] = None,
    scale: Optional[float] = None,
    softplus_beta: float = 1.0,
    softplus_threshold: float = 20.0,
    use_qk_l2norm_in_kernel: bool = True,
    cu_seqlens: Optional[torch.Tensor] = None,
    disable_state_update: bool = False,
    intermediate_states_buffer: Optional[torch.Tensor] = None,
    intermediate_state_indices: Optional[torch.Tensor] = None,
    cache_steps: Optional[int] = None,
    retrieve_parent_token: Optional[torch.Tensor] = None,
    block_dv: Optional[int] = None,
    assume_regular: bool = False,
    b_is_beta: bool = False,
    a_is_log_decay: bool = False,
) -> torch.Tensor:
    """One GDN step per token, state ``[slots, Hv, V, K]`` (fp32, or bf16 as an addition to the reference)
    updated in place; returns ``o``.  Out-of-range slots, parents or cu_seqlens boundaries never touch memory and
    are reported through ``check_device_status()``.

    ``g = a`` if ``a_is_log_decay`` else ``-exp(A_log) * softplus(a + dt_bias)``; ``beta = b`` if
    ``b_is_beta`` else ``sigmoid(b)``.  Unlike the reference, both flags are honoured on every
    path (the reference drops them outside single-token decode, recurrent_fused.py:7364-7393).
    ``block_dv`` is accepted for compatibility; values <= 16 select the 16-row tile.
    """
    if q.shape[0] != 1 or k.shape[0] != 1 or v.shape[0] != 1:
        raise ValueError("FlashQLA recurrent GDN kernel expects flattened [1, total_tokens, ...] inputs")
    if q.dtype != k.dtype or q.dtype != v.dtype:
        raise ValueError("q, k, and v must have the same dtype")
    if not q.is_cuda:
        raise ValueError("FlashQLA recurrent GDN kernel requires CUDA tensors")
    if a_is_log_decay:  # not used, whatever they are
        A_log = dt_bias = None
    return _cabi.host().recurrent_update(
        A_log, a, dt_bias, q, k, v, b, initial_state_source, initial_state_indices, scale, softplus_beta,
        softplus_threshold, use_qk_l2norm_in_kernel, cu_seqlens, disable_state_update, intermediate_states_buffer,
        intermediate_state_indices, cache_steps, retrieve_parent_token, block_dv, assume_regular, b_is_beta,
        a_is_log_decay)


flashqla_recurrent_gdn_update = fused_sigmoid_gating_delta_rule_update


def commit_verified_state(
    initial_state_source: torch.Tensor,
    intermediate_states_buffer: torch.Tensor,
    num_accepted: torch.Tensor,
    initial_state_indices: Optional[torch.Tensor] = None,
    intermediate_state_indices: Optional[torch.Tensor] = None,
) -> None:
    """After a verify step (``disable_state_update=True`` with ``intermediate_states_buffer``): write the state
    that follows the last ACCEPTED draft token of every sequence back into the pool, in place,
    ``state[initial_state_indices[n]] = intermediate[intermediate_state_indices[n], num_accepted[n] - 1]``;
    ``num_accepted[n] == 0`` leaves a sequence's state as it was.  Argument names follow
    ``fused_sigmoid_gating_delta_rule_update``; the reference leaves this step to its caller."""
    _cabi.host().state_commit(initial_state_source, intermediate_states_buffer, num_accepted, initial_state_indices,
                              intermediate_state_indices)
