"""An attention-only stack runner over the C ABI: the part of Hydra's TextModelRunner protocol
(Sources/HydraMetal/TextModelRunner.swift:14-95) that the attention path carries.

The reference's runners embed tokens, run every layer (attention half and mixture-of-experts half)
and project to logits.  Only the attention half is in this library, so the runner here takes and
returns HIDDEN STATES instead of tokens and logits and runs, per layer, the attention block of
ReferenceLayer.decode (Sources/HydraReference/ReferenceLayer.swift:126-187), all layers in one call
of the library (hc_attention_stack_host), because a token's kernels take less time than calling them
one by one from here does:

    normed = rms_norm(hidden, input_norm)                      hc_rms_norm
    q, k, v = normed W_q^T + b_q, ...                           hc_linear_group (one launch)
    rotate q and k, append k and v, attend (sinks, window)      hc_layer_step
    hidden += attention W_o^T + b_o                             hc_linear with the residual

with the protocol's bookkeeping around it: `position`, `prefill` in chunks of `prefill_chunk_tokens`
(the reference's loop: every chunk through every layer before the next chunk), `forward` for one
token, `verify` (a draft's tokens in one pass, one output per position: the prefill kernels
already return every position), `can_rewind` / `rewind` / `reset` on the KV cache.  Device memory
comes from torch; nothing here computes.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import List, Optional, Sequence

import numpy as np

from . import capi
from .backend import AttentionBackend, AttnParams, Context, KVCache, RopeTable, _check, _ptr

_WEIGHTS = ("input_norm", "wq", "bq", "wk", "bk", "wv", "bv", "wo", "bo")       # as hc_block_weights has them


@dataclass
class AttentionLayerWeights:
    """One layer's attention weights as Hydra stores them: bf16, projections row-major [out][in]."""
    input_norm: np.ndarray      # [hidden]
    wq: np.ndarray              # [q_heads * head_dim][hidden]
    bq: np.ndarray
    wk: np.ndarray              # [kv_heads * head_dim][hidden]
    bk: np.ndarray
    wv: np.ndarray
    bv: np.ndarray
    wo: np.ndarray              # [hidden][q_heads * head_dim]
    bo: np.ndarray
    sinks: Optional[np.ndarray] = None      # [q_heads]
    window: int = 0                         # 0 = full causal
    inv_freq: Optional[Sequence[float]] = None
    rope_concentration: float = 1.0


class AttentionStackRunner:
    """Hidden states in, hidden states out, through the attention blocks of a stack of layers."""

    prefill_chunk_tokens = 256          # TextModelRunner.prefillChunkTokens

    def __init__(self, ctx: Context, layers: List[AttentionLayerWeights], hidden: int, q_heads: int, kv_heads: int,
                 head_dim: int, context_length: int, eps: float = 1e-5, prefill_chunk_tokens: Optional[int] = None):
        import torch
        self.torch = torch
        self.ctx = ctx
        self.hidden, self.q_heads, self.kv_heads, self.d = hidden, q_heads, kv_heads, head_dim
        self.eps = eps
        if prefill_chunk_tokens is not None:
            self.prefill_chunk_tokens = prefill_chunk_tokens
        self.backend = AttentionBackend(ctx)
        self.kv_cache = KVCache(ctx, [dict(q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, window=w.window)
                                      for w in layers], context_length, prefill_chunk=self.prefill_chunk_tokens)
        bf = torch.bfloat16

        def dev(array):
            return torch.from_numpy(np.ascontiguousarray(array, dtype=np.float32)).cuda().to(bf)

        self.weights, self.tables, self.params = [], [], []
        for w in layers:
            t = {name: dev(getattr(w, name)) for name in _WEIGHTS}
            t["sinks"] = dev(w.sinks) if w.sinks is not None else None
            self.weights.append(t)
            table = RopeTable(ctx, list(w.inv_freq), context_length, w.rope_concentration) if w.inv_freq is not None else None
            self.tables.append(table)
            self.params.append(AttnParams(q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, window=w.window,
                                          sm_scale=1.0 / np.sqrt(head_dim), io_dtype=capi.HC_BF16, sinks=t["sinks"],
                                          rope=table))

        # What a call needs besides the hidden states: the C structs of the layers (filled on every pass), the
        # device workspace, and pinned host buffers (a copy from or to pageable memory is two).
        self._blocks = (capi.BlockWeightsStruct * len(layers))()
        # A block begins with the nine weight pointers; as one array they are stored by one assignment.
        self._parts = [(block, (ctypes.c_void_p * len(_WEIGHTS)).from_buffer(block)) for block in self._blocks]
        self._fill_blocks()
        self._lib = capi.load()
        chunk = self.prefill_chunk_tokens
        need = self._lib.hc_attention_stack_bytes(self._blocks, len(layers), chunk, hidden)
        self._workspace = torch.empty(need, dtype=torch.uint8, device="cuda")
        self._pinned = [torch.empty((chunk, hidden), dtype=torch.float32, pin_memory=True) for _ in range(2)]
        self._host = [p.numpy() for p in self._pinned]

    # -- TextModelRunner's bookkeeping ------------------------------------------------------------
    @property
    def position(self) -> int:
        return self.kv_cache.length()

    def can_rewind(self, to: int) -> bool:
        return self.kv_cache.can_rewind(to)

    def rewind(self, to: int) -> None:
        self.kv_cache.rewind(to)

    def reset(self) -> None:
        self.kv_cache.reset()

    # -- the passes -------------------------------------------------------------------------------
    def _fill_blocks(self) -> None:
        """The layers' weights and parameters as they are now: a program may have put other tensors in the lists."""
        for (block, pointers), t, params in zip(self._parts, self.weights, self.params):
            try:
                pointers[:] = [t[name].data_ptr() for name in _WEIGHTS]
            except AttributeError:                             # no bias, or a plain address
                pointers[:] = [_ptr(t[name]) for name in _WEIGHTS]
            block.params = params.struct()

    def _layers(self, tokens: int, first_position: int) -> None:
        """`tokens` hidden states from the first pinned buffer through every layer's attention block to the second."""
        self._fill_blocks()
        _check(self._lib.hc_attention_stack_host(
            self.ctx.handle, self.kv_cache.handle, self._blocks, len(self._parts), 0, self._pinned[0].data_ptr(),
            self._pinned[1].data_ptr(), tokens, self.hidden, first_position, self.eps, self._workspace.data_ptr(), None))

    def prefill(self, hidden_states: np.ndarray) -> np.ndarray:
        """A prompt's hidden states [tokens][hidden] in chunks, each chunk through every layer before
        the next (ModelRunner.prefill's order); returns the last position's output, as the protocol's
        prefill returns the last position's logits."""
        out = self.verify(hidden_states)
        return out[-1]

    def forward(self, hidden_state: np.ndarray) -> np.ndarray:
        """One token: TextModelRunner.forward(token:)."""
        return self.verify(np.asarray(hidden_state, np.float32).reshape(1, self.hidden))[0]

    def verify(self, hidden_states: np.ndarray) -> np.ndarray:
        """Several tokens in one pass, one output per position (TextModelRunner.verify): the caller
        keeps the accepted prefix by rewinding to it."""
        states = np.asarray(hidden_states, np.float32).reshape(-1, self.hidden)
        outputs = np.empty_like(states)
        total, chunk = states.shape[0], self._host[0].shape[0]
        for start in range(0, total, chunk):
            n = min(chunk, total - start)
            self._host[0][:n] = states[start:start + n]
            self._layers(n, self.position)
            outputs[start:start + n] = self._host[1][:n]
            self.kv_cache.advance(n)
        return outputs

    def close(self) -> None:
        self.kv_cache.close()
        for table in self.tables:
            if table is not None:
                table.close()
