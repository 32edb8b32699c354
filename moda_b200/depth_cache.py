"""In-place depth-KV cache for a stack of MoDA layers.

The reference's only in-tree caller rebuilds the depth cache before EVERY layer from the list of
all earlier layers' K/V (``torch.stack(..., dim=2)`` + ``reshape`` + ``contiguous``:
vision_tasks/deit/models.py:361-390), so a model of N layers copies O(N^2) K/V tensors per forward,
and autograd un-stacks as many gradients in the backward.  ``DepthKVCache`` keeps one persistent
``[B, T, Lmax, H, D]`` buffer per K and V instead: each layer's K/V is copied into its slot once
(``moda_b200_depth_append``), the attention kernels read the first ``L`` layers of the buffer in
place (``moda_problem.depth_rows_per_pos``), and in the backward every layer ADDS its depth
gradients into one gradient cache of the same layout, from which each producing layer takes its
slice.

    cache = DepthKVCache(B, T, n_layers - 1, Hkv, D, dtype, device)
    for blk in blocks:
        q, k, v = ...                                   # this layer's projections
        o = cache.attend(q, k, v, moda_group_num=G, is_causal=False)
        cache.append(k, v)                              # visible to the layers after this one

Autograd: ``append`` returns nothing to the caller but keeps a scalar token, an input of every later
``attend`` until the next ``append``, which takes it as an input in turn; the engine therefore runs
an ``append``'s backward only after all later layers have added their depth gradients, and that
backward hands the slot's slice of the gradient cache to the layer's ``k`` and ``v``.  (The nodes are
native: ``csrc/torch_binding.cpp``.)
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _cabi
from . import ops
from ._cabi import MODE_CAUSAL, MODE_CHUNK_VISIBLE, MODE_NONCAUSAL


class DepthKVCache:
    """K/V of the preceding layers at every position, written in place layer by layer."""

    def __init__(self, batch: int, seq_len: int, max_layers: int, num_kv_heads: int, head_dim: int,
                 dtype: torch.dtype = torch.bfloat16, device=None):
        assert max_layers >= 1
        self.B, self.T, self.capacity, self.H, self.D = batch, seq_len, max_layers, num_kv_heads, head_dim
        self.k = torch.empty(batch, seq_len * max_layers, num_kv_heads, head_dim, dtype=dtype, device=device)
        self.v = torch.empty_like(self.k)
        self.L = 0
        self._token: Optional[torch.Tensor] = None
        self._state = None               # gradient caches of the pass in progress, made by its first call

    def reset(self) -> None:
        """Start a new forward pass: no layers cached, gradient cache dropped."""
        self.L = 0
        self._token = None
        self._state = None

    def _grad(self, which: int) -> Optional[torch.Tensor]:
        return None if self._state is None else _cabi.native().cache_grads(self._state)[which]

    @property
    def grad_k(self) -> Optional[torch.Tensor]:
        """Gradient cache of ``k`` (allocated by the first backward that needs it)."""
        return self._grad(0)

    @property
    def grad_v(self) -> Optional[torch.Tensor]:
        return self._grad(1)

    def _pass_state(self):
        if self._state is None:
            self._state = _cabi.native().cache_state()
        return self._state

    # Copies and pickles hold the gradient caches as tensors: the native state is one of this process.
    def __getstate__(self):
        state = dict(self.__dict__)
        if self._state is not None:
            state["_state"] = tuple(_cabi.native().cache_grads(self._state))
        return state

    def __setstate__(self, state):
        self.__dict__.update(state)
        if state["_state"] is not None:
            self._state = _cabi.native().cache_state(*state["_state"])

    def bytes_copied_per_forward(self, n_layers: int) -> int:
        """Bytes of K/V this cache copies for a model of ``n_layers`` attention layers (each of the
        first n_layers - 1 layers once)."""
        per_layer = 2 * self.B * self.T * self.H * self.D * self.k.element_size()
        return (n_layers - 1) * per_layer

    def bytes_copied_by_rebuilding(self, n_layers: int) -> int:
        """The same for the rebuild-before-every-layer scheme of the reference caller: layer i
        stacks i earlier layers and makes the result contiguous."""
        per_layer = 2 * self.B * self.T * self.H * self.D * self.k.element_size()
        return sum(2 * i for i in range(n_layers)) * per_layer      # stack copy + contiguous copy

    # ------------------------------------------------------------------ forward API
    def append(self, k: torch.Tensor, v: torch.Tensor) -> None:
        """Copy this layer's ``k, v [B, T, H, D]`` into the next free slot."""
        assert self.L < self.capacity, "DepthKVCache is full"
        assert k.shape == (self.B, self.T, self.H, self.D) and v.shape == k.shape
        ops._check_tensors(k, v, self.k)
        self._token = _cabi.native().cache_append(k, v, self.k, self.v, self.capacity, self.L, self._token,
                                                  self._pass_state())
        self.L += 1

    def attend(self, q, k, v, scale=None, moda_group_num: int = 1, is_causal: bool = True,
               chunk_visible: bool = False, need_lse: bool = False):
        """MoDA attention of this layer over its own ``k, v`` and the cached layers (same results
        as ``parallel_moda`` / ``parallel_moda_chunk_visible`` on the stacked cache)."""
        mode = MODE_CHUNK_VISIBLE if chunk_visible else (MODE_CAUSAL if is_causal else MODE_NONCAUSAL)
        assert q.shape[1] == k.shape[1] * moda_group_num and q.shape[2] == k.shape[2]
        ops._check_tensors(q, k, v, self.k)
        r = _cabi.native().cache_attention(q, k, v, self.k, self.v, scale, moda_group_num, mode, self.L, self.capacity,
                                           self._token, self._pass_state())
        return r if need_lse else r[0]

    def _slot(self, x: torch.Tensor, slot: int) -> torch.Tensor:
        return x.view(self.B, self.T, self.capacity, self.H, self.D)[:, :, slot]
