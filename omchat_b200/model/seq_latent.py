"""Latent attention of the sequence-step decoders, host side: rotary tables, the work lists of the tensor-core kernel, and which kernel
attends (csrc/latent_attention.cu). Projections, norms and what is cached stay with the model.
"""
from __future__ import annotations

import json
from typing import Dict, List, Optional

import torch

from .. import seqlib
from ..config import RotarySpec


class RotaryTables:
    """fp32 (cos, sin) [positions, dims / 2, 2] per rotation, shared by the layers that turn alike; angles and functions are evaluated in
    double precision on the host. A table that grows leaves its predecessor alive: captured graphs hold its address."""

    def __init__(self, device):
        self.device = device
        self._tables: Dict[tuple, torch.Tensor] = {}
        self._outgrown: List[torch.Tensor] = []

    def get(self, rot: RotarySpec, positions: int) -> torch.Tensor:
        key = (rot.dims, rot.base, json.dumps(rot.scaling, sort_keys=True) if rot.scaling else None)
        t = self._tables.get(key)
        if t is None or t.shape[0] < positions:
            if t is not None:
                self._outgrown.append(t)
            n = max(positions, 1024)
            f, mult = rot.frequencies()
            ang = torch.arange(n, dtype=torch.float64)[:, None] * torch.tensor(f, dtype=torch.float64)[None, :]
            t = (torch.stack([ang.cos(), ang.sin()], dim=-1) * mult).to(torch.float32).contiguous().to(self.device)
            if t.numel() == 0:   # no rotated dimensions: the kernels still want a valid pointer
                t = torch.zeros(n, 1, 2, device=self.device)
            self._tables[key] = t
        return t


class LatentAttention:
    """Chooses the kernel and keeps the work lists. `plans` describes one step and collects its lists: {"portions": [...]} as the host
    knows the batch, {"decode_parts": n} or {"decode_keys": n} for a step of one row per request (the lists are then written on the
    device, in buffers that live as long as this object, so that a captured graph may use them; the tcgen05 kernel needs none), or None: the plain kernel."""

    def __init__(self, device, dtype: torch.dtype):
        self.device, self.dtype = device, dtype
        self.rotary = RotaryTables(device)
        self.tensor_attention = True    # False: the plain attention kernel for every shape (A/B, tests)
        self._decode_plans = {}         # (rows, heads, parts, window) -> seqlib.DecodeAttnPlan

    def _plan(self, plans: dict, T: int, H: int, r: int, window: int, pos, slot, tcgen05: bool):
        if tcgen05 and "portions" in plans:
            key = ("tcgen05", H, r, window)
            if key not in plans:
                plans[key] = self._tcgen05_pays(plans["portions"], H, r, window)
            tcgen05 = plans[key]
        plan = plans.get((H, window, tcgen05))
        if plan is None:
            if "portions" in plans:
                plan = self._prompt_plan(plans["portions"], H, self.device, window, tcgen05)
            else:
                keys = min(window, plans["decode_keys"]) if "decode_keys" in plans else 0
                parts = plans["decode_parts"] if "decode_parts" in plans else self._decode_parts(T, keys, tcgen05)
                if tcgen05:
                    plan = seqlib.DecodeRows(pos, slot, T, H, parts, window)
                else:
                    key = (T, H, parts, window)
                    plan = self._decode_plans.get(key)
                    if plan is None:
                        plan = self._decode_plans[key] = seqlib.DecodeAttnPlan(T, H, parts, self.device, window=window)
                    plan.fill(pos, slot)
            plans[(H, window, tcgen05)] = plan
        return plan

    @staticmethod
    def _tcgen05_pays(portions, H: int, r: int, window: int) -> bool:
        """Not where no row tile meets more than 64 keys: a tile of 128 is half empty then, and the mma.sync kernel starts on one of 64 sooner (64
        rows of 16 heads, latents of 512 / 256 / 128: 18 / 11.9 / 10.0 us there, 14.4 / 10.9 / 9.0; 100 keys: 18.2, 22.0). Nor for latents of 128,
        whose few products per key do not hide a tile's softmax, in steps of many tiles over short windows (1564 tiles, a window of 256: 160 us,
        134; 196 tiles: 48, 38; without a window 75, 187)."""
        tok = max(1, seqlib.MMA_ROWS // H)
        longest = max((min(p0 + n, window + tok - 1) for _, n, _, p0 in portions), default=0)
        return longest > (320 if r == 128 and sum(-(-n // tok) for _, n, _, _ in portions) >= 148 else 64)

    @staticmethod
    def _prompt_plan(portions, H: int, device, window: int, tcgen05: bool) -> seqlib.LatentAttnPlan:
        if not tcgen05:
            return seqlib.LatentAttnPlan(portions, H, device, window=window, mma_sync=True)
        # the tcgen05 kernel runs one CTA per SM on tiles of 128 keys: contexts are cut only while that leaves half the SMs idle
        return seqlib.LatentAttnPlan(portions, H, device, window=window, target_ctas=148, min_keys=128)

    @staticmethod
    def _decode_parts(T: int, keys: int, tcgen05: bool) -> int:
        """Key ranges per row of a decode-only step; of the mma.sync kernel 128 keys or more, 64 where a short window would leave SMs without a CTA."""
        if tcgen05:
            return seqlib.DecodeAttnPlan.parts_for_tcgen05(T, keys)
        parts = seqlib.DecodeAttnPlan.parts_for(T, keys)
        return parts if T * parts >= 148 else seqlib.DecodeAttnPlan.parts_for(T, keys, min_keys=64)

    def attend(self, qcat: torch.Tensor, r: int, dr: int, pool: torch.Tensor, cache, pos, slot, plans: Optional[dict], scale: float, *,
               sink: Optional[torch.Tensor] = None, window: Optional[int] = None, gate: Optional[torch.Tensor] = None) -> torch.Tensor:
        """qcat [T, H, r + dr] (absorbed query | rotated query) -> [T, H, r], the weighted sums of cached latents, times
        sigmoid(gate [T, H]) with a gate."""
        T, H = qcat.shape[0], qcat.shape[1]
        window = seqlib.WINDOW_ALL if window is None else min(window, seqlib.WINDOW_ALL)
        if plans is not None and self.tensor_attention and seqlib.latent_attn_mma_ok(H, r, dr, self.dtype):
            out = torch.empty(T, H, r, device=qcat.device, dtype=self.dtype)
            tcgen05 = seqlib.latent_attn_tcgen05_ok(H, r, dr, cache.page_size)
            return seqlib.latent_attn_mma(qcat, r, dr, pool, cache.block_table, cache.page_size, self._plan(plans, T, H, r, window, pos, slot, tcgen05), sink, scale,
                                          out, window=window, gate=gate)
        out = torch.empty(T, H, r, device=qcat.device, dtype=torch.float32)
        return seqlib.latent_attn(qcat, r, dr, pool, cache.block_table, cache.page_size, pos, slot, sink, scale, out, window=window, gate=gate)
