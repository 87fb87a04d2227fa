"""Latent attention: queries, keys and values through low-rank latents, and a cache of the latents alone.

For the rows of a step, with H heads, D unrotated and R rotated query/key values per head, V value values per head,
a query latent of `q_rank` and a key/value latent of C = `kv_rank` values:
    cq = RMSNorm(h Wdq^T) * w_dq;   q = cq Wuq^T, per head [D unrotated | R rotated]
    [c_raw | r_raw] = h Wdkv^T (C + R values; one product with Wdq over the stacked weight);   c = RMSNorm(c_raw) * w_dkv;   r = rotate(r_raw) (one part for all heads)
    per head: k = [Wuk_h c | r],  v = Wuv_h c,   s = (q_plain . Wuk_h c + rotate(q_rot) . r) * scale
    o = softmax over the keys lo..p (lo = 0, or p - window + 1 under a sliding window) of s, times v
    residual += o Wo^T
Only [c | r] is cached, one vector per token (a cache entry of one plane).  The rotation pairs neighbours
(2i, 2i + 1) of the first `rot_dims` values of the rotated part by the angle p * base^(-2i / rot_dims).  The general
kernels (csrc/latent_attention.cu) never make keys or values of cached tokens: the query goes through Wuk once, the
weighted sum of latents through Wuv once.  For requests with many rows a step makes them once, in a workspace, and the
rows' attention over them runs on the tensor cores (csrc/latent_prompt_tc.cu).

Options for designs that vary it:
    q_rank None        no query latent: q = h Wq^T straight from the input (tensor role `q` instead of dq, dq.norm, uq)
    pairing "halves"   rotation pair i is (i, i + rot_dims / 2) instead of neighbours
    rot_scaling        (factor, original, fast, slow): frequencies blended for contexts longer than the original one and
                       a factor on cosines and sines (`parts.rope.blended_frequencies`); the score scale stays as given
    gate True          the concatenated heads are multiplied by sigmoid(h Wg^T) before the output product (role `g`)
Whatever reads h is one product over the stacked weight.
"""
from __future__ import annotations

from typing import Dict, Optional

import numpy as np
import torch

from .. import ops, runtime
from ..cache.manager import KVSpec
from ..weights.spec import TensorSpec
from .base import Part, PartPlan, Precision, StepBatch, StepShape
from .linear import Linear, add_product, stored_product
from .rope import blended_frequencies, power_frequencies


# Requests that bring at least this many rows, and one for this many of the keys they see, have their keys and values made
# (csrc/latent_prompt_tc.cu): making them costs the same for one row as for many.  Their tiles walk all keys one stage after the
# other, a block a tile and head, so when the step has few tiles its time is that of the longest walk, once for every group of
# heads, while the general form cuts keys into ranges that fill the device: beyond PROMPT_FEW_KEYS keys the step's rows x heads (weighted by their
# keys) must also reach `_rows_needed`.  Measured, us, that form / the general one:
#   16 heads of 128 + 64 over latents of 512, one group: after nothing 32 rows 46 / 50, 512 rows 80 / 419; after 1,000 tokens 32 rows 93 / 106;
#   after 2,000 32 rows 148 / 134, 40 148 / 175; after 4,000 32 rows 265 / 181, 40 269 / 259, 48 269 / 294; after 8,000 48 rows
#   490 / 484, 64 490 / 607; two groups after 12,000 96 rows 1,291 / 1,236, 128 1,302 / 1,557
#   32 heads: after 4,000 32 rows 310 / 359; two groups after 5,000 48 rows 644 / 550, 64 648 / 722; four after 16,000 128 rows 3,388 / 3,823
#   several requests, 16 heads: 2 x 32 rows after 4,000 312 / 359, 4 x 33 after 2,000 228 / 433; in groups 2 x 32 after 8,000 974 / 609,
#   8 x 32 after 4,000 (four groups) 1,231 / 1,123
PROMPT_ROWS, PROMPT_KEYS_A_ROW, PROMPT_FEW_KEYS = 32, 128, 1280


def _rows_needed(keys: int, groups: int) -> int:
    """Rows x heads from which making keys and values is the faster form, for walks of `keys` keys and heads in `groups`."""
    return 480 + keys // 24 if groups == 1 else groups * (900 + 600000 // keys)


# The workspace of made keys and values: heads are taken in groups that fit these bytes, or what the general form's queries
# and sums over the same rows would take if that is more.
PROMPT_BYTES = 256 << 20


class _TilePlan(PartPlan):
    """How a step's rows are cut for the kernels.  A run is a stretch of neighbouring rows for the tiled kernels: (first row,
    rows, first int, tiles, key ranges), its ints (first row in the stretch, rows) per tile, rows of one request each.
    `whole` is the run of all rows.  `wide`, where some requests have many rows: (first int of those requests, how many, the
    largest share of the workspace, first int of their tiles, how many, workspace tokens, heads a group); `runs` are then the
    stretches between them.  All follows the step's row counts and the context it has room for, so a recorded step's plan
    never changes."""

    def __init__(self, whole, runs, wide, ints):
        self.whole, self.runs, self.wide = whole, runs, wide
        self.values = np.asarray(ints, dtype=np.int32)
        self.ints = int(self.values.size)

    def fill(self, histories, out: np.ndarray) -> None:
        out[:self.ints] = self.values


class LatentAttention(Part):
    def __init__(self, hidden: int, heads: int, key_dim: int, rot_dim: int, value_dim: int, q_rank: Optional[int], kv_rank: int,
                 scale: float, rot_base: float, rot_dims: int, norm_eps: float, window: Optional[int] = None,
                 pairing: str = "neighbours", rot_scaling=None, gate: bool = False):
        if rot_dims % 2 or rot_dims > rot_dim or rot_dims < 0:
            raise ValueError("latent attention: the rotated width must be even and at most the rotated part's width")
        if pairing not in ("neighbours", "halves"):
            raise ValueError("latent attention: rotation pairs are neighbours or halves")
        self.hidden, self.heads, self.key_dim, self.rot_dim, self.value_dim = int(hidden), int(heads), int(key_dim), int(rot_dim), int(value_dim)
        self.q_rank, self.kv_rank, self.scale = int(q_rank or 0), int(kv_rank), float(scale)
        self.pairing, self.gate = pairing, bool(gate)
        self.rot_scaling = tuple(float(x) for x in rot_scaling) if rot_scaling is not None else None
        self.rot_magnitude = 1.0
        self.rot_base, self.rot_dims, self.norm_eps = float(rot_base), int(rot_dims), float(norm_eps)
        self.window = int(window) if window else None
        self.q_width = self.heads * (self.key_dim + self.rot_dim)
        self.v_width = self.heads * self.value_dim
        self.freq: Optional[torch.Tensor] = None
        self.plain_cores = False      # True: the tiled scores stay on the CUDA cores also where the tensor-core form would run

    def stored_products(self):
        """The products whose result is stored (not added to the residual): a block may clear their outputs in passing."""
        return (self.down, self.uq) if self.q_rank else (self.down,)

    def output_product(self) -> Linear:
        return self.o

    def cache_spec(self):
        return KVSpec(1, self.kv_rank + self.rot_dim, self.window, planes=1)

    def tensor_specs(self) -> Dict[str, TensorSpec]:
        E, C, R = self.hidden, self.kv_rank, self.rot_dim
        specs = {"dkv": TensorSpec((C + R, E)), "dkv.norm": TensorSpec((C,), "vector", init="one_plus_normal", std=0.01),
                 "uk": TensorSpec((self.heads * self.key_dim, C)), "uv": TensorSpec((self.v_width, C)),
                 "o": TensorSpec((E, self.v_width))}
        if self.q_rank:
            specs.update({"dq": TensorSpec((self.q_rank, E)), "dq.norm": TensorSpec((self.q_rank,), "vector", init="one_plus_normal", std=0.01),
                          "uq": TensorSpec((self.q_width, self.q_rank))})
        else:
            specs["q"] = TensorSpec((self.q_width, E))
        if self.gate:
            specs["g"] = TensorSpec((self.v_width, E))
        return specs

    def frequencies(self):
        """(float32 frequencies [rot_dims / 2] rounded once from double, the factor on cosines and sines)."""
        if self.rot_scaling is not None and self.rot_dims:
            f, magnitude = blended_frequencies(self.rot_base, self.rot_dims, *self.rot_scaling)
        else:
            f, magnitude = power_frequencies(self.rot_base, self.rot_dims), 1.0
        return f.astype(np.float32), float(magnitude)

    def load(self, tensors, precision: Precision) -> None:
        super().load(tensors, precision)
        self.cleared_outputs = {}
        t = tensors
        # One product for everything that reads h: [query latent | key/value latent | rotated part], or without a query
        # latent [key/value latent | rotated part | queries], then the gate's input.
        stacked = [t["dq"], t["dkv"]] if self.q_rank else [t["dkv"], t["q"]]
        if self.gate:
            stacked.append(t["g"])
        self.down = Linear(torch.cat(stacked, dim=0), precision)
        self.o = Linear(t["o"], precision)
        self.uq = Linear(t["uq"], precision) if self.q_rank else None
        self.dq_norm = t["dq.norm"].to(torch.float32).contiguous() if self.q_rank else None
        self.dkv_norm = t["dkv.norm"].to(torch.float32).contiguous()
        self.w_uk = t["uk"].to(precision.act).contiguous()
        self.w_uv = t["uv"].to(precision.act).contiguous()
        # Frequencies in double precision, rounded once; the angle is the float product with the position.
        freq, self.rot_magnitude = self.frequencies()
        self.freq = torch.from_numpy(freq).to(self.w_uk.device)
        self._sms = torch.cuda.get_device_properties(self.w_uk.device).multi_processor_count if self.w_uk.is_cuda else 148

    # -- how the tiled kernels cut a step (the same on the host when the plan is made and when the step runs) -------
    def _tiling(self, counts, max_context: int):
        """(tiles [(first row, rows)], ranges a tile's keys are cut into so that the blocks fill the device twice)."""
        ht, rt = ops.latent_tile_shape(self.heads)
        tiles, start = [], 0
        for n in counts:
            tiles += [(start + i, min(rt, n - i)) for i in range(0, n, rt)]
            start += n
        keys = max(int(max_context), 1) if self.window is None else min(max(int(max_context), 1), self.window + rt - 1)
        blocks = len(tiles) * -(-self.heads // ht)
        splits = max(1, min(-(-2 * self._sms // blocks), keys // 128))
        return tiles, splits

    def _wide(self, counts, contexts):
        """The requests whose keys and values are made: (ints of the requests, ints of their tiles, largest share of the
        workspace, workspace tokens, heads a group), or None when there are none, their workspace would not fit or the general
        form is the faster one for them."""
        requests, tiles, start, tokens, rows, longest, work = [], [], 0, 0, 0, 0, 0
        for n, context in zip(counts, contexts):
            keys = context if self.window is None else min(context, self.window + n - 1)
            if n >= PROMPT_ROWS and n * PROMPT_KEYS_A_ROW >= keys:
                share = -(-(keys + 63) // 128) * 128             # the first key lies up to 63 tokens into its share
                requests.append((start, n, tokens, share))
                tiles += [(start + i, min(128, n - i), tokens, start) for i in reversed(range(0, n, 128))]
                tokens, rows, longest, work = tokens + share, rows + n, max(longest, keys), work + n * self.heads * keys
            start += n
        if not requests:
            return None
        room = max(PROMPT_BYTES, rows * self.heads * (2 * self.kv_rank + self.rot_dim + 2) * 4)
        group = min(self.heads, room // (tokens * ops.LATENT_EXPANDED * 2))
        if group < 1 or (longest > PROMPT_FEW_KEYS and work < _rows_needed(longest, -(-self.heads // group)) * longest):
            return None
        return requests, tiles, max(r[3] for r in requests), tokens, group

    def plan_step(self, shape: StepShape) -> Optional[PartPlan]:
        if getattr(self, "precision", None) is None or self.precision.invariant:
            return None
        counts = shape.counts
        contexts = [shape.room] * len(counts) if shape.room > 0 else [h + c for h, c in zip(shape.histories, counts)]
        ints = []

        def run(first, some):
            tiles, splits = self._tiling(some, max(contexts))
            at = len(ints)
            ints.extend(x for t in tiles for x in t)
            return first, sum(some), at, len(tiles), splits

        whole, runs, wide = run(0, counts), [], None
        if self.key_dim == 128 and self.value_dim == 128 and self.w_uk.dtype is torch.bfloat16:
            wide = self._wide(counts, contexts)
        if wide is not None:
            requests, tiles, share, tokens, group = wide
            made = {r[0] for r in requests}
            first = at = 0
            small = []
            for n in counts:
                if at not in made:
                    small.append(n)
                else:
                    if small:
                        runs.append(run(first, small))
                    first, small = at + n, []
                at += n
            if small:
                runs.append(run(first, small))
            wide = (len(ints), len(requests), share, len(ints) + 4 * len(requests), len(tiles), tokens, group)
            ints += [x for r in requests + tiles for x in r]
        return _TilePlan(whole, runs, wide, ints)

    def forward(self, h: torch.Tensor, step: StepBatch, cache_entry: int, residual: torch.Tensor,
                write_cache: bool = True) -> None:
        rows = h.shape[0]
        if not (h.is_cuda and h.is_contiguous() and h.dtype is self.precision.act and tuple(h.shape) == (rows, self.hidden)
                and residual.dtype is torch.float32 and residual.is_contiguous() and tuple(residual.shape) == (rows, self.hidden)):
            raise runtime.KernelError("latent attention: rows of the path's type and the mixer's width, a float32 residual")
        group, cache = step.kv(cache_entry)
        slots = group.slots if write_cache else torch.full((rows,), -1, dtype=torch.int32, device=h.device)
        halves, mag = self.pairing == "halves", self.rot_magnitude
        proj = stored_product(self, self.down, h)
        latents = self.q_rank + self.kv_rank + self.rot_dim
        if self.q_rank:
            cq = torch.empty((rows, self.q_rank), dtype=self.precision.act, device=h.device)
            ops.latent_write(proj[:, :latents], self.q_rank, self.dq_norm, cq, self.dkv_norm, self.norm_eps, self.freq, step.positions,
                             slots, cache, self.kv_rank, self.rot_dim, halves=halves, magnitude=mag)
            q = stored_product(self, self.uq, cq)
            gate_at = latents
        else:
            ops.latent_write(proj[:, :latents], 0, None, None, self.dkv_norm, self.norm_eps, self.freq, step.positions,
                             slots, cache, self.kv_rank, self.rot_dim, halves=halves, magnitude=mag)
            q = proj[:, latents:latents + self.q_width]
            gate_at = latents + self.q_width
        o = torch.empty((rows, self.v_width), dtype=self.precision.act, device=h.device)
        # The tiled kernels hold a cache row in a warp's registers: rows of up to 768 values.
        ints = None if self.precision.invariant or self.kv_rank + self.rot_dim > 768 else step.plan_ints(self)
        if ints is not None:
            plan = step.plan.plan_of(self)
            sizes = (self.heads, self.key_dim, self.rot_dim, self.value_dim, self.kv_rank, group.page_size, self.window, self.scale)
            runs = [plan.whole]
            if plan.wide is not None and not self.plain_cores and ops.latent_prompt_fits(
                    self.key_dim, self.rot_dim, self.value_dim, self.kv_rank, group.page_size, self.w_uk.dtype, cache.dtype):
                at, n_requests, share, tiles_at, n_tiles, tokens, heads = plan.wide
                ops.latent_attention_prompt(q, cache, self.w_uk, self.w_uv, o, self.freq, step.row_request, step.positions,
                                            group.block_tables, ints[at:at + 4 * n_requests], n_requests, share,
                                            ints[tiles_at:tiles_at + 4 * n_tiles], n_tiles, tokens, heads, *sizes, halves=halves, magnitude=mag)
                runs = plan.runs
            # The tiled kernels: 16 (row, head) pairs share the keys they read; key ranges fill the device when rows are few.
            for first, n, at, n_tiles, splits in runs:
                rows_of = slice(first, first + n)
                ops.latent_attention_tiled(q[rows_of], cache, self.w_uk, self.w_uv, o[rows_of], self.freq, step.row_request[rows_of],
                                           step.positions[rows_of], group.block_tables, ints[at:at + 2 * n_tiles], n_tiles, splits,
                                           *sizes, plain_cores=self.plain_cores, halves=halves, magnitude=mag)
        else:
            # One block per (row, head): the schedule follows the sizes alone (an invariant path, or a step without a plan).
            ops.latent_attention(q, cache, self.w_uk, self.w_uv, o, self.freq, step.row_request, step.positions, group.block_tables,
                                 self.heads, self.key_dim, self.rot_dim, self.value_dim, self.kv_rank, group.page_size, self.window,
                                 self.scale, halves=halves, magnitude=mag)
        if self.gate:
            ops.sigmoid_gate_(o, proj[:, gate_at:gate_at + self.v_width])
        add_product(self, self.o, o, residual)
