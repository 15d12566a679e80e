"""Attention over a compressed cache ("latent attention"), as a mixer part.

Per token the mixer keeps ONE vector of `kv_rank + rot_dim` numbers instead of keys and values for every head:
    q = W_q x                      per head [plain_dim plain | rot_dim rotated by position]
    W_dkv x                        kv_rank + rot_dim numbers: the first kv_rank, RMS-normed with a weight, are the
                                   latent c; the last rot_dim, rotated by position, are a key part all heads share
    head h:  key = [W_uk,h c | shared rotated part],  value = W_uv,h c
    score = scale * (q_plain . W_uk,h c + q_rot . k_rot),  causal softmax,  y = W_o (concat_h(sum_j p_j W_uv,h c_j) [* sigmoid(W_g x)])
Nothing but c and the rotated part is cached, and the per-head keys and values are never formed: because the score
is linear in c, the query is carried into the latent space instead (q_lat,h = W_uk,h^T q_plain,h, one small product
per head), the attention runs as H query heads over one shared key/value head whose key is the cache row
[c | k_rot] and whose value is the row's first kv_rank dims, and W_uv,h is applied to the attention's result
(sum_j p_j c_j).  A decode step therefore reads kv_rank + rot_dim numbers per cached token, whatever the number of
heads.  Sizes, the norm's eps, the position encoding (its pairing, scaling and magnitude), the scale, a window and
the output gate are parameters; `names` renames the tensors (keys q, dkv, dkv_norm, uk, uv, gate, o, dq, dq_norm, uq).
  `q_rank`: the queries come through a latent of their own, q = W_uq (rms(W_dq x) * weight), instead of W_q x;
  `gate="head"`: one gate number per head (tensor [n_heads, hidden]) instead of one per output of a head;
  `out_scale` is a factor on the mixer's result that the gate carries.

Prompt portions, when serving in bfloat16 with heads of 128 plain dims, 64 rotated ones (or none) and values of 128: a query
meets 128 + 64 numbers of a key and 128 of a value instead of kv_rank + rot_dim and kv_rank of a cache row, a third of the
arithmetic, where enough queries share the making of keys and values.  A request that brings `MADE_FROM` tokens or more to a
step has them made from the cache rows it sees (one product for all heads) and runs on the tcgen05 prompt kernel; the others
stay in the latent space.
"""
from __future__ import annotations

from dataclasses import dataclass
from types import SimpleNamespace
from typing import Dict, List, Optional, Tuple

import torch

from ..csrc import ops
from .base import KVCacheSpec, MATRIX, VECTOR, ParamSpec, Part, Precision, StepTables, register_part, stacked_rows
from .position import RotaryEmbedding


@dataclass
class LatentInfo:
    """The host-side facts of a step in which requests have their keys and values made: the latent kernel's plan for the others
    (or None), runs of neighbouring rows (first, one past the last, made or not), the made rows with what fills their tiles up, and
    the most that a request sees."""
    plan: object
    single_tokens: bool
    runs: List[Tuple[int, int, bool]]
    rows: int
    most_rows: int


class LatentAttention(Part):
    graph_safe = True   # reads the batch from device tensors only
    # Measured at 32 heads, prompt mixer alone, latent space against made: 2,048 tokens 1,213 us against 364; 128 tokens behind
    # 4,000 348 against 220, 64 behind 2,000 176 against 172 (level: 32 rows made for a query); 64 to 128 tokens level, bound by
    # the launches.  Rows made are bounded to 16 a query.
    MADE_FROM = 64
    MADE_ROWS = 16
    # What is made for a step takes at most so many bytes (16 KB a row at 32 heads), or where that is more what the latent space takes
    # for the same queries (76 KB each at 32 heads and a rank of 512).  The requests with the most rows a query go first.
    MADE_SCRATCH = 1 << 30
    MADE_BESIDE = 256   # beside requests that stay in the latent space: so many tokens at least, for the further launches
    MADE_RUNS = 4       # a step whose kinds of requests alternate more often stays in the latent space: every run is launched apart

    def __init__(self, hidden: int, n_heads: int, plain_dim: int, rot_dim: int, v_head_dim: int, kv_rank: int, prefix: str,
                 norm_eps: float, scale: float, position: Optional[RotaryEmbedding] = None, gate=False,
                 window: Optional[int] = None, names: Optional[Dict[str, str]] = None, q_rank: Optional[int] = None,
                 out_scale: float = 1.0):
        if min(n_heads, plain_dim, v_head_dim, kv_rank) < 1 or rot_dim < 0:
            raise ValueError("heads, plain_dim, v_head_dim and kv_rank must be positive, rot_dim not negative")
        if kv_rank + rot_dim > 640:
            raise ValueError(f"a cache row of {kv_rank + rot_dim} numbers is above 640")
        if position is not None and position.rotary_dim > rot_dim:
            raise ValueError("the rotary width exceeds rot_dim")
        self.hidden, self.H, self.dn, self.dr, self.vd, self.r = hidden, n_heads, plain_dim, rot_dim, v_head_dim, kv_rank
        self.prefix, self.norm_eps, self.scale = prefix, float(norm_eps), float(scale)
        self.position, self.gate, self.window = position, bool(gate), window
        self.gate_per_head = gate == "head"
        if q_rank is not None and q_rank < 1:
            raise ValueError("q_rank must be positive (or absent)")
        if out_scale != 1.0 and not gate:
            raise ValueError("out_scale rides on the output gate: it needs a gate")
        self.q_rank, self.out_scale = q_rank, float(out_scale)
        self.names = {"q": "q", "dkv": "dkv", "dkv_norm": "dkv.norm", "uk": "uk", "uv": "uv", "gate": "g", "o": "o",
                      "dq": "dq", "dq_norm": "dq.norm", "uq": "uq"}
        self.names.update(names or {})
        self.w_in = self.w_uq = self.w_uk_t = self.w_uv = self.w_o = self.c_norm = self.q_norm = None
        self._tables_key = None        # set at bind: the flash kernels' work items, when they take a row of this size
        self._sm_count = 0
        self._wide = False             # set at bind: the row is too wide for the flash kernels, the latent kernel takes it
        self._w_ukv = None             # set at bind, where prompt portions have keys and values made: per head [W_uk,h | W_uv,h]

    def _flash_takes(self) -> bool:
        """The flash kernels run H query heads over ONE key/value head whose keys and values are both the cache row
        (the last rot_dim dims of their result are not used), when the row has a head size they know."""
        from ..csrc import attention_fast
        return attention_fast.supported(self.r + self.dr, self.H)

    def _latent_kernel_takes(self) -> bool:
        """Wider rows: the kernel that keeps the query tile in shared memory and splits the value columns among warps."""
        from ..csrc import attention_fast
        return attention_fast.latent_supported(self.H, self.r + self.dr, self.r)

    def _made_takes(self) -> bool:
        """The tcgen05 prompt kernel takes keys and values of these sizes (and the gate's logits lie on 16-byte boundaries)."""
        from ..csrc import attention_fast
        first = self.q_rank if self.q_rank is not None else self.H * (self.dn + self.dr)
        return attention_fast.made_supported(self.dn, self.dr, self.vd, self.r) \
            and (not self.gate or self.gate_per_head or (first + self.r + self.dr) % 4 == 0)

    def kernel_libraries(self, bfloat16: bool):
        from ..csrc import attention_fast
        if not bfloat16:
            return ()
        if not self._flash_takes():
            made = ("attention_prefill_tc",) if self._made_takes() else ()
            return ("gemm_heads", "attention_latent") + made if self._latent_kernel_takes() else ("gemm_heads",)
        return ("gemm_heads", "attention_flash", "attention_prefill_tc") if attention_fast.tc_prefill_supported(self.r + self.dr, self.H) \
            else ("gemm_heads", "attention_flash")

    def step_tables_key(self):
        return self._tables_key

    def step_tables(self, ctx):
        from .attention import flash_step_tables
        if self._w_ukv is not None and not ctx.fixed_shape:
            tables = self._made_tables(ctx)
            if tables is not None:
                return tables
        if self._wide:
            # items of at most 64 / H tokens, all heads of a token in one item; never the tcgen05 prompt kernels' tiles
            return flash_step_tables(ctx, self.H, 1, self.r + self.dr, self.window or 0, 0, self._sm_count, tensor_prompt=False)
        return flash_step_tables(ctx, self.H, 1, self.r + self.dr, self.window or 0, 0, self._sm_count)

    def _made_tables(self, ctx) -> Optional[StepTables]:
        from ..csrc import attention_fast
        from .attention import flash_step_tables
        window = self.window or 0
        seen = [int(c) + (min(int(p), window - 1) if window else int(p)) for c, p in zip(ctx.q_lens, ctx.start_positions)]
        made = [int(c) >= self.MADE_FROM and v <= self.MADE_ROWS * int(c) for c, v in zip(ctx.q_lens, seen)]
        self._fit_scratch(made, [int(c) for c in ctx.q_lens], seen, attention_fast.MADE_TILE)
        runs: List[Tuple[int, int, bool]] = []
        for start, count, m in zip(ctx.q_starts, ctx.q_lens, made):
            if runs and runs[-1][2] == m:
                runs[-1] = (runs[-1][0], start + count, m)
            else:
                runs.append((start, start + count, m))
        if not any(made) or len(runs) > self.MADE_RUNS:
            return None
        if not all(made) and sum(int(c) for c, m in zip(ctx.q_lens, made) if m) < self.MADE_BESIDE:
            return None

        def those(kind):
            return [[x for x, m in zip(xs, made) if m == kind] for xs in (ctx.slots, ctx.q_starts, ctx.q_lens, ctx.start_positions)]

        items, segments, firsts, rows = attention_fast.made_items(*those(True), window, attention_fast.MADE_TILE)
        arrays, plan, single = {"made_items": items, "made_segments": segments, "made_firsts": firsts}, None, False
        if not all(made):
            slots, q_starts, q_lens, starts = those(False)
            rest = SimpleNamespace(slots=slots, q_starts=q_starts, q_lens=q_lens, start_positions=starts, n_tokens=ctx.n_tokens,
                                   fixed_shape=False, max_context=ctx.max_context, page_tokens=ctx.page_tokens)
            got = flash_step_tables(rest, self.H, 1, self.r + self.dr, window, 0, self._sm_count, tensor_prompt=False)
            if got is None:
                return None
            arrays.update(got.arrays)
            plan, single = got.info, all(int(c) == 1 for c in q_lens)
        return StepTables(arrays, LatentInfo(plan, single, runs, rows, int(segments[:, 2].max())))

    def _fit_scratch(self, made: List[bool], rows: List[int], seen: List[int], tile: int) -> None:
        """Takes requests back into the latent space until the arrays of the others fit (MADE_SCRATCH)."""
        def needed():       # packed queries, cache rows side by side, keys and values; two tiles a request may be filled up
            return sum(2 * (c * self.H * (self.dn + self.dr) + (v + 2 * tile) * (self.r + self.dr + self.H * (self.dn + self.vd)))
                       for c, v, m in zip(rows, seen, made) if m)

        def latent():       # plain and absorbed queries, latent sums
            return sum(2 * c * self.H * (self.dn + 2 * self.r + self.dr) for c, m in zip(rows, made) if m)
        order = sorted((i for i, m in enumerate(made) if m), key=lambda i: seen[i] / rows[i])
        while order and needed() > max(self.MADE_SCRATCH, latent()):
            made[order.pop()] = False

    def children(self):
        return (self.position,) if self.position is not None else ()

    def own_param_specs(self) -> Dict[str, ParamSpec]:
        p, nm, H, d = self.prefix, self.names, self.H, self.hidden
        specs = {
            p + nm["dkv"]: ParamSpec((self.r + self.dr, d), MATRIX),
            p + nm["dkv_norm"]: ParamSpec((self.r,), VECTOR, "one_plus_normal"),
            p + nm["uk"]: ParamSpec((H * self.dn, self.r), MATRIX),
            p + nm["uv"]: ParamSpec((H * self.vd, self.r), MATRIX),
            p + nm["o"]: ParamSpec((d, H * self.vd), MATRIX),
        }
        if self.q_rank is None:
            specs[p + nm["q"]] = ParamSpec((H * (self.dn + self.dr), d), MATRIX)
        else:
            specs[p + nm["dq"]] = ParamSpec((self.q_rank, d), MATRIX)
            specs[p + nm["dq_norm"]] = ParamSpec((self.q_rank,), VECTOR, "one_plus_normal")
            specs[p + nm["uq"]] = ParamSpec((H * (self.dn + self.dr), self.q_rank), MATRIX)
        if self.gate:
            specs[p + nm["gate"]] = ParamSpec((H if self.gate_per_head else H * self.vd, d), MATRIX)
        return specs

    def cache_spec(self):
        """One shared head whose row is [latent | rotated key part]; no value tensor."""
        return KVCacheSpec(1, self.r + self.dr, self.window, 0)

    def own_bind(self, tensors, precision: Precision) -> None:
        p, nm, H = self.prefix, self.names, self.H
        # one product: q (or its latent), compressed row, gate
        self.w_in = stacked_rows([tensors[p + nm["q" if self.q_rank is None else "dq"]], tensors[p + nm["dkv"]]]
                                 + ([tensors[p + nm["gate"]]] if self.gate else []), multiple=8 if self.q_rank is not None else 1)
        if self.q_rank is not None:
            self.w_uq, self.q_norm = tensors[p + nm["uq"]], tensors[p + nm["dq_norm"]]
        dt = precision.compute
        # q_lat,h = W_uk,h^T q_plain,h: as a product with weights [out = kv_rank, in = plain_dim] per head
        self.w_uk_t = tensors[p + nm["uk"]].to(dt).view(H, self.dn, self.r).transpose(1, 2).contiguous()
        self.w_uv = tensors[p + nm["uv"]].to(dt).view(H, self.vd, self.r).contiguous()
        self.w_o = tensors[p + nm["o"]]
        self.c_norm = tensors[p + nm["dkv_norm"]]
        if precision.compute == torch.bfloat16 and self._flash_takes():
            self._tables_key = ("paged_attention_items", self.window or 0, self.H, 1, self.r + self.dr, False, 0, False)
            self._sm_count = torch.cuda.get_device_properties(precision.device).multi_processor_count
        elif precision.compute == torch.bfloat16 and self._latent_kernel_takes():
            self._wide = True
            self._tables_key = ("latent_attention_items", self.window or 0, self.H, self.r + self.dr)
            self._sm_count = torch.cuda.get_device_properties(precision.device).multi_processor_count
            if self._made_takes() and (not self.gate or self.gate_per_head or self.w_in.shape[0] % 4 == 0):
                self._tables_key += (self.dn, self.dr, self.vd)
                self._w_ukv = torch.cat([tensors[p + nm["uk"]].to(dt).view(H, self.dn, self.r), self.w_uv], dim=1) \
                    .reshape(H * (self.dn + self.vd), self.r).contiguous()

    def _forward_made(self, q, proj, at: int, xb, ctx, cache, rotation, write_cache: bool, gate, att) -> None:
        """The attention of a step in which some requests (or all) have their keys and values made: rows of `att`."""
        from ..csrc import attention_fast
        arrays, info = ctx.tables[self._tables_key]
        n, dev, dt = xb.shape[0], xb.device, xb.dtype
        H, dn, dr, r, vd = self.H, self.dn, self.dr, self.r, self.vd
        packed = torch.empty((n, H * (dn + dr)), dtype=dt, device=dev)
        q_full = torch.empty((n, H * (r + dr)), dtype=dt, device=dev) if info.plan is not None else None
        plain = {}
        for a, b, made in info.runs:
            if not made:
                plain[a] = torch.empty((b - a, H * dn), dtype=dt, device=dev)
            ops.latent_prep(q[a:b], proj[a:b, at:at + r + dr], plain.get(a), None if made else q_full[a:b], self.c_norm, self.norm_eps,
                            *rotation, ctx.positions[a:b], ctx.slot_of_token[a:b], cache.block_table, cache.k_pages, H, dn, dr, r,
                            cache.page_tokens, write_kv=write_cache, q_packed=packed[a:b] if made else None)
        c = torch.empty((info.rows, r), dtype=dt, device=dev)
        rope = torch.empty((info.rows, dr), dtype=dt, device=dev) if dr else None
        ops.latent_rows(cache.k_pages, cache.block_table, arrays["made_segments"], info.most_rows, c, rope, attention_fast.MADE_TILE)
        kv = torch.empty((info.rows, H * (dn + vd)), dtype=dt, device=dev)
        ops.gemm_narrow(c, self._w_ukv, kv)
        attention_fast.run_made(packed, kv, rope, arrays["made_items"], att, H, self.window or 0, self.scale, c, self.w_uv,
                                arrays["made_firsts"], gate, self.gate_per_head, self.out_scale)
        if info.plan is None:
            return
        for a, b, made in info.runs:
            if not made:
                ops.gemm_heads(plain[a].view(b - a, H, dn), self.w_uk_t, q_full[a:b].view(b - a, H, r + dr)[:, :, :r], H)
        lat = torch.empty((n, H * r), dtype=dt, device=dev)
        plan = attention_fast.plan_on_device(info.plan, arrays["items"], arrays.get("merge"))
        if not attention_fast.run_latent(q_full, cache.k_pages, cache.block_table, lat, H, r + dr, r, cache.page_tokens, self.window or 0,
                                         self.scale, plan, single_tokens=info.single_tokens):
            raise ops.KernelError("latent attention: the kernel refuses a step that its plan was made for")
        for a, b, made in info.runs:
            if not made:
                ops.gemm_heads(lat[a:b].view(b - a, H, r), self.w_uv, att[a:b].view(b - a, H, vd), H, gate=gate[a:b] if gate is not None else None,
                               gate_scale=self.out_scale, gate_per_head=self.gate_per_head)

    def _attend(self, q_full: torch.Tensor, ctx, cache) -> torch.Tensor:
        """The attention over the cache rows: a view [n, H, kv_rank] of the heads' latent sums.  In bfloat16 a tensor-core
        kernel takes it where one knows the row's size; else (and in 32-bit) the generic kernel."""
        from .attention import flash_plan
        n, dev, dt = q_full.shape[0], q_full.device, q_full.dtype
        H, dr, r = self.H, self.dr, self.r
        plan = flash_plan(ctx, self._tables_key) if dt == torch.bfloat16 and ops.forced("attention") != "generic" else None
        if plan is not None and self._wide:
            from ..csrc import attention_fast
            lat = torch.empty((n, H * r), dtype=dt, device=dev)
            # which variant runs depends on the batch's shape alone (single tokens or not), as a captured step's launches must
            if attention_fast.run_latent(q_full, cache.k_pages, cache.block_table, lat, H, r + dr, r, cache.page_tokens,
                                         self.window or 0, self.scale, plan,
                                         single_tokens=all(int(c) == 1 for c in ctx.q_lens)):
                return lat.view(n, H, r)
        elif plan is not None:
            # the flash kernels, with the cache rows as keys AND values: the first r dims of a head's result are its latent sums
            wide = torch.empty((n, H * (r + dr)), dtype=dt, device=dev)
            ops.paged_attention(q_full, cache.k_pages, cache.k_pages, cache.block_table, ctx.positions, ctx.slot_of_token, wide,
                                H, 1, r + dr, cache.page_tokens, self.window or 0, self.scale, plan=plan)
            return wide.view(n, H, r + dr)[:, :, :r]
        lat = torch.empty((n, H * r), dtype=dt, device=dev)
        ops.paged_attention(q_full, cache.k_pages, None, cache.block_table, ctx.positions, ctx.slot_of_token, lat,
                            H, 1, r + dr, cache.page_tokens, self.window or 0, self.scale)
        return lat.view(n, H, r)

    def forward(self, xb: torch.Tensor, residual: torch.Tensor, ctx, cache, write_cache: bool = True,
                accumulate: bool = True) -> None:
        n, dev, dt = xb.shape[0], xb.device, xb.dtype
        H, dn, dr, r, vd = self.H, self.dn, self.dr, self.r, self.vd
        proj = torch.empty((n, self.w_in.shape[0]), dtype=torch.float32, device=dev)
        ops.gemm(xb, self.w_in, proj)
        if self.q_rank is None:
            at = H * (dn + dr)
            q = proj[:, :at]
        else:
            at = self.q_rank
            c_q = torch.empty((n, at), dtype=dt, device=dev)
            ops.rms_norm(proj[:, :at], self.q_norm, self.norm_eps, c_q)
            q = torch.empty((n, H * (dn + dr)), dtype=torch.float32, device=dev)
            ops.gemm(c_q, self.w_uq, q)
        cos = sin = None
        rot, pairing = 0, "half"
        if self.position is not None:
            cos, sin, rot = self.position.tables()
            pairing = self.position.pairing
        # the output gate's logits, which the last step of either way applies
        gate = proj[:, at + r + dr:at + r + dr + (H if self.gate_per_head else H * vd)] if self.gate else None
        att = torch.empty((n, H * vd), dtype=dt, device=dev)
        if self._w_ukv is not None and dt == torch.bfloat16 and ops.forced("attention") != "generic" \
                and isinstance(ctx.tables.get(self._tables_key, (None, None))[1], LatentInfo):
            self._forward_made(q, proj, at, xb, ctx, cache, (cos, sin, rot, pairing), write_cache, gate, att)
            ops.gemm(att, self.w_o, residual, accumulate=accumulate)
            return
        q_plain = torch.empty((n, H * dn), dtype=dt, device=dev)
        q_full = torch.empty((n, H * (r + dr)), dtype=dt, device=dev)
        ops.latent_prep(q, proj[:, at:at + r + dr], q_plain, q_full, self.c_norm, self.norm_eps, cos, sin, rot, pairing, ctx.positions,
                        ctx.slot_of_token, cache.block_table, cache.k_pages, H, dn, dr, r, cache.page_tokens,
                        write_kv=write_cache)
        ops.gemm_heads(q_plain.view(n, H, dn), self.w_uk_t, q_full.view(n, H, r + dr)[:, :, :r], H)
        lat = self._attend(q_full, ctx, cache)                  # [n, H, r]: sum_j p_j c_j per head
        # the values' up-projection per head, with the output gate in its epilogue
        ops.gemm_heads(lat, self.w_uv, att.view(n, H, vd), H, gate=gate, gate_scale=self.out_scale, gate_per_head=self.gate_per_head)
        ops.gemm(att, self.w_o, residual, accumulate=accumulate)


register_part("mixer", "latent_attention", LatentAttention)
