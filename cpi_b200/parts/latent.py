"""Attention over a cached latent: what a position keeps is one low-rank vector and one rotated key part.

"latent_attention"   c_q = rmsnorm(W_dq h) * dq_norm;  q = W_uq c_q, head by head [dim plain | rot_dim rotated];
                     [c' | r] = W_dkv h;  c = rmsnorm(c') * dkv_norm (kv_rank elements), r rotated (rot_dim elements,
                     one for all heads);  head n: key [W_uk,n c | r], value W_uv,n c;
                     score = (q . key) * scale over all earlier positions and the token's own, softmax with an optional
                     learned sink per head (its exponential joins the denominator, without a key or a value);
                     out = W_o concat_heads(sum_j p_j value_j).
                     params: hidden_size, heads, head_dim (plain), rot_dim, value_dim, q_rank, kv_rank, softmax_scale,
                     norm_eps, position (PartSpec; a rotation of rot_dim elements, or "none"; its amplitude multiplies the
                     sines and cosines of both rotated parts), sink (bool), window (None, {"kind": "full"} or {"kind":
                     "sliding", "size": n}: a position sees itself and the n - 1 before it),
                     output_gate (bool; tensor "g" [heads * value_dim, hidden]: the concatenated heads are multiplied by
                     sigmoid(g h) element by element),
                     tensor_names {"dq", "dq_norm", "uq", "dkv", "dkv_norm", "uk", "uv", "o", "sink", "g"}.
                     cache: one stream "latent" of one head of kv_rank + rot_dim elements per position.  A layer that only
                     runs on another run entry's cache has no dkv and dkv_norm: it reads that entry's latents and rotated
                     key parts with its own queries, W_uk and W_uv (their kv_rank, rot_dim and rotation are the same).

How it runs.  Only [c | r] is cached.  Decode steps, float32, and prompts of few tokens behind many positions never form the
heads' keys and values: since q_n . (W_uk,n c) = (W_uk,n^T q_n) . c, the plain part of a query is first taken through
W_uk,n^T (a grouped product, one group per head, over rows laid out head by head), and attention then runs over the cached
rows themselves as ONE key/value head of kv_rank + rot_dim elements that all query heads share, with the library's
attention kernels.  Its output per head is a weighted sum of rows [c | r]; the first kv_rank elements go through W_uv,n (the
second grouped product) and the result through W_o.  Other bfloat16 prompts with heads of 128 + 64 elements and values of
128 form the keys and values of the rows that their queries see, for this step only, by one product, and attend over those
(`_forms_keys` has the rule, csrc/latent_prefill.cu the kernel); that takes a copy of W_uk and W_uv side by side (heads * 256 *
kv_rank elements) and scratch for the rows and for up to FORMED_BYTES of keys and values, and is left out where there is no room for
them.  Norms, the rotation, scores and softmax are float32 in both precisions.
"""
from __future__ import annotations

import torch

from ..cache.manager import KVRequirement
from ..csrc import lib as K
from ..phases import phase
from ..weights.store import TensorReq
from . import attention as _attention
from .attention import attend
from .base import Mixer, RotaryEncoding, build_part, register_mixer
from .linear import MODE_ADD, MODE_STORE, project


# set to False to run every prompt over the cached rows themselves (tests compare the two forms)
use_formed_keys = True
# Bytes of keys and values formed at a time; a step with more forms and attends a few heads after another.  The mixer's us with
# 64, 128 and 512 MB: 16 heads x 16,384 tokens 2,202, 2,157, 2,154; 64 x 4,096 934, 897, 897; 128 x 8,192 4,874, 4,777, 4,855.
FORMED_BYTES = 128 << 20


def use_tensor_core_kernels() -> bool:
    """The switch of the attention part: off, every attention runs through the general kernel."""
    return _attention.use_tensor_core_kernels


@register_mixer("latent_attention")
class LatentAttentionMixer(Mixer):
    graph_safe = True
    can_store = True

    def __init__(self, spec, prefix="", workspace=None, owns_cache=True):
        super().__init__(spec, prefix)
        p = spec.params
        self.has_kv = bool(owns_cache)                # False: every run entry of this layer reads another's cache
        self.hidden, self.nh = int(p["hidden_size"]), int(p["heads"])
        self.d, self.r, self.dv = int(p["head_dim"]), int(p["rot_dim"]), int(p["value_dim"])
        self.q_rank, self.kv_rank = int(p["q_rank"]), int(p["kv_rank"])
        self.scale, self.eps = float(p["softmax_scale"]), float(p["norm_eps"])
        self.has_sink = bool(p.get("sink", False))
        self.gate_rows = self.nh * self.dv if p.get("output_gate", False) else 0
        w = p.get("window") or {"kind": "full"}
        if w["kind"] not in ("full", "sliding"):
            raise ValueError(f"latent_attention: a window of kind '{w['kind']}' (full or sliding)")
        self.window_kind = w["kind"]
        self.window = int(w["size"]) if w["kind"] == "sliding" else 0
        if w["kind"] == "sliding" and self.window < 1:
            raise ValueError(f"latent_attention: a window of {self.window} positions")
        self.row = self.kv_rank + self.r              # what a position keeps, and the size of a query head
        if self.r % 2 or self.r < 0:
            raise ValueError(f"latent_attention: a rotated part of {self.r} elements (an even number)")
        if self.row > K.GENERAL_ATTENTION_MAX_DIM:
            raise ValueError(f"latent_attention: kv_rank + rot_dim = {self.row} exceeds the attention kernels' "
                             f"{K.GENERAL_ATTENTION_MAX_DIM}")
        self.position = build_part("position", p["position"])
        tn = {"dq": "mixer.q_a_proj.weight", "dq_norm": "mixer.q_a_norm.weight", "uq": "mixer.q_b_proj.weight",
              "dkv": "mixer.kv_a_proj.weight", "dkv_norm": "mixer.kv_a_norm.weight", "uk": "mixer.k_b_proj.weight",
              "uv": "mixer.v_b_proj.weight", "o": "mixer.o_proj.weight", "sink": "mixer.sinks",
              "g": "mixer.g_proj.weight"}
        tn.update(p.get("tensor_names") or {})
        self.tn = {k: prefix + v for k, v in tn.items()}
        self.ws = workspace
        self.w_down = self.w_uq = self.w_ukT = self.w_uv = self.w_o = None
        self.w_qnorm = self.w_cnorm = self.sink = self.rotary = self.w_kv = None

    def requirements(self):
        t, H = self.tn, self.hidden
        reqs = [TensorReq(t["dq"], (self.q_rank, H)), TensorReq(t["dq_norm"], (self.q_rank,), init="ones+normal"),
                TensorReq(t["uq"], (self.nh * (self.d + self.r), self.q_rank)),
                TensorReq(t["uk"], (self.nh * self.d, self.kv_rank)), TensorReq(t["uv"], (self.nh * self.dv, self.kv_rank)),
                TensorReq(t["o"], (H, self.nh * self.dv))]
        if self.has_kv:
            reqs += [TensorReq(t["dkv"], (self.row, H)), TensorReq(t["dkv_norm"], (self.kv_rank,), init="ones+normal")]
        if self.gate_rows:
            reqs.append(TensorReq(t["g"], (self.gate_rows, H)))
        if self.has_sink:
            reqs.append(TensorReq(t["sink"], (self.nh,)))
        return reqs

    def load(self, source, device):
        t = self.tn
        f32 = lambda name: source.get(t[name], device).to(torch.float32).contiguous()
        # one product for all that reads the layer's input: [gate | query latent | latent and rotated key part]
        parts = [source.get(t[n], device) for n, on in (("g", self.gate_rows), ("dq", True), ("dkv", self.has_kv)) if on]
        dt = torch.float32 if any(w.dtype == torch.float32 for w in parts) else torch.bfloat16
        self.w_down = torch.cat([w.to(dt) for w in parts], dim=0).contiguous()
        self.w_uq = source.get(t["uq"], device).contiguous()
        uk = source.get(t["uk"], device).view(self.nh, self.d, self.kv_rank)
        self.w_ukT = uk.transpose(1, 2).contiguous()                                   # [heads, kv_rank, dim]
        self.w_uv = source.get(t["uv"], device).view(self.nh, self.dv, self.kv_rank).contiguous()
        if uk.is_cuda and uk.dtype == self.w_uv.dtype == torch.bfloat16 \
                and K.latent_prefill_supported(self.d, self.r, self.dv, self.kv_rank, 64):
            # for prompts whose keys and values are formed: head after head its rows of W_uk, then of W_uv (without the
            # room for this copy prompts stay with the cached rows)
            try:
                self.w_kv = torch.cat([uk, self.w_uv], dim=1).view(self.nh * (self.d + self.dv), self.kv_rank)
            except torch.OutOfMemoryError:
                self.w_kv = None
        self.w_o = source.get(t["o"], device).contiguous()
        self.w_qnorm = f32("dq_norm")
        if self.has_kv:
            self.w_cnorm = f32("dkv_norm")
        if self.has_sink:
            self.sink = f32("sink")
        self.position.prepare(device)
        enc = self.position.encoding()
        if enc is not None and not isinstance(enc, RotaryEncoding):
            raise TypeError(f"latent_attention: the position part '{self.position.spec.kind}' describes itself as "
                            f"{type(enc).__name__}; this mixer takes a rotation or none")
        self.rotary = enc
        if enc is not None and enc.inv_freq.numel() != self.r // 2:
            raise ValueError(f"latent_attention: the rotation turns {2 * enc.inv_freq.numel()} elements, the rotated "
                             f"part has {self.r}")

    def kv_requirement(self):
        return KVRequirement(1, self.row, self.window_kind, self.window, streams=(("latent", 1, self.row),))

    def forward(self, h, residual, batch, cache, add=True):
        T, f32, dt = h.shape[0], torch.float32, h.dtype
        H, D, R, rank = self.nh, self.d, self.r, self.kv_rank
        pages, table, page_size = cache.stream("latent")
        inv_freq = None if self.rotary is None else self.rotary.inv_freq
        inter = self.rotary is not None and self.rotary.interleaved
        amp = 1.0 if self.rotary is None else self.rotary.amplitude
        down = self.ws.get("latent_down", (T, self.w_down.shape[0]), f32)
        gate, low = down[:, :self.gate_rows], down[:, self.gate_rows:]
        with phase("qkv"):
            project(h, self.w_down, down)
        cq = self.ws.get("latent_cq", (T, self.q_rank), dt)
        if self.has_kv and cache.owns:
            # the normed latent and the rotated key part of every token go into its page; the queries' latent is normed beside
            beside = pages.dtype == dt
            with phase("kv_store"):
                K.latent_kv_write(low[:, self.q_rank:], self.w_cnorm, self.eps, inv_freq, inter, pages, table, page_size,
                                  batch.token_seq, batch.token_pos, batch.seq_slot, rank=rank, rot=R, amplitude=amp,
                                  queries=(low[:, :self.q_rank], self.w_qnorm, cq) if beside else None)
        else:
            beside = False
        if not beside:
            with phase("rmsnorm"):
                K.rmsnorm(low[:, :self.q_rank], self.w_qnorm, self.eps, cq)
        q = self.ws.get("latent_q", (T, H * (D + R)), f32)
        with phase("qkv"):
            project(cq, self.w_uq, q)
        out = self.ws.get("latent_values", (T, H * self.dv), dt)
        if not (self._forms_keys(batch, dt, page_size) and self._attend_formed(q, out, pages, table, batch, inv_freq, inter, amp)):
            self._attend_latent(q, out, pages, table, page_size, batch, inv_freq, inter, amp)
        if self.gate_rows:
            with phase("head_post"):
                K.head_turn(out, out, batch.token_pos, n_heads=H, value_dim=self.dv, gate=gate)
        with phase("wo"):
            project(out, self.w_o, residual, MODE_ADD if add else MODE_STORE)

    # ---- keys and values formed for the step
    def _forms_keys(self, batch, dt, page_size) -> bool:
        """Whether a step forms the heads' keys and values: prompts in bfloat16 with heads of the kernel's sizes.

        Forming costs time with the rows of all sequences together (0.7 ns a row and head at a latent rank of 512);
        the other form takes a sequence's keys one tile after another in one block, 0.1 us a key, however few its queries
        are, and with many queries it does 3.4 times the arithmetic.  So forming loses only where few queries meet a key
        AND many sequences share the launch.  Measured with 16 heads (formed / not): one prompt of 2,048 tokens 180 / 723
        us, of 4,096 309 / 2,188; 2 tokens behind 2,000 positions 95 / 233; 8 prompts of 20 tokens 82 / 93; but 16 sequences
        of 2 tokens behind 1,000 positions 221 / 153, and the line lies between the last two."""
        if (self.w_kv is None or not use_formed_keys or not use_tensor_core_kernels() or dt != torch.bfloat16 or batch.is_decode
                or not batch.n_q_tiles or not K.latent_prefill_supported(self.d, self.r, self.dv, self.kv_rank, page_size)):
            return False
        rows = pairs = longest = 0
        for start, n in zip(batch.starts, batch.n_new):
            keys = start + n - K.latent_first_row(start, self.window)
            rows, longest = rows + keys, max(longest, keys)
            pairs += n * min(start + (n + 1) // 2, self.window or start + n)
        return pairs >= 32 * rows or rows * self.nh <= 128 * longest

    def _attend_formed(self, q, out, pages, table, batch, inv_freq, inter, amp) -> bool:
        """False, with nothing done, if there is no room for the rows, keys and values."""
        H, D, R, rank, bf16 = self.nh, self.d, self.r, self.kv_rank, torch.bfloat16
        n_rows = sum(start + n - K.latent_first_row(start, self.window) for start, n in zip(batch.starts, batch.n_new))
        per = D + self.dv
        group = max(1, min(H, FORMED_BYTES // (2 * n_rows * per)))
        rows, formed = self.ws.scratch(n_rows * self.row, bf16), self.ws.scratch(n_rows * group * per, bf16)
        if rows is None or formed is None:
            return False
        rows = rows.view(n_rows, self.row)
        heads = self.ws.get("latent_q_heads", (batch.n_tokens, H * (D + R)), bf16)
        with phase("kv_store"):
            K.latent_key_rows(pages, rows, table, batch, window=self.window)
            K.latent_q_rows(q, inv_freq, inter, heads, batch.token_pos, n_heads=H, dim=D, rot=R, amplitude=amp)
        for h0 in range(0, H, group):
            h1 = min(H, h0 + group)
            kv = formed[:n_rows * (h1 - h0) * per].view(n_rows, (h1 - h0) * per)
            with phase("qkv"):
                project(rows[:, :rank], self.w_kv[h0 * per:h1 * per], kv)
            with phase("latent_attention"):
                K.latent_prefill(heads, kv, rows, out, batch, heads=(h0, h1), out_heads=H, rank=rank, scale=self.scale,
                                 sink=self.sink, window=self.window)
        return True

    # ---- attention over the cached rows themselves
    def _attend_latent(self, q, out, pages, table, page_size, batch, inv_freq, inter, amp):
        T, dt = q.shape[0], out.dtype
        H, D, R, rank, row = self.nh, self.d, self.r, self.kv_rank, self.row
        plain = self.ws.get("latent_q_plain", (H * T, D), dt)               # head-major rows
        full = self.ws.get("latent_q_full", (T, H * row), dt)
        offsets = self.ws.get("latent_offsets", (H + 1,), torch.int32)
        rows = self.ws.get("latent_rows", (H * T,), torch.int32)
        with phase("kv_store"):
            K.latent_q_split(q, inv_freq, inter, plain, full, offsets, rows, batch.token_pos, n_heads=H, dim=D, rot=R,
                             rank=rank, amplitude=amp)
        with phase("qkv"):               # the plain part of every query through its head's W_uk^T, into full[t, head, :rank]
            project(plain, self.w_ukT, full.view(T * H, row)[:, :rank], MODE_STORE, out_rows=rows, group_offsets=offsets,
                    n_groups=H, rows_per_group_hint=T, even_groups=H)
        lat = self.ws.get("latent_att_heads", (H * T, rank), dt)            # head-major, the latent part only
        if use_tensor_core_kernels() and dt == torch.bfloat16 and K.latent_attention_supported(row, rank):
            with phase("latent_attention"):
                if batch.is_decode:
                    # key splits from a bucketed bound of the context, so that a captured graph keeps its shape
                    groups = -(-H // 64)
                    keys = batch.ctx_bucket if not self.window else min(batch.ctx_bucket, self.window + K.LATENT_KEY_TILE)
                    tiles = -(-keys // K.LATENT_KEY_TILE)
                    n_splits = max(1, min(K.sm_count() // max(1, T * groups), tiles // 2,
                                          K.latent_attention_max_splits()))
                    K.latent_attention(full, lat, pages, table, page_size, batch.token_seq, batch.token_pos,
                                       batch.seq_slot, n_heads=H, rank=rank, scale=self.scale, sink=self.sink,
                                       n_splits=n_splits, window=self.window)
                else:
                    K.latent_attention(full, lat, pages, table, page_size, batch.token_seq, batch.token_pos,
                                       batch.seq_slot, n_heads=H, rank=rank, scale=self.scale, sink=self.sink,
                                       tile_tok0=batch.tile_tok0, tile_rows=batch.tile_rows, window=self.window)
        else:
            att = self.ws.get("latent_att", (T, H * row), dt)
            with phase("latent_attention"):
                attend(full, att, pages, pages, table, page_size, batch, n_heads=H, n_kv_heads=1, head_dim=row,
                       value_dim=row, window_kind=self.window_kind, window_size=self.window, scale=self.scale, sink=self.sink)
            with phase("wo"):
                K.head_major_rows(att, lat, n_heads=H, n=rank)
        with phase("wo"):
            project(lat, self.w_uv, out.view(T * H, self.dv), MODE_STORE, out_rows=rows, group_offsets=offsets,
                    n_groups=H, rows_per_group_hint=T, even_groups=H)
