"""Weights, caches and the operator sequence of one Rozesun layer.

A layer norms the input and the output of its sublayers: x += n1b(attention(n1(x))), x += n2b(ff(n2(x))).  Attention goes
through latents: the queries' own, and one of keys and values, which (with a rotated key part shared by the heads) is all
that is cached.  Three forms of it:

* ``decode`` -- one token, f32 vectors, eight launches per layer: the products of the normed input (both latents, key part,
  gate), queries, key expansion moved onto the queries + rotation + cache row, attention over the latent rows, merge +
  value expansion + gate, output product, gate/up, down.  What lies between two sublayers rides on the next launch's
  input staging (``Stream``).
* ``prefill``, absorbed -- the same algebra for a portion of tokens (few tokens, or the exact f32 mode).
* ``prefill``, expanded -- keys and values of the cache rows in use are expanded first: more work per key, less per query
  and key, for portions of many tokens.
"""

from __future__ import annotations

import torch

from tilert_b200 import gqa_ops as ops
from tilert_b200.gqa_ops import BF16, F32, pad
from tilert_b200.kv_cache import LatentCache

from ..blocks import Pending, RowStream, Scratch, Stream, layer_norm, padded_rows, padded_vec
from .model_args import GATE_ALPHA, LayerArgs, MixerArgs, RozesunArgs


def _row_blocks(*parts: torch.Tensor) -> torch.Tensor:
    """The parts' rows below each other, each part filled with zero rows to a multiple of eight."""
    return torch.cat([torch.nn.functional.pad(p, (0, 0, 0, pad(p.shape[0]) - p.shape[0])) for p in parts])


def _head_rows(w: torch.Tensor, heads: int, m: int) -> torch.Tensor:
    """[heads * n, k] -> [heads, n filled with zero rows to a multiple of m, k]."""
    w = w.reshape(heads, -1, w.shape[-1])
    return torch.nn.functional.pad(w, (0, 0, 0, pad(w.shape[1], m) - w.shape[1]))


class LayerWeights:
    """One layer's tensors, read under their checkpoint names from ``sd`` (any key -> tensor mapping)."""

    def __init__(self, args: RozesunArgs, sd, li: int, device, expanded: bool):
        """``expanded``: the weights of the expanded form too."""
        a = args.layers[li]
        m, f, dev = a.mixer, a.mlp, torch.device(device)
        mix, mlp = f"l{li}.mix", f"l{li}.mlp"
        h, r = m.heads, m.kv_rank
        want = {"dq": (m.q_rank, args.dim), "dq.norm": (m.q_rank,), "uq": (h * (m.dim + m.rot_dim), m.q_rank), "dkv": (r + m.rot_dim, args.dim),
                "dkv.norm": (r,), "uk": (h * m.dim, r), "uv": (h * m.vdim, r), "g": (m.gate_rows, args.dim), "o": (args.dim, h * m.vdim)}
        if m.sink:
            want["sink"] = (h,)
        t = {n: sd[f"{mix}.{n}"].to(dev) for n in want}
        if f is not None:
            want |= {"gate": (f.ff, args.dim), "up": (f.ff, args.dim), "down": (args.dim, f.ff)}
            t |= {n: sd[f"{mlp}.{n}"].to(dev) for n in ("gate", "up", "down")}
        for n, shape in want.items():
            if tuple(t[n].shape) != shape:
                raise ValueError(f"layer {li}: {n} has shape {tuple(t[n].shape)}, the configuration says {shape}")

        # everything that reads the layer's normed input, one product: [query latent | latent | key part | gate]
        self.off_c = pad(m.q_rank)
        self.off_r = self.off_c + pad(r)
        self.off_g = self.off_r + pad(m.rot_dim)
        self.z = padded_rows(_row_blocks(t["dq"], t["dkv"][:r], t["dkv"][r:], t["g"]), dev)
        self.q_gain, self.c_gain = padded_vec(t["dq.norm"], dev), padded_vec(t["dkv.norm"], dev)
        # per head [unrotated, zero rows | rotated, zero rows]
        uq = t["uq"].view(h, m.dim + m.rot_dim, m.q_rank)
        self.uq = padded_rows(torch.cat([_head_rows(p.reshape(-1, m.q_rank), h, 8) for p in (uq[:, : m.dim], uq[:, m.dim:])], dim=1)
                              .flatten(0, 1), dev)
        self.uk_t = padded_rows(t["uk"].view(h, m.dim, r).transpose(1, 2), dev)            # [heads, rank, pad8(dim)]
        self.kv = None
        if expanded:  # keys of all heads, then values, in rows of 16
            self.kv = padded_rows(torch.cat([_head_rows(t[n], h, 16).flatten(0, 1) for n in ("uk", "uv")]), dev)
        if expanded and m.vdim % 16 == 0:
            self.uv = self.kv[h * pad(m.dim, 16):].view(h, m.vdim, -1)                    # [heads, vdim, pad8(rank)]
        else:
            self.uv = padded_rows(t["uv"].view(h, m.vdim, r), dev)
        self.sink = t["sink"].to(F32).contiguous() if m.sink else None
        self.o = padded_rows(t["o"], dev)
        self.norm1, self.norm1b = (layer_norm(sd, f"l{li}.{n}", dev) for n in ("norm1", "norm1b"))
        self.norm2 = self.norm2b = self.gate_up = self.down = None
        if f is not None:
            self.norm2, self.norm2b = (layer_norm(sd, f"l{li}.{n}", dev) for n in ("norm2", "norm2b"))
            self.gate_up = padded_rows(torch.stack([t["gate"], t["up"]]), dev)
            self.down = padded_rows(t["down"], dev)

    def weight_bytes(self) -> int:
        """Bytes of weights one decode step streams from HBM."""
        ts = [self.z, self.uq, self.uk_t, self.uv, self.o] + ([self.gate_up, self.down] if self.down is not None else [])
        return 2 * sum(t.numel() for t in ts)


def expansion_pays(m: MixerArgs, rows: int, visible: int, cached: int) -> bool:
    """Whether expanding the keys and values of ``cached`` rows costs a portion of ``rows`` tokens, that see ``visible``
    keys each, fewer products than working on the latents."""
    absorbed = rows * (visible * (2 * m.kv_rank + m.rot_dim) + m.kv_rank * (m.dim + m.vdim))
    expanded = rows * visible * (m.dim + m.rot_dim + m.vdim) + cached * m.kv_rank * (m.dim + m.vdim)
    return expanded < absorbed


class RozesunLayer:
    def __init__(self, args: RozesunArgs, li: int, weights: LayerWeights, rope: ops.Rotation, scratch: Scratch, portion: int, dtype,
                 device, passes: int):
        self.args, self.a, self.w, self.rope, self.sc = args, args.layers[li], weights, rope, scratch
        self.dtype, self.portion = dtype, portion
        m = self.a.mixer
        self.caches = [LatentCache(m.kv_rank, m.rot_dim, m.window, args.max_seq_len, portion, device, dtype) for _ in range(passes)]
        self.sms = ops.num_sms(device)
        self.z_len = weights.off_g + m.gate_rows
        self.ldh = pad(m.dim) + pad(m.rot_dim)
        self._native = None  # of a portion's call: made when the first prompt comes

    def _splits(self, tokens: int, keys: int) -> int:
        """Parts of the key range, of ``per`` tiles of 64 keys each: no more than fill the SMs, and no more than pay (a tile
        takes about as long as the merge of 24 parts)."""
        tiles = (keys + 63) // 64
        least = -(-tiles // max(1, self.sms // ops.latent_blocks(self.a.mixer, tokens, self.dtype)))
        return min((-(-tiles // per) for per in range(least, least + 4)), key=lambda n: 24 * -(-tiles // n) + n)

    # -- one token --
    def decode(self, st: Stream, nr: int, cur_pos: torch.Tensor, length: int) -> None:
        """Pass ``nr``; ``length``: an upper bound of the sequence's length including this token."""
        m, w, sc, eps, dim, cache = self.a.mixer, self.w, self.sc, self.args.eps, self.args.dim, self.caches[nr]
        z = sc.get("vec_z", pad(self.z_len))
        st.dense(w.z, z, self.z_len, dim, eps, gain2=w.norm1)
        q = sc.get("vec_q", m.heads * self.ldh)
        ops.vec_dense(z, w.uq, q, m.heads * self.ldh, m.q_rank, gain2=w.q_gain, eps=eps)
        lat = sc.get("vec_lat", m.heads, cache.rows.shape[1])
        ops.vec_absorb(q, w.uk_t, m, self.rope, z[w.off_c:], z[w.off_r:], w.c_gain, eps, cur_pos, cache, lat)
        n_splits = self._splits(1, cache.visible(length))
        part = sc.get("vec_part", m.heads * n_splits * (pad(m.kv_rank, 16) + 2))
        ops.latent_attn(lat, cache, 1, m, cur_pos, n_splits, part)
        att = sc.get("vec_att", pad(m.heads * m.vdim))
        ops.vec_value(part, w.uv, m, n_splits, w.sink, z[w.off_g:], m.gate_per_head, att)
        y = sc.get("vec_y", pad(dim))
        ops.vec_dense(att, w.o, y, dim, m.heads * m.vdim)
        st.pending = Pending(y, w.norm1b)
        f = self.a.mlp
        if f is None:
            return
        hidden = sc.get("vec_hidden", pad(f.ff))
        st.gated(w.gate_up, hidden, f.ff, dim, f.limit, GATE_ALPHA, eps, gain2=w.norm2)
        ops.vec_dense(hidden, w.down, y, dim, f.ff)
        st.pending = Pending(y, w.norm2b)

    # -- a portion of tokens --
    def prefill(self, st: RowStream, nr: int, cur_pos: torch.Tensor, pos: int) -> None:
        """Pass ``nr``; ``pos``: the position of the first row, as ``cur_pos`` holds it."""
        m, w, sc, t, n = self.a.mixer, self.w, self.sc, self.dtype, st.rows
        cache, hn = self.caches[nr], m.heads * n
        if self._native is None:
            self._native = self._structure()
        s, length = self._native, pos + n
        s.cache = cache.rows.data_ptr()
        s.work_rows = n
        s.z = sc.room("z", n * pad(self.z_len))
        s.q = sc.room("q", n * m.heads * self.ldh)
        s.qe = s.kv = s.qn = s.lat = s.part = s.c = s.o = None  # (of the form that is taken, below)
        cached, n_splits = min(length, cache.ring), 0
        if w.kv is not None and expansion_pays(m, n, min(length, cache.window or length), cached):
            s.qe = sc.room("qe", hn * (pad(m.dim, 16) + pad(m.rot_dim, 16)), t)
            s.kv = sc.room("kv", cached * w.kv.shape[0], t)
        else:
            cached, n_splits = 0, self._splits(n, cache.visible(length, n))
            s.qn = sc.room("qn", hn * pad(m.dim), t)
            s.lat = sc.room("lat", hn * cache.rows.shape[1])
            s.part = sc.room("part", hn * n_splits * (pad(m.kv_rank, 16) + 2))
            s.c = sc.room("c", hn * pad(m.kv_rank), t)
            s.o = sc.room("o", hn * pad(m.vdim))
        s.work_cached, s.work_splits = cached, n_splits
        p = st.pending
        ops.latent_layer(s, n, cached, n_splits, cur_pos, st.x, st.xh, None if p is None else p.y, None if p is None else p.norm, st.add)
        st.add = None
        st.pending = Pending(self._y(), w.norm1b if self.a.mlp is None else w.norm2b)

    def _y(self) -> torch.Tensor:
        return self.sc.get("y", self.portion, pad(self.args.dim))

    def _structure(self):
        m, f, w, sc, p, t = self.a.mixer, self.a.mlp, self.w, self.sc, self.portion, self.dtype
        fields = dict(dim=self.args.dim, f32=int(t is F32), eps=self.args.eps, portion=p, heads=m.heads, head_dim=m.dim, rot=m.rot_dim, vdim=m.vdim, q_rank=m.q_rank,
                      kv_rank=m.kv_rank, window=self.caches[0].window, ring=self.caches[0].ring, scale=m.scale, gate_rows=m.gate_rows,
                      rope=self.rope.table, positions=self.rope.table.shape[0], rope_dims=self.rope.table.shape[1], interleaved=int(self.rope.interleaved),
                      w_z=w.z, q_gain=w.q_gain, c_gain=w.c_gain, w_uq=w.uq, w_uk_t=w.uk_t, w_kv=w.kv, w_uv=w.uv, sink=w.sink, w_o=w.o,
                      cq=sc.get("cq", p, pad(m.q_rank), dtype=t), att=sc.get("att", p, pad(m.heads * m.vdim), dtype=t), y=self._y())
        if f is not None:
            fields |= dict(ff=f.ff, limit=f.limit, alpha=GATE_ALPHA, w_gate_up=w.gate_up, w_down=w.down, hid=sc.get("hid", p, pad(f.ff), dtype=t))
        for name in ("norm1", "norm1b", "norm2"):
            norm = getattr(w, name)
            if norm is not None:
                fields |= {f"{name}_gain": norm.gain, f"{name}_bias": norm.bias}
        return ops.structure(ops.LatentLayer, **fields)

    def weight_bytes(self) -> int:
        return self.w.weight_bytes() * len(self.caches)
