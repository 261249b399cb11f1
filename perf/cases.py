"""The work a program has this framework do, as cases that can be timed and checked.

A case names an operation ("op") and its sizes:
  vision   images through the vision tower: the patch embedding and the first blocks of InternViT-6B or InternViT-300M
  prefill  prompts of unequal length through the Qwen2-7B decoder (two of its layers, the real head): logits of the last rows, cache
  decode   one token per request through the same decoder over a filled cache
  latent   the attention of a latent-attention layer (Voduzen, Munevik, Sorupel): norm + rotation + cache append, absorbed queries,
           attention over the cached latents, value product with its gate
  window   the attention of a layer with a sliding window, a soft cap and a distance bias (Tifisun) or with chunks of positions,
           rotation, head gates and one more denominator term (Sorupel)
  scan     a recurrent layer between its projections: convolution, recurrence, gated norm - state space with one step size per head
           (Sorupel), gated delta rule with one decay per head or per key channel (Tifisun)
  serve    a whole Sorupel model behind the step scheduler: prompts in one step, then decoding steps; logits of every step

Portions of requests are written "rows@first position", one per request.
"""
from __future__ import annotations

import math

import torch

from omchat_b200 import lib, seqlib
from omchat_b200.config import InternVisionConfig, OmChatQwen2Config, RotarySpec, SorupelConfig
from omchat_b200.model import sorupel
from omchat_b200.model.decoder import Qwen2Decoder
from omchat_b200.model.paged_cache import PagedLatentCache
from omchat_b200.model.seq_latent import LatentAttention
from omchat_b200.model.seq_linear import dense_linear
from omchat_b200.model.vision import build_vision_tower
from omchat_b200.model.weights import random_init
from omchat_b200.serving import StepScheduler

DEV = "cuda"
F64, F32, BF16, I32 = torch.float64, torch.float32, torch.bfloat16, torch.int32
DTYPES = {"bf16": BF16, "f32": F32}
QWEN_LAYERS = 2
EPS = 1e-6


# ------------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one picture of a chat request: the latency of the tower at batch 1
        {"name": "vision_one_crop", "op": "vision", "tower": "6b", "crops": 1, "blocks": 2},
        # the tiles of a few high-resolution pictures (7 crops each), the tower's throughput
        {"name": "vision_21_crops", "op": "vision", "tower": "6b", "crops": 21, "blocks": 1},
        # prompts with an image (1024 patch tokens and text) beside short ones, packed into one prefill
        {"name": "prefill_ragged", "op": "prefill", "lens": "1088,61,1301,517"},
        # the decode step of a single chat
        {"name": "decode_one", "op": "decode", "ctx": "1210"},
        # the decode step of a full batch at serving time, contexts of every age
        {"name": "decode_batch", "op": "decode", "ctx": ",".join(str(1024 + (i * 37) % 257) for i in range(32))},
        # prompt portions of a serving step, one of them a later portion of a long prompt
        {"name": "latent_prompts", "op": "latent", "dtype": "bf16", "heads": 16, "rank": 512, "rot": 64, "head": 128, "window": 0, "sink": True,
         "gate": True, "portions": "1024@0,777@0,1024@1024,301@0"},
        # a decode step of a batch: latency over contexts of unequal length
        {"name": "latent_decode", "op": "latent", "dtype": "bf16", "heads": 16, "rank": 512, "rot": 64, "head": 128, "window": 0, "sink": True,
         "gate": True, "portions": ",".join("1@%d" % (700 + (i * 173) % 1400) for i in range(32))},
        # sliding-window attention of prompts
        {"name": "window_prompts", "op": "window", "dtype": "bf16", "kind": "window", "heads": 32, "kv_heads": 8, "head": 128, "window": 512,
         "portions": "1024@0,777@0,1024@1024,301@0"},
        # chunked attention of a decode step
        {"name": "chunk_decode", "op": "window", "dtype": "bf16", "kind": "chunk", "heads": 16, "kv_heads": 4, "head": 128, "window": 512,
         "portions": ",".join("1@%d" % (700 + (i * 173) % 1400) for i in range(32))},
        # the state-space layer over prompts
        {"name": "scan_steps", "op": "scan", "dtype": "bf16", "kind": "steps", "heads": 64, "groups": 8, "dim": 128, "vdim": 64,
         "portions": "1024@0,777@0,1024@0,301@0"},
        # the delta rule over prompts
        {"name": "scan_delta", "op": "scan", "dtype": "bf16", "kind": "delta", "heads": 16, "groups": 8, "dim": 128, "vdim": 128,
         "portions": "1024@0,777@0,1024@0,301@0"},
        # a small model in full precision, as a trace is replayed for checking: short prompts, then decoding steps
        {"name": "serve_f32", "op": "serve", "dtype": "f32", "width": 1024, "heads": 8, "vocab": 8192, "lens": "37,211,128", "steps": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["vision", "prefill", "decode", "latent", "latent", "window", "window", "scan", "scan", "serve"])
    if op == "vision":
        tower = rng.choice(["6b", "300m"])
        return {"op": op, "tower": tower, "crops": _log(rng, 1, 20), "blocks": rng.choice([1, 2]) if tower == "300m" else 1}
    if op == "prefill":
        return {"op": op, "lens": ",".join(str(_log(rng, 16, 1400)) for _ in range(rng.choice([1, 2, 3, 5])))}
    if op == "decode":
        b = _log(rng, 1, 48)
        return {"op": op, "ctx": ",".join(str(_log(rng, 64, 2000)) for _ in range(b))}
    dtype = rng.choice(["bf16", "bf16", "bf16", "f32"])
    if op == "serve":
        width = rng.choice([512, 1024])
        return {"op": op, "dtype": dtype, "width": width, "heads": width // 128, "vocab": 4096,
                "lens": ",".join(str(_log(rng, 5, 300)) for _ in range(rng.choice([1, 2, 4]))), "steps": rng.randint(1, 6)}
    fresh = op == "scan"   # a recurrence that continues would start the next pass from other states
    long = dtype == "bf16" or fresh
    if rng.random() < 0.4 and not fresh:
        portions = ",".join("1@%d" % _log(rng, 30, 3000 if long else 600) for _ in range(_log(rng, 1, 48 if long else 8)))
    else:
        top = 1100 if long else 150
        portions = ",".join("%d@%d" % (_log(rng, 2, top), 0 if fresh or rng.random() < 0.6 else _log(rng, 16, top)) for _ in range(rng.choice([1, 2, 4])))
    if op == "latent":
        return {"op": op, "dtype": dtype, "heads": rng.choice([8, 16, 32]), "rank": rng.choice([256, 512]), "rot": rng.choice([32, 64]), "head": 128,
                "window": rng.choice([0, 0, 1024, 256]), "sink": rng.random() < 0.5, "gate": rng.random() < 0.5, "portions": portions}
    if op == "window":
        g = rng.choice([2, 4, 8])
        return {"op": op, "dtype": dtype, "kind": rng.choice(["window", "chunk"]), "heads": g * rng.choice([1, 2, 4]), "kv_heads": g,
                "head": rng.choice([64, 128]), "window": rng.choice([128, 512, 1024]), "portions": portions}
    kind = rng.choice(["steps", "delta", "channel"])
    if kind == "steps":
        g = rng.choice([1, 4, 8])
        return {"op": op, "dtype": dtype, "kind": kind, "heads": 8 * rng.choice([2, 4, 8]), "groups": g, "dim": rng.choice([64, 128]), "vdim": 64,
                "portions": portions}
    h = rng.choice([4, 8, 16])
    return {"op": op, "dtype": dtype, "kind": kind, "heads": h, "groups": h // 2 if kind == "delta" else h, "dim": rng.choice([64, 128]),
            "vdim": rng.choice([64, 128]), "portions": portions}


# -------------------------------------------------------------------------------------------------------------- small helpers
class State:
    pass


def _numbers(text):
    return [int(t) for t in text.split(",")]


def _portions(case):
    """[(first row, rows, slot, first position)], one entry per request."""
    out, row = [], 0
    for slot, part in enumerate(case["portions"].split(",")):
        n, first = (int(t) for t in part.split("@"))
        out.append((row, n, slot, first))
        row += n
    return out


def _rows(portions):
    return sum(p[1] for p in portions)


def _decoding(portions):
    return all(p[1] == 1 for p in portions)


def _addresses(portions):
    pos = torch.cat([torch.arange(p0, p0 + n) for _, n, _, p0 in portions]).to(I32).to(DEV)
    slot = torch.cat([torch.full((n,), s) for _, n, s, _ in portions]).to(I32).to(DEV)
    return pos, slot


def _seeded(seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))

    def rn(*shape, std=1.0, mean=0.0, dtype=F32):
        return (torch.randn(*shape, generator=gen, device=DEV) * std + mean).to(dtype)
    return rn


def _paged(widths, portions, dtype, seed, page=64):
    """A cache with pages in no order, as a server's free list leaves them."""
    need = [-(-(p0 + n) // page) for _, n, _, p0 in portions]
    cache = PagedLatentCache(widths, sum(need) + 1, len(portions), page, dtype, DEV, max_pages_per_slot=max(need))
    order = (torch.randperm(sum(need), generator=torch.Generator().manual_seed(int(seed))) + 1).tolist()
    for (_, n, s, p0), k in zip(portions, need):
        cache.set_pages(s, 0, order[:k])
        cache.host_lens[s] = p0 + n
        order = order[k:]
    cache.sync()
    return cache


def _places(cache, slot, n):
    """Indices of a slot's first n rows in the flattened pool."""
    j = torch.arange(n)
    return (cache.table_host[slot][j // cache.page_size].long() * cache.page_size + j % cache.page_size).to(DEV)


# --------------------------------------------------------------------------------------------------------------------- vision
def _vision_config(case):
    vc = (InternVisionConfig(num_hidden_layers=case["blocks"]) if case["tower"] == "6b"
          else InternVisionConfig.intern_vit_300m(num_hidden_layers=case["blocks"]))
    return OmChatQwen2Config(vision_config=vc, mm_hidden_size=vc.hidden_size, num_hidden_layers=0, hidden_size=128, vocab_size=8,
                             mm_vision_tower="InternViT-6B-448px-V1-5" if case["tower"] == "6b" else "InternViT-300M-448px")


def _prepare_vision(case, seed):
    s = State()
    s.cfg = _vision_config(case)
    s.tower = build_vision_tower(s.cfg, random_init(s.cfg, DEV, seed, vision=True, text=False).vit)
    s.pixels = _seeded(seed + 1)(case["crops"], 3, 448, 448)
    return s


def _run_vision(s):
    return s.tower(s.pixels)


def _rms64(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.to(F64)


def _exact_vision(case, s):
    vc, w = s.cfg.vision_config, s.tower.w
    n, C, H = case["crops"], vc.hidden_size, vc.num_attention_heads
    patches = torch.nn.functional.unfold(s.pixels.to(F64), 14, stride=14).transpose(1, 2)      # [n, 1024, 588]
    x = patches @ w.patch_w[:, :588].to(F64).T + w.patch_b.to(F64)
    x = torch.cat([w.cls.to(F64).expand(n, 1, C), x], 1) + w.pos.to(F64)

    def norm(x, wt, b):
        return _rms64(x, wt, vc.layer_norm_eps) if b is None else torch.nn.functional.layer_norm(x, (C,), wt.to(F64), b.to(F64), vc.layer_norm_eps)

    for l in w.layers:
        qkv = norm(x, l.norm1, l.norm1_b) @ l.qkv.to(F64).T
        if l.qkv_b is not None:
            qkv = qkv + l.qkv_b.to(F64)
        q, k, v = qkv.split(C, -1)
        if vc.qk_normalization:
            q, k = _rms64(q, l.q_norm, vc.layer_norm_eps), _rms64(k, l.k_norm, vc.layer_norm_eps)
        out = torch.empty_like(q)
        for i in range(n):
            qi, ki, vi = (t[i].view(-1, H, C // H).transpose(0, 1) for t in (q, k, v))
            a = torch.softmax(qi @ ki.transpose(1, 2) * (C // H) ** -0.5, -1) @ vi
            out[i] = a.transpose(0, 1).reshape(-1, C)
        x = x + (out @ l.proj_w.to(F64).T + l.proj_b.to(F64)) * l.ls1.to(F64)
        h = torch.nn.functional.gelu(norm(x, l.norm2, l.norm2_b) @ l.fc1_w.to(F64).T + l.fc1_b.to(F64))
        x = x + (h @ l.fc2_w.to(F64).T + l.fc2_b.to(F64)) * l.ls2.to(F64)
    return x[:, 1:]


def _work_vision(case):
    vc = _vision_config(case).vision_config
    C, I, n, S = vc.hidden_size, vc.intermediate_size, case["crops"], vc.num_patches + 1
    weights = case["blocks"] * (4 * C * C + 2 * C * I)
    return {"bytes": 2 * weights + 2 * 588 * C + n * 3 * 448 * 448 * 4 + n * (S - 1) * C * 2,
            "flops": 2 * n * S * weights + case["blocks"] * 4 * n * S * S * C + 2 * n * (S - 1) * 588 * C}


# ------------------------------------------------------------------------------------------------------------- Qwen2 decoder
def _qwen(seed):
    cfg = OmChatQwen2Config(num_hidden_layers=QWEN_LAYERS)
    return cfg, Qwen2Decoder(cfg, random_init(cfg, DEV, seed, vision=False).llm)


def _shuffled_pages(cache, seed):
    ids = torch.randperm(cache.block_table.numel(), generator=torch.Generator().manual_seed(int(seed)))
    cache.block_table.copy_(ids.to(I32).view_as(cache.block_table))


def _prepare_prefill(case, seed):
    s = State()
    s.cfg, s.dec = _qwen(seed)
    s.lens = _numbers(case["lens"])
    s.offsets = [sum(s.lens[:i]) for i in range(len(s.lens) + 1)]
    s.pos = torch.cat([torch.arange(n) for n in s.lens]).to(I32).to(DEV)
    s.seq = torch.cat([torch.full((n,), i) for i, n in enumerate(s.lens)]).to(I32).to(DEV)
    s.ids = torch.randint(0, s.cfg.vocab_size, (s.offsets[-1],), generator=torch.Generator().manual_seed(int(seed))).to(DEV)
    s.cache = s.dec.new_cache(len(s.lens), max(s.lens) + 64)
    _shuffled_pages(s.cache, seed)
    return s


def _run_prefill(s):
    embeds = lib.embed_lookup(s.ids, s.dec.w.embed)
    logits = s.dec.prefill(embeds, s.pos, s.seq, s.offsets, s.cache, logits="last")
    return {"logits": logits, "kv": s.cache.pool}


def _prepare_decode(case, seed):
    s = State()
    s.cfg, s.dec = _qwen(seed)
    s.ctx = _numbers(case["ctx"])
    rn = _seeded(seed + 1)
    s.tokens = torch.randint(0, s.cfg.vocab_size, (len(s.ctx),), generator=torch.Generator().manual_seed(int(seed))).to(DEV)
    s.cache = s.dec.new_cache(len(s.ctx), max(s.ctx) + 64)
    _shuffled_pages(s.cache, seed)
    for layer in s.cache.pool:
        layer.copy_(rn(*layer.shape, dtype=BF16))
    s.lens = torch.tensor(s.ctx, dtype=I32, device=DEV)
    if s.dec.use_stream(len(s.ctx)):
        s.dec.packed_weights()   # laid out once, when a server starts
    return s


def _run_decode(s):
    s.cache.ctx_lens.copy_(s.lens)          # the step is taken from the same contexts every time
    s.cache.host_lens = list(s.ctx)
    return {"logits": s.dec.decode_step(s.tokens, s.cache), "kv": s.cache.pool}


def _rope64(x, pos, theta):
    """x [T, heads, 128]: dimensions i and i + 64 turn by pos * theta^(-i / 64)."""
    f = theta ** (-torch.arange(64, dtype=F64, device=DEV) / 64)
    a = pos.to(F64)[:, None, None] * f
    u, v = x[..., :64], x[..., 64:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _qwen64(s, ids, pos, rows_of, kv):
    """Layers of the decoder in 64 bits over packed rows. rows_of: [(slice of rows, sequence, first position)]; kv: the cache's pool in
    64 bits, read for the positions in front of a sequence's first row and written for its rows. Returns the stream."""
    c, w = s.cfg, s.dec.w
    Hq, Hkv, page = c.num_attention_heads, c.num_key_value_heads, c.kv_page_size
    table = s.cache.block_table.long()
    x = w.embed.to(F64)[ids]
    for li, l in enumerate(w.layers):
        qkv = _rms64(x, l.ln1, c.rms_norm_eps) @ l.qkv_w.to(F64).T + l.qkv_b.to(F64)
        q, k, v = (t.view(len(ids), -1, 128) for t in qkv.split([Hq * 128, Hkv * 128, Hkv * 128], -1))
        q, k = _rope64(q, pos, c.rope_theta), _rope64(k, pos, c.rope_theta)
        out = torch.empty(len(ids), Hq * 128, dtype=F64, device=DEV)
        for rows, i, first in rows_of:
            n = rows.stop - rows.start
            j = torch.arange(first + n, device=DEV)
            pages, place = table[i][j // page], j % page
            kv[li][pages[first:], 0, :, place[first:]] = k[rows]
            kv[li][pages[first:], 1, :, place[first:]] = v[rows]
            keys, values = (kv[li][pages, m, :, place].transpose(0, 1) for m in (0, 1))      # [Hkv, keys, 128]
            qi = q[rows].view(n, Hkv, Hq // Hkv, 128).permute(1, 2, 0, 3)
            sc = qi @ keys[:, None].transpose(2, 3) * 128 ** -0.5
            sc.masked_fill_(j[None, :] > (first + torch.arange(n, device=DEV))[:, None], -math.inf)
            out[rows] = (torch.softmax(sc, -1) @ values[:, None]).permute(2, 0, 1, 3).reshape(n, -1)
        x = x + out @ l.o_w.to(F64).T
        gu = _rms64(x, l.ln2, c.rms_norm_eps) @ l.gate_up_w.to(F64).T
        x = x + (torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ l.down_w.to(F64).T
    return x


def _head64(s, x):
    return _rms64(x, s.dec.w.norm, s.cfg.rms_norm_eps) @ s.dec.w.lm_head.to(F64).T


def _exact_prefill(case, s):
    kv = s.cache.pool.to(F64)
    rows = [(slice(a, b), i, 0) for i, (a, b) in enumerate(zip(s.offsets, s.offsets[1:]))]
    x = _qwen64(s, s.ids, s.pos, rows, kv)
    return {"logits": _head64(s, x[[b - 1 for b in s.offsets[1:]]]), "kv": kv}


def _exact_decode(case, s):
    kv = s.cache.pool.to(F64)
    x = _qwen64(s, s.tokens, s.lens, [(slice(i, i + 1), i, n) for i, n in enumerate(s.ctx)], kv)
    return {"logits": _head64(s, x), "kv": kv}


def _work_qwen(case, lens, firsts):
    c = OmChatQwen2Config(num_hidden_layers=QWEN_LAYERS)
    C, I, T = c.hidden_size, c.intermediate_size, sum(lens)
    layer = (c.num_attention_heads * 2 + 2 * c.num_key_value_heads) * 128 * C + 3 * C * I
    head = c.vocab_size * C
    pairs = sum(n * f + n * (n + 1) // 2 for n, f in zip(lens, firsts))
    kv = 2 * c.num_key_value_heads * 128 * 2 * QWEN_LAYERS
    return {"bytes": 2 * (QWEN_LAYERS * layer + head) + T * C * 2 + kv * (T + sum(firsts)) + len(lens) * c.vocab_size * 4,
            "flops": 2 * T * layer * QWEN_LAYERS + 2 * len(lens) * head + QWEN_LAYERS * 4 * pairs * c.num_attention_heads * 128}


# ------------------------------------------------------------------------------------------------------------ latent attention
def _prepare_latent(case, seed):
    s, rn, dt = State(), _seeded(seed), DTYPES[case["dtype"]]
    s.portions = _portions(case)
    s.pos, s.slot = _addresses(s.portions)
    T, H, r, dr, dn = _rows(s.portions), case["heads"], case["rank"], case["rot"], case["head"]
    s.dims = (T, H, r, dr, dn)
    s.short = dt == F32 or T <= 64       # short steps take queries and latents from one fp32 product
    s.cache = _paged([r + dr], s.portions, dt, seed)
    s.cache.pools[0].copy_(rn(*s.cache.pools[0].shape, dtype=dt))
    s.latent = LatentAttention(torch.device(DEV, torch.cuda.current_device()), dt)
    s.rot = RotarySpec(dims=dr, base=1e6, halves=True)
    s.q = rn(T, H * (dn + dr), dtype=F32 if s.short else dt)
    s.dkv = rn(T, r + dr)
    s.norm = rn(r, std=0.2, mean=1.0, dtype=dt)
    s.uk_t = rn(H, r, dn, std=1.5 * r ** -0.5, dtype=dt)
    s.uv = rn(H * dn, r, std=r ** -0.5, dtype=dt)
    s.sink = rn(H, std=1.5, mean=1.0) if case["sink"] else None
    s.gate = rn(T, H * dn, dtype=F32 if s.short else dt) if case["gate"] else None
    s.window = case["window"] or None
    s.scale = (dn + dr) ** -0.5
    s.latent.rotary.get(s.rot, s.cache.capacity)
    return s


def _run_latent(s):
    T, H, r, dr, dn = s.dims
    dt, cache = s.cache.pools[0].dtype, s.cache
    plans = {"decode_keys": 1 << max(max(cache.host_lens) - 1, 0).bit_length()} if _decoding(s.portions) else {"portions": s.portions}
    qcat = torch.empty(T, H, r + dr, device=DEV, dtype=dt)
    qn = torch.empty(T, H * dn, device=DEV, dtype=dt) if s.short and dt != F32 else None
    seqlib.latent_rope_store(s.dkv, r, dr, s.norm, EPS, s.latent.rotary.get(s.rot, cache.capacity), dr, s.pos, s.slot, cache.block_table,
                             cache.page_size, cache.pools[0], s.q, H, dn, qcat, qn=qn, rot_halves=True)
    qa, sx = (s.q, dn + dr) if qn is None else (qn, dn)
    seqlib.linear(qa, s.uk_t, qcat, M=T, N=r, K=dn, ldx=qa.stride(0), sx=sx, ldw=dn, sw=r * dn, ldy=H * (r + dr), sy=r + dr, batch=H)
    olat = s.latent.attend(qcat, r, dr, cache.pools[0], cache, s.pos, s.slot, plans, s.scale, sink=s.sink, window=s.window)
    att = torch.empty(T, H * dn, device=DEV, dtype=dt)
    seqlib.linear(olat, s.uv, att, M=T, N=dn, K=r, ldx=H * r, sx=r, ldw=r, sw=dn * r, ldy=H * dn, sy=dn, batch=H, gate=s.gate)
    return {"att": att, "cache": cache.pools[0]}


def _halves64(x, pos, dims, base):
    """x [T, ..., d]: dimensions i and i + dims / 2 turn by pos * base^(-2i / dims)."""
    h = dims // 2
    a = pos.to(F64)[:, None] * base ** (-torch.arange(h, dtype=F64, device=DEV) / h)
    a = a.view(len(pos), *([1] * (x.dim() - 2)), h)
    u, v = x[..., :h], x[..., h:dims]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., dims:]], -1)


def _softmax64(sc, hidden, sink):
    """Softmax over the last axis of sc [heads, rows, keys] with an optional further term exp(sink) of the denominator."""
    sc = sc.masked_fill(hidden, -math.inf)
    if sink is None:
        return torch.softmax(sc, -1)
    full = torch.cat([sc, sink.to(F64)[:, None, None].expand(-1, sc.shape[1], 1)], -1)
    return torch.softmax(full, -1)[..., :-1]


def _hidden(n, first, window=None, chunk=None):
    i, j = first + torch.arange(n, device=DEV)[:, None], torch.arange(first + n, device=DEV)[None, :]
    hid = j > i
    if window:
        hid = hid | (i - j >= window)
    return hid | (i // chunk != j // chunk) if chunk else hid


def _exact_latent(case, s):
    T, H, r, dr, dn = s.dims
    pool = s.cache.pools[0].to(F64).view(-1, r + dr)
    dkv, q = s.dkv.to(F64), s.q.to(F64).view(T, H, dn + dr)
    new = torch.cat([_rms64(dkv[:, :r], s.norm, EPS), _halves64(dkv[:, r:], s.pos, dr, 1e6)], 1)
    qcat = torch.cat([torch.einsum("thd,hrd->thr", q[..., :dn], s.uk_t.to(F64)), _halves64(q[..., dn:], s.pos, dr, 1e6)], -1)
    o = torch.empty(T, H, r, dtype=F64, device=DEV)
    for row, n, slot, first in s.portions:
        at = _places(s.cache, slot, first + n)
        pool[at[first:]] = new[row:row + n]
        keys = pool[at]
        p = _softmax64(qcat[row:row + n].transpose(0, 1) @ keys.T * s.scale, _hidden(n, first, s.window), s.sink)
        o[row:row + n] = (p @ keys[:, :r]).transpose(0, 1)
    att = torch.einsum("thr,hvr->thv", o, s.uv.to(F64).view(H, dn, r)).reshape(T, H * dn)
    if s.gate is not None:
        att = att * torch.sigmoid(s.gate.to(F64))
    return {"att": att, "cache": pool.view_as(s.cache.pools[0])}


def _seen(portions, window=None, chunk=None):
    """(pairs of row and visible key, cached rows that are visible to any row of the step)."""
    pairs = keys = 0
    for _, n, _, first in portions:
        for p in range(first, first + n):
            pairs += min(p + 1, window or p + 1, p % chunk + 1 if chunk else p + 1)
        low = max(0, first + 1 - window) if window else 0
        keys += first - min(first, max(low, first // chunk * chunk if chunk else 0)) + n
    return pairs, keys


def _work_latent(case):
    portions = _portions(case)
    T, H, r, dr, dn = _rows(portions), case["heads"], case["rank"], case["rot"], case["head"]
    e = 2 if case["dtype"] == "bf16" else 4
    eq = 4 if case["dtype"] == "f32" or T <= 64 else 2
    pairs, keys = _seen(portions, case["window"] or None)
    return {"bytes": T * H * (dn + dr) * eq + T * (r + dr) * 4 + keys * (r + dr) * e + 2 * H * r * dn * e + T * H * dn * (e + (eq if case["gate"] else 0)),
            "flops": 4 * T * H * r * dn + 2 * pairs * H * (2 * r + dr)}


# ---------------------------------------------------------------------------------------------- windowed and chunked attention
def _prepare_window(case, seed):
    s, rn, dt = State(), _seeded(seed), DTYPES[case["dtype"]]
    s.portions = _portions(case)
    s.pos, s.slot = _addresses(s.portions)
    T, H, G, d = _rows(s.portions), case["heads"], case["kv_heads"], case["head"]
    s.dims, s.chunked = (T, H, G, d), case["kind"] == "chunk"
    s.cache = _paged([2 * G * d], s.portions, dt, seed)
    s.cache.pools[0].copy_(rn(*s.cache.pools[0].shape, dtype=dt))
    s.z = rn(T, H * d + 2 * G * d + H)           # q | k | v | head gates, as the stacked projection leaves them
    s.q_norm, s.k_norm = rn(H * d, std=0.3, mean=1.3, dtype=dt), rn(G * d, std=0.3, mean=1.3, dtype=dt)
    s.window, s.scale, s.softcap = case["window"], d ** -0.5, 50.0
    s.bias = None if s.chunked else rn(s.window, H, std=0.5)
    s.one = torch.zeros(H, device=DEV) if s.chunked else None
    s.latent = LatentAttention(torch.device(DEV, torch.cuda.current_device()), dt)   # for its rotary tables
    s.rot = RotarySpec(dims=d // 2, base=1e5, halves=True)
    s.latent.rotary.get(s.rot, s.cache.capacity)
    return s


def _run_window(s):
    (T, H, G, d), cache, pool = s.dims, s.cache, s.cache.pools[0]
    dt, nq, nk = pool.dtype, H * d, G * d
    z, k = s.z, s.z[:, nq:nq + nk]
    q = torch.empty(T, nq, device=DEV, dtype=dt)
    att = torch.empty(T, nq, device=DEV, dtype=dt)
    if s.chunked:      # keys as projected serve as values; the normed keys are rotated
        turn = dict(cs=s.latent.rotary.get(s.rot, cache.capacity), head=d, rot_dims=s.rot.dims, rot_halves=True)
        seqlib.qk_norm_kv_store(z[:, :nq], s.q_norm, k, s.k_norm, k, EPS, s.pos, s.slot, cache.block_table, cache.page_size, pool, q, **turn)
        window, kw = seqlib.WINDOW_ALL, dict(sink=s.one, gate=z[:, nq + 2 * nk:], gate_act=seqlib.GATE_SIGMOID, gate_heads=True, chunk=s.window)
    else:
        seqlib.qk_norm_kv_store(z[:, :nq], s.q_norm, k, s.k_norm, z[:, nq + nk:nq + 2 * nk], EPS, s.pos, s.slot, cache.block_table, cache.page_size,
                                pool, q)
        window, kw = s.window, {}
    if seqlib.window_attn_mma_ok(H, G, d, d, dt):
        items = None
        if not _decoding(s.portions):
            items = seqlib.window_attn_items(s.portions, H // G, DEV, s.window if s.chunked else seqlib.WINDOW_ALL)
        seqlib.window_attn_mma(q, H, G, d, d, pool, cache.block_table, cache.page_size, items, s.pos, s.slot, window, s.scale, s.softcap, s.bias, att, **kw)
    else:
        seqlib.window_attn(q, H, G, d, d, pool, cache.block_table, cache.page_size, s.pos, s.slot, window, s.scale, s.softcap, s.bias, att, **kw)
    return {"att": att, "cache": pool}


def _exact_window(case, s):
    T, H, G, d = s.dims
    nq, nk = H * d, G * d
    z = s.z.to(F64)
    q, k = _rms64(z[:, :nq], s.q_norm, EPS).view(T, H, d), _rms64(z[:, nq:nq + nk], s.k_norm, EPS).view(T, G, d)
    v = (z[:, nq:nq + nk] if s.chunked else z[:, nq + nk:nq + 2 * nk]).view(T, G, d)
    if s.chunked:
        q, k = _halves64(q, s.pos, d // 2, 1e5), _halves64(k, s.pos, d // 2, 1e5)
    pool = s.cache.pools[0].to(F64).view(-1, 2 * nk)
    att = torch.empty(T, H, d, dtype=F64, device=DEV)
    for row, n, slot, first in s.portions:
        at = _places(s.cache, slot, first + n)
        pool[at[first:]] = torch.cat([k[row:row + n].reshape(n, nk), v[row:row + n].reshape(n, nk)], 1)
        keys, values = (t.view(-1, G, d).transpose(0, 1).repeat_interleave(H // G, 0) for t in pool[at].split(nk, 1))
        sc = q[row:row + n].transpose(0, 1) @ keys.transpose(1, 2) * s.scale
        sc = s.softcap * torch.tanh(sc / s.softcap)
        hid = _hidden(n, first, None if s.chunked else s.window, s.window if s.chunked else None)
        if s.bias is not None:
            back = (first + torch.arange(n, device=DEV)[:, None] - torch.arange(first + n, device=DEV)[None, :]).clamp(0, s.window - 1)
            sc = sc + s.bias.to(F64)[back].permute(2, 0, 1)
        att[row:row + n] = (_softmax64(sc, hid, s.one) @ values).transpose(0, 1)
    if s.chunked:
        att = att * torch.sigmoid(z[:, nq + 2 * nk:])[:, :, None]
    return {"att": att.reshape(T, nq), "cache": pool.view_as(s.cache.pools[0])}


def _work_window(case):
    portions = _portions(case)
    T, H, G, d = _rows(portions), case["heads"], case["kv_heads"], case["head"]
    chunked, e = case["kind"] == "chunk", 2 if case["dtype"] == "bf16" else 4
    pairs, keys = _seen(portions, None if chunked else case["window"], case["window"] if chunked else None)
    return {"bytes": T * (H * d + (1 if chunked else 2) * G * d + (H if chunked else 0)) * 4 + keys * 2 * G * d * e + T * H * d * e
            + (0 if chunked else case["window"] * H * 4), "flops": 4 * pairs * H * d}


# ----------------------------------------------------------------------------------------------------------- recurrent layers
TAPS = 4


def _prepare_scan(case, seed):
    s, rn, dt = State(), _seeded(seed), DTYPES[case["dtype"]]
    s.portions, s.kind = _portions(case), case["kind"]
    s.pos, s.slot = _addresses(s.portions)
    T, P, H, G, d, dv = _rows(s.portions), len(s.portions), case["heads"], case["groups"], case["dim"], case["vdim"]
    s.dims, s.dtype = (T, P, H, G, d, dv), dt
    s.row_begin = torch.tensor([p[0] for p in s.portions] + [T], dtype=I32, device=DEV)
    ch = 2 * G * d + H * dv
    s.z = rn(T, ch)                                     # what the convolution reads
    s.conv, s.conv_b = rn(ch, TAPS, std=TAPS ** -0.5, dtype=dt), rn(ch, std=0.1, dtype=dt) if s.kind == "steps" else None
    s.ring = torch.zeros(P, TAPS - 1, ch, device=DEV)
    s.S = torch.zeros(P, H, d, dv, device=DEV)
    s.a, s.beta = rn(T, H), rn(T, H)
    s.A_log = rn(H)
    s.gate = rn(T, H * dv, dtype=dt if s.kind == "steps" else F32)
    if s.kind == "steps":
        s.dt_bias, s.D = rn(H, std=1.5, mean=-3.0), rn(H, mean=1.0)      # decays from a few tokens to hundreds
        s.norm = rn(H * dv, std=0.2, mean=1.0, dtype=dt)
    else:
        s.dt_bias, s.norm = rn(H, std=1.0, mean=-2.0), rn(dv, std=0.2, mean=1.0, dtype=dt)
    if s.kind == "channel":                             # decays per key channel come from a narrow product
        s.low, s.a2, s.dt_bias = rn(T, 64), rn(H * d, 64, std=0.125, dtype=dt), rn(H * d, std=1.0, mean=-2.0)
    return s


def _run_scan(s):
    T, P, H, G, d, dv = s.dims
    nqk = G * d
    u = torch.empty(T, s.z.shape[1], device=DEV)
    y = torch.empty(T, H * dv, device=DEV)
    out = torch.empty(T, H * dv, device=DEV, dtype=s.dtype)
    if s.kind == "steps":                               # x | B | C behind the convolution
        seqlib.causal_conv_silu(s.z, s.conv, s.pos, s.slot, s.ring, u, bias=s.conv_b, single_rows=P == T)
        seqlib.linear_state_scan(u[:, H * dv + nqk:], u[:, H * dv:H * dv + nqk], u[:, :H * dv], s.S, y, s.row_begin, P, s.pos, s.slot, H, G, d, dv,
                                 step_size=True, a=s.a, A_log=s.A_log, dt_bias=s.dt_bias, D=s.D)
        seqlib.gate_rms_rows(y, G, s.norm, EPS, s.gate, seqlib.GATE_SILU, out)
    else:                                               # q | k | v, unit queries and keys
        seqlib.causal_conv_silu(s.z, s.conv, s.pos, s.slot, s.ring, u, unit_channels=2 * nqk, unit_group=d, unit_eps=1e-6, scaled_channels=nqk,
                                unit_mult=d ** -0.5, single_rows=P == T)
        a, prep = s.a, False
        if s.kind == "channel":
            a = dense_linear(s.low, s.a2, F32, tensor_gemm=s.dtype == BF16)
            prep = T >= 32 * P                          # long portions: the decays in a pass of their own
            if prep:
                seqlib.map_rows(a, seqlib.MAP_DECAY, s.A_log, s.dt_bias, d)
        seqlib.linear_state_scan(u[:, :nqk], u[:, nqk:2 * nqk], u[:, 2 * nqk:], s.S, y, s.row_begin, P, s.pos, s.slot, H, G, d, dv, a=a, A_log=s.A_log,
                                 dt_bias=s.dt_bias, channel_decay=s.kind == "channel", beta=s.beta, decay_given=prep)
        seqlib.gated_rms_rows(y, H, dv, s.norm, EPS, s.gate, seqlib.GATE_SIGMOID if s.kind == "channel" else seqlib.GATE_SILU, out)
    return {"out": out, "state": s.S, "ring": s.ring}


def _conv64(z, w, b):
    u = torch.zeros_like(z) if b is None else b.to(F64).expand_as(z).clone()
    for j in range(TAPS):
        back = TAPS - 1 - j
        if back < z.shape[0]:
            u[back:] += w[:, j].to(F64) * z[:z.shape[0] - back]
    return torch.nn.functional.silu(u)


def _recurrence64(q, k, v, g, u_scale, delta, S):
    """q / k [T, P, H, d], v [T, P, H, dv], g [T, P, H, d or 1], u_scale [T, P, H, 1]; rows past a portion's end have g = 1 and u_scale = 0."""
    y = torch.empty_like(v)
    for t in range(q.shape[0]):
        S *= g[t][..., None]
        u = v[t] - torch.einsum("phdv,phd->phv", S, k[t]) if delta else v[t]
        S += k[t][..., None] * (u_scale[t] * u)[..., None, :]
        y[t] = torch.einsum("phdv,phd->phv", S, q[t])
    return y


def _exact_scan(case, s):
    T, P, H, G, d, dv = s.dims
    nqk, z = G * d, s.z.to(F64)
    u = torch.cat([_conv64(z[row:row + n], s.conv, s.conv_b) for row, n, _, _ in s.portions])
    ring = s.ring.to(F64)
    for row, n, slot, _ in s.portions:
        for p in range(max(0, n - TAPS + 1), n):
            ring[slot, p % (TAPS - 1)] = z[row + p]
    if s.kind == "steps":
        v, k, q = u[:, :H * dv], u[:, H * dv:H * dv + nqk], u[:, H * dv + nqk:]
        step = torch.nn.functional.softplus(s.a.to(F64) + s.dt_bias.to(F64), threshold=1e9)
        g, scale = torch.exp(-torch.exp(s.A_log.to(F64)) * step)[..., None], step[..., None]
    else:
        q, k, v = u.split([nqk, nqk, H * dv], 1)
        q, k = (t.view(T, G, d) / torch.sqrt((t.view(T, G, d) ** 2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q = q * d ** -0.5
        scale = torch.sigmoid(s.beta.to(F64))[..., None]
        a = s.a.to(F64)[..., None] + s.dt_bias.to(F64).view(H, -1) if s.kind == "delta" else (s.low.to(F64) @ s.a2.to(F64).T + s.dt_bias.to(F64)).view(T, H, d)
        g = torch.exp(-torch.exp(s.A_log.to(F64))[:, None] * torch.nn.functional.softplus(a, threshold=1e9))
    q, k = (t.reshape(T, G, d).repeat_interleave(H // G, 1) for t in (q, k))
    v = v.reshape(T, H, dv)
    most = max(p[1] for p in s.portions)

    def side(x, fill):   # rows [T, ...] -> [longest portion, portions, ...]
        o = torch.full((most, P, *x.shape[1:]), fill, dtype=F64, device=DEV)
        for row, n, slot, _ in s.portions:
            o[:n, slot] = x[row:row + n]
        return o
    S = torch.zeros(P, H, d, dv, dtype=F64, device=DEV)
    o = _recurrence64(side(q, 0.0), side(k, 0.0), side(v, 0.0), side(g, 1.0), side(scale, 0.0), s.kind != "steps", S)
    y = torch.cat([o[:n, slot] for _, n, slot, _ in s.portions])
    gate = s.gate.to(F64)
    if s.kind == "steps":
        y = (y + s.D.to(F64)[:, None] * v).reshape(T, H * dv) * torch.nn.functional.silu(gate)
        y = y.view(T, G, -1)
        y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + EPS)).reshape(T, -1) * s.norm.to(F64)
    else:
        act = torch.sigmoid(gate) if s.kind == "channel" else torch.nn.functional.silu(gate)
        y = _rms64(y, s.norm, EPS).reshape(T, -1) * act
    return {"out": y, "state": S, "ring": ring}


def _work_scan(case):
    portions = _portions(case)
    T, P, H, G, d, dv = _rows(portions), len(portions), case["heads"], case["groups"], case["dim"], case["vdim"]
    e, steps = 2 if case["dtype"] == "bf16" else 4, case["kind"] == "steps"
    a = T * H * 4 if case["kind"] != "channel" else T * 64 * 4 + H * d * 64 * e
    return {"bytes": T * (2 * G * d + H * dv) * 4 + a + (0 if steps else T * H * 4) + T * H * dv * ((e if steps else 4) + e) + P * H * d * dv * 4,
            "flops": T * H * d * dv * (6 if steps else 8)}


# ------------------------------------------------------------------------------------------------------------ a model in service
def _serve_dict(case):
    C, H = case["width"], case["heads"]
    mlp = {"ff": 2 * C, "kind": "dense"}
    return {"architecture": "Sorupel", "vocab": case["vocab"], "width": C, "norm": {"eps": 1e-5},
            "embedding": {"bigram": {"buckets": 4096, "mul_cur": 7919, "mul_prev": 104729}},
            "layers": [
                {"type": "mamba2", "mlp": mlp, "mixer": {"conv": TAPS, "groups": 4, "heads": C // 32, "norm_groups": 4, "state": 64, "vdim": 64}},
                {"type": "latent_attention", "mlp": mlp, "mixer": {"dim": 128, "heads": H, "kv_rank": 256, "rot": {"base": 1e6, "dims": 64}, "rot_dim": 64,
                                                                   "scale": 192 ** -0.5, "vdim": 128}},
                {"type": "attention", "mlp": mlp, "mixer": {"dim": 128, "heads": H, "kv_heads": max(1, H // 4), "mask": {"size": 256},
                                                            "rot": {"base": 1e5, "dims": 64}, "scale": 128 ** -0.5, "softcap": 50.0, "vdim": 128}}]}


def _prepare_serve(case, seed):
    s = State()
    s.cfg = _serve_dict(case)
    config = SorupelConfig.from_dict(s.cfg)
    s.sd = sorupel.random_state_dict(config, seed)
    model = sorupel.SorupelForCausalLM.from_state_dict(s.sd, config, device=DEV, dtype=DTYPES[case["dtype"]])
    gen = torch.Generator().manual_seed(int(seed))
    s.prompts = [torch.randint(0, case["vocab"], (n + case["steps"],), generator=gen).tolist() for n in _numbers(case["lens"])]
    s.steps = case["steps"]
    s.sched = StepScheduler(model, max_tokens=sum(-(-len(p) // 64) * 64 for p in s.prompts), slots=len(s.prompts))
    return s


def _run_serve(s):
    names = ["r%d" % i for i in range(len(s.prompts))]
    fed = [len(p) - s.steps for p in s.prompts]
    got = [s.sched.run_step([(k, p[:n], [n - 1]) for k, p, n in zip(names, s.prompts, fed)]).clone()]
    for t in range(s.steps):
        last = s.sched.run_step([(k, [p[n + t]], [0]) for k, p, n in zip(names, s.prompts, fed)], end=names if t == s.steps - 1 else ())
        got.append(last.clone())      # the step's logits are overwritten by the next one
    return torch.stack(got)


def _exact_serve(case, s):
    W = {k: v.to(DEV).to(F64) for k, v in s.sd.items()}
    eps, silu = s.cfg["norm"]["eps"], torch.nn.functional.silu
    big = s.cfg["embedding"]["bigram"]
    out = []
    for tokens in s.prompts:
        T = len(tokens)
        t = torch.tensor(tokens, device=DEV)
        pair = (t[:-1] * big["mul_prev"] + t[1:] * big["mul_cur"]) % big["buckets"]
        x = W["embed"][t] + W["bigram"][torch.cat([torch.tensor([big["buckets"]], device=DEV), pair])]
        pos = torch.arange(T, device=DEV)
        for i, layer in enumerate(s.cfg["layers"]):
            m, p = layer["mixer"], "l%d.mix." % i
            h = _rms64(x, W["l%d.norm1" % i], eps)
            if layer["type"] == "mamba2":
                H, dv, d, G = m["heads"], m["vdim"], m["state"], m["groups"]
                z, xbc, dt = (h @ W[p + "in"].T).split([H * dv, H * dv + 2 * G * d, H], 1)
                v, k, q = _conv64(xbc, W[p + "conv"], W[p + "conv.b"]).split([H * dv, G * d, G * d], 1)
                k, q = (a.reshape(T, 1, G, d).repeat_interleave(H // G, 2) for a in (k, q))
                dt = torch.nn.functional.softplus(dt + W[p + "dt_bias"], threshold=1e9).view(T, 1, H, 1)
                v = v.reshape(T, 1, H, dv)
                y = _recurrence64(q, k, v, torch.exp(-torch.exp(W[p + "A_log"])[:, None] * dt), dt, False,
                                  torch.zeros(1, H, d, dv, dtype=F64, device=DEV))
                y = (y + W[p + "D"][:, None] * v).reshape(T, H * dv) * silu(z)
                y = y.view(T, m["norm_groups"], -1)
                y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps)).reshape(T, -1) * W[p + "norm"]
            elif layer["type"] == "latent_attention":
                H, dn, dr, r = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
                q, dkv = (h @ W[p + "q"].T).view(T, H, dn + dr), h @ W[p + "dkv"].T
                c, kr = _rms64(dkv[:, :r], W[p + "dkv.norm"], eps), _halves64(dkv[:, r:], pos, dr, m["rot"]["base"])
                k, v = (c @ W[p + "uk"].T).view(T, H, dn), (c @ W[p + "uv"].T).view(T, H, -1)
                qr = _halves64(q[..., dn:], pos, dr, m["rot"]["base"])
                sc = (q[..., :dn].transpose(0, 1) @ k.permute(1, 2, 0) + qr.transpose(0, 1) @ kr.T) * m["scale"]
                y = (_softmax64(sc, _hidden(T, 0), W[p + "sink"]) @ v.transpose(0, 1)).transpose(0, 1).reshape(T, -1) * torch.sigmoid(h @ W[p + "g"].T)
            else:
                H, G, d, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
                q, k0 = h @ W[p + "q"].T, h @ W[p + "k"].T
                q, k = (_halves64(_rms64(a, W[p + n], eps).view(T, -1, d), pos, rot["dims"], rot["base"]).transpose(0, 1)
                        for a, n in ((q, "q.norm"), (k0, "k.norm")))
                k, v = (a.repeat_interleave(H // G, 0) for a in (k, k0.view(T, G, d).transpose(0, 1)))
                sc = m["softcap"] * torch.tanh(q @ k.transpose(1, 2) * m["scale"] / m["softcap"])
                y = _softmax64(sc, _hidden(T, 0, chunk=m["mask"]["size"]), torch.zeros(H, dtype=F64, device=DEV)) @ v
                y = (y.transpose(0, 1) * torch.sigmoid(h @ W[p + "g"].T)[:, :, None]).reshape(T, -1)
            x = x + y @ W[p + "o"].T
            q = "l%d.mlp." % i
            h = _rms64(x, W["l%d.norm2" % i], eps)
            x = x + (torch.nn.functional.gelu(h @ W[q + "gate"].T, approximate="tanh") * (h @ W[q + "up"].T)) @ W[q + "down"].T
        out.append((_rms64(x, W["final.norm"], eps) @ W["head"].T)[T - s.steps - 1:])
    return torch.stack(out, 1)


def _work_serve(case):
    C, H, lens, steps = case["width"], case["heads"], _numbers(case["lens"]), case["steps"]
    sH, G = C // 32, max(1, H // 4)
    inner = sH * 64
    mix = [C * (2 * inner + 2 * 4 * 64 + sH) + inner * C,
           C * (H * 192 + H * 128 + 320) + H * 256 * 256 + H * 128 * C,
           C * (H * 128 + G * 128 + H) + H * 128 * C]
    weights, head = sum(mix) + 3 * 6 * C * C, case["vocab"] * C
    T, n = sum(lens) + steps * len(lens), len(lens)
    e = 2 if case["dtype"] == "bf16" else 4
    pairs = sum((L + steps) * (L + steps + 1) // 2 for L in lens)
    # every step reads the weights once; the scan's states are read and written by every decoding step
    return {"bytes": (1 + steps) * (weights + head) * e + 2 * steps * n * sH * 64 * 64 * 4 + (1 + steps) * n * case["vocab"] * 4,
            "flops": 2 * T * weights + 2 * (1 + steps) * n * head + 6 * T * sH * 64 * 64 + 2 * pairs * H * 320 + 4 * pairs * H * 128}


# ------------------------------------------------------------------------------------------------------------- what is asked for
_PREPARE = {"vision": _prepare_vision, "prefill": _prepare_prefill, "decode": _prepare_decode, "latent": _prepare_latent, "window": _prepare_window,
            "scan": _prepare_scan, "serve": _prepare_serve}
_RUN = {"vision": _run_vision, "prefill": _run_prefill, "decode": _run_decode, "latent": _run_latent, "window": _run_window, "scan": _run_scan,
        "serve": _run_serve}
_EXACT = {"vision": _exact_vision, "prefill": _exact_prefill, "decode": _exact_decode, "latent": _exact_latent, "window": _exact_window,
          "scan": _exact_scan, "serve": _exact_serve}


@torch.no_grad()
def prepare(case, seed):
    state = _PREPARE[case["op"]](case, seed)
    state.op = case["op"]
    return state


@torch.no_grad()
def run(state):
    return _RUN[state.op](state)


@torch.no_grad()
def exact(case, seed):
    return _EXACT[case["op"]](case, prepare(case, seed))


def work(case):
    op = case["op"]
    if op == "vision":
        return _work_vision(case)
    if op == "prefill":
        lens = _numbers(case["lens"])
        return _work_qwen(case, lens, [0] * len(lens))
    if op == "decode":
        ctx = _numbers(case["ctx"])
        return _work_qwen(case, [1] * len(ctx), ctx)
    return {"latent": _work_latent, "window": _work_window, "scan": _work_scan, "serve": _work_serve}[op](case)


def tolerance(case):
    """About four times what these paths are from the same sums in 64 bits (measured over listed and drawn cases): 0.012 for the logits of a
    few bf16 layers, 0.004 for one attention or vision block in bf16, 2e-6 for a whole model and 7e-7 for a layer in fp32."""
    op = case["op"]
    if op in ("prefill", "decode"):
        return {"rel": 0.03, "max": 0.25}
    if case.get("dtype") == "f32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.02 if op == "serve" else 0.015, "max": 0.3}
