"""CPU ORACLE (test infrastructure only) — torch restatement of the reference model graph.

This file is the checker for the CUDA path. It is imported only by tests/,
__graft_entry__.smoke() and bench.py's cpu_baseline / --impl reference legs.
Nothing in the product package may import it.

PARITY STATUS: *partly pinned*. The reference (MLX 0.15) cannot be executed in
this image (no mlx wheel), and its own test.py holds no numeric goldens,
so the arithmetic below is pinned two ways instead:
  * decoder (B=1, no pad) against transformers.Phi3ForCausalLM, CLIP tower
    against transformers.CLIPVisionModel hidden_states[-2][:,1:]
    (tests/test_oracle_vs_hf.py);
  * processors / index math against the reference's own numpy/PIL code executed
    with MLX stubbed (tests/golden/*, generated by tests/golden/make_golden.py).
MLX-internal rounding behaviour (dtype promotion, quantiser edge rule) is
restated from mlx 0.15 semantics and marked [mlx-inferred].

Each function cites the reference lines it follows (phi: = phi.py).

Precision modes (``prec``):
  'fp32' : every op in float32 (ideal arithmetic, HF cross-check mode)
  'ref'  : reference dtype flow with bf16 checkpoints [mlx-inferred]: bf16
           activations at module boundaries, fp32 rope/attention/KV (phi:451-460).
           The vision branch is the exception, by the same promotion rule: pixel_values
           enter as float32 (phi:279), fp32 x bf16 promotes to fp32, so the CLIP tower
           and img_projection run with fp32 activations end to end; the result is
           rounded to bf16 only when it is assigned into the bf16 text embeddings
           (phi:412-415)
  'b200' : as 'ref' but q,k,v are rounded to bf16 after rope (bf16 KV cache) and
           the attention output is rounded to bf16 — the precision delta
           the CUDA path takes deliberately
"""
import math
import torch
import torch.nn.functional as F


def _r(x, prec):
    """Round to bf16 and back when emulating a bf16 activation boundary."""
    if prec == 'fp32':
        return x
    return x.to(torch.bfloat16).to(torch.float32)


_W32 = {}


def _w(p):
    """fp32 view of a (bf16) parameter; converted once per tensor and memoised (full-size runs)."""
    if p.dtype == torch.float32:
        return p
    key = (p.data_ptr(), tuple(p.shape))
    t = _W32.get(key)
    if t is None or t[0] is not p:
        t = (p, p.to(torch.float32))
        _W32[key] = t
    return t[1]


def clear_weight_cache():
    _W32.clear()


# ----------------------------------------------------------------------------- quantiser
def quantize_q4g32(w, prec='ref', group=32, dtype=torch.float32):
    """Affine 4-bit, group 32 over the last axis. Restates mx.quantize(w, group_size=32)
    (bits=4) as called at phi:532 [mlx-inferred edge rule: the larger-magnitude edge of
    each group is exact and 0 stays representable]. Returns (q uint8 [...,G,32], scale, bias).
    In 'b200' mode scale/bias are rounded to bf16 before the codes are computed (the GPU
    cache stores bf16 scale+bias; stated rule). ``group`` generalises the same rule
    to nn.quantize(model, 64, 4) (quantize_model_weights below)."""
    shp = w.shape
    g = w.reshape(*shp[:-1], shp[-1] // group, group).to(dtype)
    w_max = g.amax(-1, keepdim=True)
    w_min = g.amin(-1, keepdim=True)
    mask = w_min.abs() > w_max.abs()
    scale = torch.clamp((w_max - w_min) / 15.0, min=1e-7)
    scale = torch.where(mask, scale, -scale)
    edge = torch.where(mask, w_min, w_max)
    q0 = torch.round(edge / scale)
    scale = torch.where(q0 != 0, edge / q0, scale)
    bias = torch.where(q0 == 0, torch.zeros_like(edge), edge)
    if prec == 'b200':
        scale = scale.to(torch.float32).to(torch.bfloat16).to(dtype)
        bias = bias.to(torch.float32).to(torch.bfloat16).to(dtype)
        scale = torch.where(scale == 0, torch.full_like(scale, 1e-7), scale)
    q = torch.clamp(torch.round((g - bias) / scale), 0, 15).to(torch.uint8)
    return q, scale, bias


def dequantize_q4g32(q, scale, bias, shape):
    """mx.dequantize counterpart (phi:536-537): q*scale + bias."""
    return (q.to(torch.float32) * scale + bias).reshape(shape)


def lora_modules(lora_cfg, lora_weights, n_layers):
    """_linear_to_lora_layers (pv:234-245): which Linear modules get a LoRALinear wrapper, and with what scale
    (phi:121: scale * alpha / r). Returns the `lora` argument of Phi3Oracle."""
    layers = lora_cfg['lora_layers']
    if isinstance(layers, int):
        layers = list(range(n_layers))[-layers:]
    lp = lora_cfg['lora_parameters']
    sc = lp['scale'] * (lp['alpha'] / lp['rank'])
    return {f'model.layers.{i}.{t}': (lora_weights[f'model.layers.{i}.{t}.lora_a'], lora_weights[f'model.layers.{i}.{t}.lora_b'], sc)
            for i in layers for t in lora_cfg['lora_targets']}


def quantize_model_weights(weights, group=64, prec='b200'):
    """`quantize_model=True`: nn.quantize(model, group_size=64, bits=4) (pv:264,291-305) turns every nn.Linear and
    nn.Embedding into its quantised counterpart [mlx-inferred: default class_predicate = modules with `to_quantized`;
    conv / norm / class-embedding / GN parameters stay]. Scales and biases have the checkpoint dtype (bf16) and the
    matmul dequantises on the fly, so the model behaves as if its 2-D `.weight` matrices were replaced by
    q * scale + bias. Returns a new dict with those matrices as fp32 dequantised images; prec='b200' additionally
    rounds the image to bf16, which is the operand the B200 tensor-core GEMMs consume (the decode-time 4-bit kernel
    applies the affine map in fp32, i.e. the unrounded image: a difference of one bf16 rounding per weight)."""
    out = {}
    for k, v in weights.items():
        if k.endswith('.weight') and v.dim() == 2 and v.shape[-1] % group == 0:
            # float64 statistics: device-independent codes (see phi3_b200/quant.py)
            q, sc, bi = quantize_q4g32(v, prec='b200', group=group, dtype=torch.float64)
            img = (q.to(torch.float32) * sc.to(torch.float32) + bi.to(torch.float32)).reshape(v.shape)
            out[k] = img.to(torch.bfloat16).to(torch.float32) if prec == 'b200' else img
        else:
            out[k] = v
    return out


# ----------------------------------------------------------------------------- rope / mask / cache
class SuRoPE:
    """phi:487-507. cos/sin table for all L_all positions, static short/long switch (H7),
    both multiplied by sqrt(1 + ln(max/orig)/ln(orig))."""

    def __init__(self, cfg, L_all, pids):
        dim = cfg.hidden_size // cfg.num_attention_heads
        sf = math.sqrt(1 + math.log(cfg.max_position_embeddings / cfg.original_max_position_embeddings)
                       / math.log(cfg.original_max_position_embeddings))
        fac = cfg.rope_scaling["long_factor"] if L_all > cfg.original_max_position_embeddings \
            else cfg.rope_scaling["short_factor"]
        if pids is None:
            pos = torch.arange(L_all, dtype=torch.float32)[None]
        else:
            pids = torch.as_tensor(pids).to(torch.float32)
            ext = pids[:, -1][:, None] + 1 + torch.arange(L_all - pids.shape[1], dtype=torch.float32)[None, :]
            pos = torch.cat([pids, ext], dim=1)
        inv_freq = 1.0 / (torch.tensor(fac, dtype=torch.float32)
                          * cfg.rope_theta ** (torch.arange(0, dim, 2, dtype=torch.float32) / dim))
        freqs = pos[:, :, None] * inv_freq[None, None, :]          # fp32 product, [B|1, L_all, dim/2]
        emb = torch.cat([freqs, freqs], dim=-1)
        self.cos = (torch.cos(emb) * sf)[:, None]                  # [B|1,1,L_all,dim]
        self.sin = (torch.sin(emb) * sf)[:, None]

    def __call__(self, past_L, new_L):
        return self.cos[:, :, past_L:past_L + new_L], self.sin[:, :, past_L:past_L + new_L]


def rotate_half(x, cos, sin):
    """phi:418-423 (half-split layout)."""
    mid = x.shape[-1] // 2
    x1, x2 = x[..., :mid], x[..., mid:]
    return x * cos + torch.cat([-x2, x1], dim=-1) * sin


class Mask4D:
    """phi:550-563 as a boolean 'allowed' predicate: j<=i and m[i]*m[j]==1, m right-padded
    with ones. (The reference materialises the additive -inf form.)"""

    def __init__(self, L_all, mask):
        allow = torch.tril(torch.ones(L_all, L_all, dtype=torch.bool))[None, None]
        if mask is not None:
            m = torch.as_tensor(mask).to(torch.bool)
            m = F.pad(m, (0, L_all - m.shape[-1]), value=True)
            allow = allow & (m[:, None, :, None] & m[:, None, None, :])
        self.allow = allow

    def __call__(self, past_L, L):
        return self.allow[:, :, past_L:past_L + L, :past_L + L]


class KVCache:
    """phi:509-548. Dense preallocated buffer with the reference's offset bookkeeping.
    Quantised mode keeps the same read semantics as phi:528-540 (prompt part read back
    through 4-bit g32 quantise->dequantise from the second call on; later tokens exact).
    Extensions (no working reference behaviour): quantised + advance_offset
    and quantised + n_beam behave like the dense cache with the quantised prompt image."""

    def __init__(self, cfg, B, L, max_tokens, prec):
        self.max_tokens = max_tokens
        self.q = bool(getattr(cfg, "use_quantized_cache", False))
        self.offset = 0
        self.prec = prec
        self.shape = (B, cfg.num_key_value_heads, L + max_tokens, cfg.hidden_size // cfg.num_key_value_heads)
        self.k = self.v = None
        self.prompt_done = False

    def __call__(self, keys, values, n_beam):
        if self.max_tokens < 1:
            return keys, values                                            # phi:521-522
        if self.k is None:
            self.k = torch.zeros(self.shape)
            self.v = torch.zeros(self.shape)
        if n_beam > 1:                                                     # phi:523-527 (read only)
            pk = self.k[:, :, :self.offset].repeat_interleave(n_beam, dim=0)
            pv = self.v[:, :, :self.offset].repeat_interleave(n_beam, dim=0)
            return torch.cat([pk, keys], dim=-2), torch.cat([pv, values], dim=-2)
        new = self.offset + keys.shape[2]
        self.k[:, :, self.offset:new] = keys
        self.v[:, :, self.offset:new] = values
        first = not self.prompt_done
        self.prompt_done = True
        out = (self.k[:, :, :new].clone(), self.v[:, :, :new].clone())
        if self.q and first:                                               # phi:531-533
            B, N, _, D = self.shape
            for buf in (self.k, self.v):
                flat = buf[:, :, :new].reshape(B * N, -1)
                buf[:, :, :new] = dequantize_q4g32(*quantize_q4g32(flat, self.prec), (B, N, new, D))
        self.offset = new
        return out


# ----------------------------------------------------------------------------- decoder
class Phi3Oracle:
    """phi:425-617 (Phi3Attention, Phi3MLP, Phi3DecoderLayer, Phi3F/V, Phi3(V)ForCausalLM).
    ``weights``: dict of HF-named tensors (bf16 or fp32)."""

    def __init__(self, cfg, weights, prec='ref', clip_cfg=None, lora=None):
        self.cfg, self.w, self.prec = cfg, weights, prec
        # lora: {module name, e.g. 'model.layers.1.self_attn.qkv_proj': (lora_a [in,r], lora_b [r,out], scale*alpha/rank)}
        # — LoRALinear evaluated op for op (phi:129-133), NOT folded into the weight
        self.lora = lora or {}
        self.clip_cfg = clip_cfg
        self.n_heads = cfg.num_attention_heads
        self.n_kv = cfg.num_key_value_heads
        self.hd = cfg.hidden_size // cfg.num_attention_heads
        self.is_vision = any(k.startswith('model.vision_embed_tokens') for k in weights)

    # -- small ops
    def rms(self, x, w):
        """nn.RMSNorm -> mx.fast.rms_norm, fp32 accumulate (phi:478-479,571)."""
        y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + self.cfg.rms_norm_eps) * _w(w)
        return _r(y, self.prec)

    def _vprec(self):
        """precision mode of the vision branch: fp32 activations in the reference flow (see module docstring)"""
        return 'fp32' if self.prec == 'ref' else self.prec

    def lin(self, x, name, bias=False, round_out=True, prec=None):
        prec = self.prec if prec is None else prec
        y = x @ _w(self.w[name + '.weight']).T
        if bias:
            y = y + _w(self.w[name + '.bias'])
        if name in self.lora:                              # y = linear(x); z = (x @ A) @ B; (y + scale z).astype(x.dtype)
            a, b, sc = self.lora[name]
            y = _r(y, prec) + sc * ((x @ a.to(torch.float32)) @ b.to(torch.float32))
        return _r(y, prec) if round_out else y

    def attention(self, i, x, cache, cos, sin, allow, n_beam):
        """phi:440-460."""
        B, L, _ = x.shape
        p = f'model.layers.{i}.self_attn.'
        qkv = self.lin(x, p + 'qkv_proj')
        c1 = self.n_heads * self.hd
        c2 = c1 + self.n_kv * self.hd
        q, k, v = qkv[..., :c1], qkv[..., c1:c2], qkv[..., c2:]
        q = q.reshape(B, L, self.n_heads, -1).transpose(1, 2)
        k = k.reshape(B, L, self.n_kv, -1).transpose(1, 2)
        v = v.reshape(B, L, self.n_kv, -1).transpose(1, 2)
        if n_beam > 1:
            cos = cos.repeat_interleave(n_beam, 0) if cos.shape[0] > 1 else cos
            sin = sin.repeat_interleave(n_beam, 0) if sin.shape[0] > 1 else sin
            allow = allow.repeat_interleave(n_beam, 0) if allow.shape[0] > 1 else allow
        q = rotate_half(q, cos, sin)
        k = rotate_half(k, cos, sin)
        if self.prec == 'b200':
            q, k = _r(q, 'b200'), _r(k, 'b200')
        k, v = cache(k, v, n_beam)
        s = (q * self.hd ** -0.5) @ k.transpose(-1, -2)
        s = s.masked_fill(~allow, float('-inf'))
        # H1: rows with every key masked (pad queries) are defined as all-zero weights.
        dead = (~allow).all(-1, keepdim=True)
        pr = torch.softmax(s.masked_fill(dead, 0.0), dim=-1).masked_fill(dead, 0.0)
        o = (pr @ v).transpose(1, 2).reshape(B, L, -1)
        if self.prec == 'b200':
            o = _r(o, 'b200')
        return self.lin(o, p + 'o_proj')

    def mlp(self, i, x):
        """phi:462-471: gate = first half, up = second half."""
        p = f'model.layers.{i}.mlp.'
        gu = self.lin(x, p + 'gate_up_proj')
        g, u = gu.chunk(2, dim=-1)
        act = _r(_r(F.silu(g), self.prec) * u, self.prec)
        return self.lin(act, p + 'down_proj')

    # -- vision (phi:135-226, 374-416)
    def clip(self, px):
        """px [N,3,336,336] -> [N,576,1024]. 23 of 24 layers, no post_layernorm (phi:216-221)."""
        cc = self.clip_cfg
        P = 'model.vision_embed_tokens.img_processor.vision_model.'
        pr = self._vprec()
        wpe = _w(self.w[P + 'embeddings.patch_embedding.weight'])          # [O,kh,kw,I] (pv:374)
        x = F.conv2d(_r(px.to(torch.float32), pr), wpe.permute(0, 3, 1, 2), stride=cc.patch_size)
        x = _r(x.flatten(2).transpose(1, 2), pr)                           # [N,576,1024] row-major patches
        cls = _w(self.w[P + 'embeddings.class_embedding'])[None, None].expand(x.shape[0], 1, -1)
        x = _r(torch.cat([cls, x], dim=1) + _w(self.w[P + 'embeddings.position_embedding.weight'])[None], pr)

        def ln(x, name, eps):
            return _r(F.layer_norm(x, (x.shape[-1],), _w(self.w[name + '.weight']), _w(self.w[name + '.bias']), eps), pr)
        x = ln(x, P + 'pre_layrnorm', 1e-5)
        nh = cc.num_attention_heads
        for j in range(cc.num_hidden_layers - 1):
            L = P + f'encoder.layers.{j}.'
            h = ln(x, L + 'layer_norm1', cc.layer_norm_eps)
            N, T, D = h.shape
            q, k, v = (self.lin(h, L + f'self_attn.{n}_proj', bias=True, prec=pr).reshape(N, T, nh, -1).transpose(1, 2)
                       for n in 'qkv')
            a = torch.softmax((q * (D // nh) ** -0.5) @ k.transpose(-1, -2), dim=-1) @ v
            a = _r(a.transpose(1, 2).reshape(N, T, D), pr)
            x = _r(x + self.lin(a, L + 'self_attn.out_proj', bias=True, prec=pr), pr)
            h = ln(x, L + 'layer_norm2', cc.layer_norm_eps)
            h = self.lin(h, L + 'mlp.fc1', bias=True, prec=pr)
            h = _r(h * torch.sigmoid(1.702 * h), pr)                       # nn.gelu_fast_approx [mlx-inferred]
            x = _r(x + self.lin(h, L + 'mlp.fc2', bias=True, prec=pr), pr)
        return x[:, 1:]

    def image_embed(self, txt, pixel_values, image_sizes, positions):
        """phi:393-416. Sub-image order is the plain reshape of phi:404,406 (H4)."""
        V = 'model.vision_embed_tokens.'
        B = pixel_values.shape[0]
        sizes = (torch.as_tensor(image_sizes) // 336).tolist()
        positions = torch.as_tensor(positions).tolist()
        feats = self.clip(torch.as_tensor(pixel_values).reshape(-1, *pixel_values.shape[2:]))
        feats = feats.reshape(B, -1, *feats.shape[1:])
        C = feats.shape[-1]
        H = int(feats.shape[2] ** 0.5)
        sub_GN, glb_GN = _w(self.w[V + 'sub_GN']), _w(self.w[V + 'glb_GN'])
        outs, lens = [], []

        def merge(img, shape, tile):
            t = img.reshape(shape).permute(0, 1, 3, 2, 4, 5).reshape(tile)
            return torch.cat([t, sub_GN.expand(1, tile[1], 1, -1)], dim=2).reshape(1, -1, 4 * C)
        for b in range(B):
            h, w = sizes[b]
            n = h * w
            glb = merge(feats[b, :1], (1, H // 2, 2, H // 2, 2, C), (1, H // 2, H // 2, 4 * C))
            sub = merge(feats[b, 1:n + 1], (n, H // 2, 2, H // 2, 2, C), (1, h * 12, w * 12, 4 * C))
            x = torch.cat([sub, glb_GN, glb], dim=1)
            x = self.lin(x, V + 'img_projection.0', bias=True, prec=self._vprec())
            x = _r(F.gelu(x), self._vprec())                               # nn.GELU() exact erf
            x = self.lin(x, V + 'img_projection.2', bias=True, prec=self._vprec())
            outs.append(_r(x, self.prec))                                  # slice-assign into the bf16 text embeddings (phi:414)
            lens.append(int((h * w + 1) * 144 + 1 + (h + 1) * 12))
        idx = 0
        txt = txt.clone()
        for i, cnt in enumerate(lens):
            r, c = positions[idx]
            txt[r, c:c + cnt] = outs[i][0]
            idx += cnt
        return txt

    # -- model call protocol (phi:606, phi:576-592)
    def __call__(self, input_ids, pixel_values=None, image_sizes=None, positions=None, cache=None, pids=None,
                 mask=None, max_tokens=0, advance_offset=None, n_beam=1, last_only=False):
        ids = torch.as_tensor(input_ids).long()
        emb = _w(self.w['model.embed_tokens.weight'])
        x = emb[ids.clamp(min=0)]                                          # H3: negative ids are overwritten below
        if pixel_values is not None and self.is_vision:
            x = self.image_embed(x, pixel_values, image_sizes, positions)
        if cache is None:
            B, L = x.shape[:2]
            cache = [KVCache(self.cfg, B, L, max_tokens, self.prec) for _ in range(self.cfg.num_hidden_layers)]
            self._masker = Mask4D(L + max_tokens, mask)
            self._roper = SuRoPE(self.cfg, L + max_tokens, pids)
        past_L, new_L = cache[0].offset, x.shape[1]
        allow = self._masker(past_L, new_L)
        cos, sin = self._roper(past_L, new_L)
        for i in range(self.cfg.num_hidden_layers):
            p = f'model.layers.{i}.'
            r = self.attention(i, self.rms(x, self.w[p + 'input_layernorm.weight']), cache[i], cos, sin, allow, n_beam)
            h = _r(x + r, self.prec)
            r = self.mlp(i, self.rms(h, self.w[p + 'post_attention_layernorm.weight']))
            x = _r(h + r, self.prec)
        if advance_offset is not None:
            for c in cache:
                c.offset = past_L + advance_offset
        x = self.rms(x, self.w['model.norm.weight'])
        if last_only:
            x = x[:, -1:]
        logits = x @ _w(self.w['lm_head.weight']).T                        # logits kept fp32 for comparison
        return logits, cache
