"""Work that programs have this framework do, as cases to be timed and compared.

Seven kinds, each through a public entry point:
  attention   PagedLM.attend: the windowed / chunked / gated attention of the engine models over the shared page pool, prompt
              portions (prefill tiles) or single decoded tokens
  scan        p3_gla_scan, p3_delta_scan, p3_decay_scan, p3_matrix_memory_scan: the recurrent mixers, whole prompts or one token
  experts     PagedLM.experts: one mixture-of-experts layer behind its router
  linear      PagedLM.linear: one dense projection, bf16 serving mode or all-fp32 mode, from one row to a prompt
  step        Engine.step: prompts admitted, run through a whole (shallow) Tagenex model, logits read, requests ended
  phi         Phi3B200.__call__: prefill of a rectangular batch at Phi-3.5-mini's layer sizes, logits of the last token and the cache
  clip        Phi3B200.clip_features: the ViT-L/14-336 tower over image crops
Sizes are those of bench.py's workloads and tests, made ragged. `exact` restates every kind in 64-bit torch."""
import math

import numpy as np
import torch

import phi3_b200  # noqa: F401
from phi3_b200 import _lib, configs
from phi3_b200._lib import PAGE, call_struct, ptr
from phi3_b200.engine import Engine
from phi3_b200.lm_base import PagedLM, StepBatch
from phi3_b200.model import Phi3B200
from phi3_b200.tagenex import TagenexB200

DEV = 'cuda'
F32, B16, F64, I32 = torch.float32, torch.bfloat16, torch.float64, torch.int32
LIMIT = 7.0                                                        # clamp of the gated units, as in bench.py


def listed():
    return [
        # a batch of prompts in one engine step: grouped heads, window, sink, distance penalty, head gates
        dict(name='attention_prompts', kind='attention', style='penalty', n_seq=4, new=2048, past=0, heads=16, kv=4, dim=128, window=1024),
        # a ragged prompt portion of one request behind its cached part: as many K/V heads as query heads, element-wise gates
        dict(name='attention_portion', kind='attention', style='gated', n_seq=1, new=333, past=704, heads=32, kv=32, dim=96, window=0),
        # one decoded token of each of sixteen live requests at 2048 tokens of context
        dict(name='attention_decode', kind='attention', style='linear', n_seq=16, new=1, past=2047, heads=16, kv=4, dim=128, window=0),
        # the gated linear attention of a step of prompts
        dict(name='scan_prompts', kind='scan', mixer='gla', n_seq=4, tokens=2048, fresh=True, heads=8, kv=8, dim=128, vdim=256),
        # the gated delta rule at decode: one token of sixteen requests, states read and written
        dict(name='scan_decode', kind='scan', mixer='delta', n_seq=16, tokens=1, fresh=False, heads=8, kv=8, dim=128, vdim=256),
        # a mixture layer over a step of prompts
        dict(name='experts_prompts', kind='experts', tokens=4096, width=2048, ff=1408, experts=8, top=2),
        # the same layer at decode with four live requests: a stream of the chosen experts' matrices
        dict(name='experts_decode', kind='experts', tokens=4, width=2048, ff=1408, experts=8, top=2),
        # a projection in the all-fp32 mode
        dict(name='linear_fp32', kind='linear', dtype='f32', rows=512, n=3072, k=1024, bias=False),
        # a projection of a single-image prompt (781 rows), bf16, with bias
        dict(name='linear_bf16', kind='linear', dtype='bf16', rows=781, n=9216, k=3072, bias=True),
        # four ragged prompts through a two-layer model: one whole engine step
        dict(name='step_prompts', kind='step', n_seq=4, tokens=1500, width=2048, heads=16, kv=4, dim=128, ff=8192, window=1024, layers=2),
        # the prompt of a single-image question (781 tokens) through two layers of Phi-3.5-mini
        dict(name='phi_prefill', kind='phi', batch=1, tokens=781, layers=2),
        # the crops of one 672 x 672 image through four layers of the vision tower
        dict(name='clip_crops', kind='clip', crops=5, layers=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['prompts', 'prompts', 'decode', 'scan', 'scan_decode', 'experts', 'experts_decode', 'f32', 'bf16', 'step', 'phi', 'clip'])
    heads, kv, dim = rng.choice([(16, 4, 128), (8, 2, 128), (32, 32, 96), (32, 8, 96), (32, 8, 64), (16, 16, 64), (8, 8, 128)])
    style = rng.choice(['penalty', 'keep', 'sigmoid', 'chunk', 'linear', 'gated', 'latent'])
    if style == 'latent':
        heads, kv, dim = rng.choice([16, 32]), 1, 128
    window = rng.choice([256, 512, 1024])
    if kind == 'prompts':
        n_seq = rng.randint(1, 6)
        return dict(kind='attention', style=style, n_seq=n_seq, new=_log(rng, 40, 8192 // n_seq if n_seq > 2 else 3000),
                    past=rng.choice([0, 0, _log(rng, 10, 2000)]), heads=heads, kv=kv, dim=dim, window=window)
    if kind == 'decode':
        n_seq = _log(rng, 1, 40)
        return dict(kind='attention', style=style, n_seq=n_seq, new=1, past=_log(rng, 60, 6000), heads=heads, kv=kv, dim=dim, window=window)
    if kind in ('scan', 'scan_decode'):
        mixer = rng.choice(['gla', 'delta', 'decay', 'memory'])
        h, g, d, dv = rng.choice([(8, 8, 128, 256), (12, 12, 64, 256), (64, 8, 64, 128), (8, 4, 128, 128), (4, 4, 96, 200)])
        if mixer in ('gla', 'memory'):
            g = h
        one = kind == 'scan_decode'
        n_seq = _log(rng, 1, 40) if one else rng.randint(1, 6)
        return dict(kind='scan', mixer=mixer, n_seq=n_seq, tokens=1 if one else _log(rng, 20, 8192 // n_seq if n_seq > 3 else 2500),
                    fresh=False if one else rng.random() < 0.6, heads=h, kv=g, dim=d, vdim=dv)
    if kind in ('experts', 'experts_decode'):
        width, ff, experts, top = rng.choice([(2048, 1408, 8, 2), (3072, 1024, 16, 4), (3072, 2048, 8, 2), (1024, 1024, 8, 2)])
        return dict(kind='experts', tokens=_log(rng, 1, 40) if kind == 'experts_decode' else _log(rng, 64, 6000), width=width, ff=ff,
                    experts=experts, top=top)
    if kind == 'f32':
        return dict(kind='linear', dtype='f32', rows=_log(rng, 1, 1200), n=rng.choice([1024, 3072, 2048, 2056, 1601, 4096]),
                    k=rng.choice([512, 1024, 2048, 3072, 1000]), bias=rng.random() < 0.5)
    if kind == 'bf16':
        return dict(kind='linear', dtype='bf16', rows=_log(rng, 1, 6000), n=rng.choice([1024, 2048, 3072, 4224, 9216, 16384, 2056]),
                    k=rng.choice([1024, 1408, 2048, 3072, 8192]), bias=rng.random() < 0.5)
    if kind == 'step':
        width, h, g, d, ff = rng.choice([(2048, 16, 4, 128, 8192), (1024, 8, 2, 128, 4096), (3072, 32, 32, 96, 8192), (2048, 32, 8, 64, 4096)])
        n_seq = rng.randint(1, 5)
        return dict(kind='step', n_seq=n_seq, tokens=_log(rng, 20, min(1200, 3000 // n_seq)), width=width, heads=h, kv=g, dim=d, ff=ff, window=window, layers=2)
    if kind == 'phi':
        batch = rng.randint(1, 4)
        return dict(kind='phi', batch=batch, tokens=_log(rng, 24, min(1100, 2800 // batch)), layers=2)
    return dict(kind='clip', crops=rng.randint(1, 14), layers=rng.randint(3, 5))


# ---------------------------------------------------------------------------------------------------------------- inputs
class _Draw:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def n(self, *shape, scale=1.0, dtype=F32):
        return (torch.randn(shape, generator=self.g, device=DEV) * scale).to(dtype)

    def u(self, *shape, lo=0.0, hi=1.0, dtype=F32):
        return (torch.rand(shape, generator=self.g, device=DEV) * (hi - lo) + lo).to(dtype)

    def ints(self, hi, *shape, lo=0):
        return torch.randint(lo, hi, shape, generator=self.g, device=DEV, dtype=torch.int64)


def _lengths(n, longest):
    """tokens of every sequence of a ragged batch: the longest first, the others shorter by uneven amounts"""
    return [max(1, longest - (i * 97) % max(1, longest // 3)) if longest > 1 else 1 for i in range(n)]


def _rows_of(c):
    if c['kind'] == 'attention':
        return _lengths(c['n_seq'], c['new']), [max(0, c['past'] - 53 * i) if c['new'] == 1 else c['past'] for i in range(c['n_seq'])]
    return _lengths(c['n_seq'], c['tokens']), None


def _mask_of(c):
    """what limits the keys of a query: (window, keep_first, chunk)"""
    return {'penalty': (c['window'], 0, 0), 'keep': (c['window'], 64, 0), 'sigmoid': (c['window'], 0, 0), 'chunk': (0, 0, 2 * c['window']),
            'linear': (0, 0, 0), 'gated': (0, 0, 0), 'latent': (c['window'], 0, 0)}[c['style']]


def _attention_inputs(c, seed):
    g, H, G, d = _Draw(seed), c['heads'], c['kv'], c['dim']
    news, pasts = _rows_of(c)
    dv = 96 if c['style'] == 'latent' else d
    T = sum(news)
    x = dict(news=news, pasts=pasts, T=T, dv=dv, q=g.n(T, H, d, dtype=B16))
    x['k'] = [g.n(p + n, G, d, dtype=B16) for n, p in zip(news, pasts)]
    x['v'] = None if c['style'] == 'latent' else [g.n(p + n, G, dv, dtype=B16) for n, p in zip(news, pasts)]
    longest = max(n + p for n, p in zip(news, pasts))
    x['sink'] = g.n(H) if c['style'] in ('penalty', 'chunk', 'gated', 'latent') else torch.zeros(H, device=DEV) if c['style'] == 'linear' else None
    x['penalty'] = None
    if c['style'] == 'penalty':
        dist = torch.arange(min(longest, c['window']), device=DEV, dtype=F32)
        x['penalty'] = g.u(H, 1, lo=0.2, hi=1.2) * torch.log1p(g.u(H, 1, lo=0.05, hi=1.0) * dist)
    elif c['style'] == 'linear':
        slope = 2.0 ** (-8.0 * (torch.arange(H, device=DEV, dtype=F32) + 1) / H)
        x['penalty'] = slope[:, None] * torch.arange(longest, device=DEV, dtype=F32)
    x['gate'] = g.u(T, H) if c['style'] == 'penalty' else None
    x['elem'] = g.n(T, H * dv) if c['style'] in ('linear', 'gated') else None
    x['sig'] = g.n(H, scale=0.5) - 2.0 if c['style'] == 'sigmoid' else None
    n_pg = [-(-(n + p) // PAGE) for n, p in zip(news, pasts)]
    x['perm'] = torch.randperm(sum(n_pg), generator=g.g, device=DEV)
    x['n_pg'] = n_pg
    return x


def _scan_inputs(c, seed):
    g, H, G, d, dv = _Draw(seed), c['heads'], c['kv'], c['dim'], c['vdim']
    news, _ = _rows_of(c)
    T, m = sum(news), c['mixer']
    x = dict(news=news, T=T, v=g.n(T, H, dv), s0=g.n(c['n_seq'], H, d, dv, scale=0.3))
    x['q'], x['k'] = g.n(T, G, d), g.n(T, G, d)
    if m in ('delta', 'decay'):
        x['q'], x['k'] = x['q'] / x['q'].norm(dim=-1, keepdim=True), x['k'] / x['k'].norm(dim=-1, keepdim=True)
        x['decay'] = torch.exp(-g.u(H, lo=0.02, hi=0.5) * torch.nn.functional.softplus(g.n(T, H)))
        x['beta'] = torch.sigmoid(g.n(T, H)) if m == 'delta' else torch.nn.functional.softplus(g.n(T, H))
        x['skip'] = g.n(H) if m == 'decay' else None
    elif m == 'gla':
        x['rank'] = 16
        x['lr'], x['a2'], x['zb'] = g.n(T, 16, scale=0.5), g.n(H * d, 16, scale=0.5), g.n(H * d) + 2.0
    else:
        x['k'] = x['k'] * d ** -0.5
        x['i'], x['f'], x['ib'], x['fb'] = g.n(T, H), g.n(T, H), g.n(H, scale=0.2) - 1.0, g.u(H, lo=3.0, hi=6.0)
        x['n0'], x['m0'] = g.n(c['n_seq'], H, d, scale=0.3), g.n(c['n_seq'], H, scale=0.2)
    return x


def _experts_inputs(c, seed):
    g, E, W, F = _Draw(seed), c['experts'], c['width'], c['ff']
    z = g.n(c['tokens'], E) + 0.5 * g.n(E)                           # some experts are wanted more than others
    val, ids = torch.topk(z, c['top'], dim=-1)
    return dict(xa=g.n(c['tokens'], W, dtype=B16), ids=ids.to(I32).contiguous(), wts=torch.softmax(val, -1).contiguous(),
                gu=g.n(E, 2 * F, W, scale=W ** -0.5, dtype=B16), down=g.n(E, W, F, scale=F ** -0.5, dtype=B16))


def _linear_inputs(c, seed):
    g, dt = _Draw(seed), F32 if c['dtype'] == 'f32' else B16
    return dict(x=g.n(c['rows'], c['k'], dtype=dt), w=g.n(c['n'], c['k'], scale=c['k'] ** -0.5, dtype=dt),
                b16=g.n(c['n'], scale=0.3, dtype=B16) if c['bias'] else None)


STEP_VOCAB = 8192


def _step_config(c):
    att = {'type': 'attention', 'mixer': {'heads': c['heads'], 'kv_heads': c['kv'], 'dim': c['dim'], 'vdim': c['dim'], 'scale': c['dim'] ** -0.5,
                                          'v_mix': True, 'mask': {'size': c['window']}}}
    return {'architecture': 'Tagenex', 'vocab': STEP_VOCAB, 'width': c['width'], 'norm': {'eps': 1e-5},
            'layers': [dict(att, mlp={'kind': 'dense', 'ff': c['ff'], 'limit': LIMIT})] * c['layers']}


def _step_inputs(c, seed):
    g, W, H, G, d, F = _Draw(seed), c['width'], c['heads'], c['kv'], c['dim'], c['ff']
    mat = lambda n, k: g.n(n, k, scale=k ** -0.5, dtype=B16)
    w = {'embed': g.n(STEP_VOCAB, W, dtype=B16), 'head': mat(STEP_VOCAB, W), 'final.norm': (1 + g.n(W, scale=0.1)).to(B16)}
    for i in range(c['layers']):
        p = f'l{i}.'
        w.update({p + 'norm1': (0.5 + g.n(W, scale=0.1)).to(B16), p + 'norm2': (0.5 + g.n(W, scale=0.1)).to(B16), p + 'mix.q': mat(H * d, W),
                  p + 'mix.k': mat(G * d, W), p + 'mix.v': mat(G * d, W), p + 'mix.g': mat(H, W), p + 'mix.o': mat(W, H * d),
                  p + 'mix.q.norm': (1 + g.n(d, scale=0.1)).to(B16), p + 'mix.k.norm': (1 + g.n(d, scale=0.1)).to(B16),
                  p + 'mix.vmix': torch.tensor(0.375, dtype=B16, device=DEV), p + 'mix.r1': g.u(H, lo=0.2, hi=1.2, dtype=B16),
                  p + 'mix.r2': g.u(H, lo=0.05, hi=1.0, dtype=B16), p + 'mix.sink': g.n(H, dtype=B16), p + 'mlp.gate': mat(F, W),
                  p + 'mlp.gate.b': g.n(F, scale=0.3, dtype=B16), p + 'mlp.up': mat(F, W), p + 'mlp.up.b': g.n(F, scale=0.3, dtype=B16),
                  p + 'mlp.down': mat(W, F), p + 'mlp.down.b': g.n(W, scale=0.3, dtype=B16)})
    news, _ = _rows_of(c)
    toks = [g.ints(STEP_VOCAB, n).tolist() for n in news]
    return dict(w=w, toks=toks, wanted=[sorted({n // 2, n - 1}) for n in news])


def _phi_config(c):
    return configs.with_overrides(configs.PHI35_MINI, num_hidden_layers=c['layers'])


def _phi_inputs(c, seed):
    g, cfg = _Draw(seed), _phi_config(c)
    H, I, V = cfg.hidden_size, cfg.intermediate_size, cfg.vocab_size
    res = 0.02 / math.sqrt(2 * c['layers'])
    w = {'model.embed_tokens.weight': g.n(V, H, dtype=B16), 'lm_head.weight': g.n(V, H, scale=0.02, dtype=B16),
         'model.norm.weight': (1 + g.n(H, scale=0.1)).to(B16)}
    for i in range(c['layers']):
        p = f'model.layers.{i}.'
        w.update({p + 'input_layernorm.weight': (1 + g.n(H, scale=0.1)).to(B16), p + 'self_attn.qkv_proj.weight': g.n(3 * H, H, scale=0.02, dtype=B16),
                  p + 'self_attn.o_proj.weight': g.n(H, H, scale=res, dtype=B16), p + 'post_attention_layernorm.weight': (1 + g.n(H, scale=0.1)).to(B16),
                  p + 'mlp.gate_up_proj.weight': g.n(2 * I, H, scale=0.02, dtype=B16), p + 'mlp.down_proj.weight': g.n(H, I, scale=res, dtype=B16)})
    return dict(w=w, ids=g.ints(32000, c['batch'], c['tokens'], lo=3))


def _clip_configs(c):
    clip = configs.tiny_clip(layers=c['layers'] + 1)                 # the tower runs all layers but the last
    return configs.tiny(vision=True, layers=1, vocab_size=256), clip


def _clip_inputs(c, seed):
    g, (cfg, cc) = _Draw(seed), _clip_configs(c)
    H, I, V, D, F = cfg.hidden_size, cfg.intermediate_size, cfg.vocab_size, cc.hidden_size, cc.intermediate_size
    lin, one = lambda *s: g.n(*s, scale=0.02, dtype=B16), lambda n: (1 + g.n(n, scale=0.1)).to(B16)
    b = lambda *s: g.n(*s, scale=0.1, dtype=B16)
    w = {'model.embed_tokens.weight': g.n(V, H, dtype=B16), 'lm_head.weight': lin(V, H), 'model.norm.weight': one(H)}
    p = 'model.layers.0.'
    w.update({p + 'input_layernorm.weight': one(H), p + 'self_attn.qkv_proj.weight': lin(3 * H, H), p + 'self_attn.o_proj.weight': lin(H, H),
              p + 'post_attention_layernorm.weight': one(H), p + 'mlp.gate_up_proj.weight': lin(2 * I, H), p + 'mlp.down_proj.weight': lin(H, I)})
    P = 'model.vision_embed_tokens.img_processor.vision_model.'
    w.update({P + 'embeddings.class_embedding': b(D), P + 'embeddings.patch_embedding.weight': lin(D, 14, 14, 3),
              P + 'embeddings.position_embedding.weight': b(577, D), P + 'pre_layrnorm.weight': one(D), P + 'pre_layrnorm.bias': b(D)})
    for j in range(cc.num_hidden_layers):
        L = P + f'encoder.layers.{j}.'
        for n in ('q_proj', 'k_proj', 'v_proj', 'out_proj'):
            w.update({L + f'self_attn.{n}.weight': lin(D, D), L + f'self_attn.{n}.bias': b(D)})
        w.update({L + 'layer_norm1.weight': one(D), L + 'layer_norm1.bias': b(D), L + 'layer_norm2.weight': one(D), L + 'layer_norm2.bias': b(D),
                  L + 'mlp.fc1.weight': lin(F, D), L + 'mlp.fc1.bias': b(F), L + 'mlp.fc2.weight': lin(D, F), L + 'mlp.fc2.bias': b(D)})
    q = 'model.vision_embed_tokens.'
    w.update({q + 'glb_GN': g.n(1, 1, 4 * D, dtype=B16), q + 'sub_GN': g.n(1, 1, 1, 4 * D, dtype=B16), q + 'img_projection.0.weight': lin(H, 4 * D),
              q + 'img_projection.0.bias': b(H), q + 'img_projection.2.weight': lin(H, H), q + 'img_projection.2.bias': b(H)})
    return dict(w=w, px=g.n(c['crops'], 3, 336, 336))


# ---------------------------------------------------------------------------------------------------------------- preparing
class _Layer(PagedLM):
    """a design of one's own on the engine models' base class: its products, attention launches and expert layers"""

    def __init__(self, width, dtype=B16):
        self.dev, self.dtype, self.W, self.eps = torch.device(DEV), dtype, width, 1e-5
        self._init_products()


def _prepare_attention(c, seed):
    x, H, G, d = _attention_inputs(c, seed), c['heads'], c['kv'], c['dim']
    dv, latent, layer = x['dv'], c['style'] == 'latent', _Layer(c['heads'] * c['dim'])
    n_pages = sum(x['n_pg'])
    kp = torch.zeros(n_pages, G, PAGE, d, dtype=B16, device=DEV)
    vp = kp if latent else torch.zeros(n_pages, G, PAGE, dv, dtype=B16, device=DEV)
    bt = torch.zeros(c['n_seq'], max(x['n_pg']), dtype=I32, device=DEV)
    at = 0
    for s, n in enumerate(x['n_pg']):
        pages = x['perm'][at:at + n]
        bt[s, :n] = pages.to(I32)
        for pool, rows in ((kp, x['k'][s]),) if latent else ((kp, x['k'][s]), (vp, x['v'][s])):
            full = torch.zeros(n * PAGE, *rows.shape[1:], dtype=B16, device=DEV)
            full[:rows.shape[0]] = rows
            pool[pages] = full.view(n, PAGE, G, -1).transpose(1, 2)
        at += n
    v_ld = d if latent else 0
    rows = layer.attention_tile_rows(H, G, d, dv, v_ld)
    b, tiles, r0 = StepBatch(), [], 0
    for s, (n, p) in enumerate(zip(x['news'], x['pasts'])):
        tiles += [(r0 + i, min(rows, n - i), s, p + i) for i in range(0, n, rows)] if n > 1 else [(r0, 1, s, p)]
        r0 += n
    td = torch.tensor(tiles, dtype=I32, device=DEV).reshape(-1)
    b.T, one = x['T'], c['new'] == 1
    b.n_pf, b.pf_tiles, b.n_dec, b.dec_tiles = (0, None, len(tiles), td) if one else (len(tiles), td, 0, None)
    b.max_pos = max(n + p for n, p in zip(x['news'], x['pasts'])) - 1
    q, out = x['q'].reshape(x['T'], H * d).contiguous(), torch.empty(x['T'], H * dv, dtype=B16, device=DEV)
    window, keep, chunk = _mask_of(c)
    w = _lib.AttnWindowArgs()
    w.q, w.ld_q, w.k_pool, w.v_pool, w.block_table, w.bt_stride = ptr(q), H * d, ptr(kp), ptr(vp), ptr(bt), bt.stride(0)
    w.sink, w.penalty, w.n_penalty = ptr(x['sink']), ptr(x['penalty']), 0 if x['penalty'] is None else x['penalty'].shape[1]
    w.gate, w.out, w.ld_out, w.v_ld = ptr(x['gate']), ptr(out), H * dv, v_ld
    w.n_heads, w.n_kv, w.dim, w.vdim, w.scale, w.window, w.keep_first, w.chunk = H, G, d, dv, d ** -0.5, window, keep, chunk
    w.sig_bias, w.elem_gate, w.ld_elem_gate = ptr(x['sig']), ptr(x['elem']), H * dv
    span = lambda n: min([n] + ([window + keep] if window else []) + ([chunk] if chunk else []))
    keep_alive = (x['sink'], x['penalty'], x['gate'], x['sig'], x['elem'], q, kp, vp, bt, td)
    return dict(layer=layer, w=w, rows=rows, b=b, G=G, key=d, val=dv, span=span, kv_bytes=G * (d + (0 if latent else dv)), out=out, alive=keep_alive)


def _prepare_scan(c, seed):
    x, H, G, d, dv, m = _scan_inputs(c, seed), c['heads'], c['kv'], c['dim'], c['vdim'], c['mixer']
    T, r0, recs = x['T'], 0, []
    for s, n in enumerate(x['news']):
        recs.append((r0, n, s, 0 if c['fresh'] else 100))
        r0 += n
    seqs = torch.tensor(recs, dtype=I32, device=DEV).reshape(-1)
    cols = [x['q'].reshape(T, -1), x['k'].reshape(T, -1), x['v'].reshape(T, -1)]
    if m == 'memory':
        cols += [x['i'], x['f']]
    proj = torch.cat(cols, 1).contiguous()
    ld, ko, vo = proj.shape[1], G * d, 2 * G * d
    out = torch.empty(T, H * dv, device=DEV)
    st = dict(mixer=m, out=out, extra=None, alive=[proj, seqs])
    if m == 'memory':
        parts = [x['s0'].reshape(c['n_seq'], H, d * dv), x['n0'], x['m0'][..., None].expand(-1, -1, -(-dv // 32))]
        st['state'] = torch.cat(parts, -1).contiguous()
        a, st['extra'] = _lib.MatrixMemoryArgs(), torch.empty(T, H, device=DEV)
        a.proj, a.ld_proj, a.q_off, a.k_off, a.v_off, a.i_off, a.f_off = ptr(proj), ld, 0, ko, vo, vo + H * dv, vo + H * dv + H
        a.i_bias, a.f_bias, a.q_scale, a.gate_cap, a.den = ptr(x['ib']), ptr(x['fb']), d ** -0.5, 15.0, ptr(st['extra'])
        st['alive'] += [x['ib'], x['fb']]
    elif m == 'gla':
        st['state'], z = x['s0'].contiguous(), torch.empty(T, H * d, device=DEV)
        a = _lib.GlaArgs()
        a.proj, a.ld_proj, a.q_off, a.k_off, a.v_off, a.z, a.ld_z, a.z_bias = ptr(proj), ld, 0, ko, vo, ptr(z), H * d, ptr(x['zb'])
        a.inv_tau, a.q_scale, a.n_rows, a.lr, a.ld_lr, a.a2, a.rank = 1.0 / 16, d ** -0.5, T, ptr(x['lr']), 16, ptr(x['a2']), 16
        st['alive'] += [z, x['lr'], x['a2'], x['zb']]
    else:
        st['state'], gates = x['s0'].contiguous(), torch.stack([x['decay'], x['beta']], -1).contiguous()
        a = _lib.DeltaScanArgs()
        a.qkv, a.ld_qkv, a.q_off, a.k_off, a.v_off, a.gates, a.n_kv, a.skip = ptr(proj), ld, 0, ko, vo, ptr(gates), G, ptr(x['skip'])
        st['alive'] += [gates, x['skip']]
    a.n_heads, a.dim, a.vdim, a.state, a.seqs, a.n_seqs, a.out, a.ld_out = H, d, dv, ptr(st['state']), ptr(seqs), c['n_seq'], ptr(out), H * dv
    st.update(args=a, entry={'gla': 'p3_gla_scan', 'delta': 'p3_delta_scan', 'decay': 'p3_decay_scan', 'memory': 'p3_matrix_memory_scan'}[m])
    return st


class _Unit:
    """sizes of a mixture layer, as the engine models' configurations hold them"""

    def __init__(self, ff, experts, top):
        self.ff, self.experts, self.top = ff, experts, top


def prepare(c, seed):
    kind = c['kind']
    if kind == 'attention':
        return dict(_prepare_attention(c, seed), kind=kind)
    if kind == 'scan':
        return dict(_prepare_scan(c, seed), kind=kind)
    if kind == 'experts':
        x, layer = _experts_inputs(c, seed), _Layer(c['width'])
        F = c['ff']
        glu = lambda gu, hid, n: _lib.call('p3_glu_clamped', ptr(gu), gu.stride(0), ptr(hid), hid.stride(0), 0, n, F, LIMIT, 1.702, None,
                                           torch.cuda.current_stream().cuda_stream)
        return dict(kind=kind, layer=layer, x=x, unit=_Unit(F, c['experts'], c['top']), glu=glu, y=torch.empty(c['tokens'], c['width'], device=DEV))
    if kind == 'linear':
        x, layer = _linear_inputs(c, seed), _Layer(c['k'], F32 if c['dtype'] == 'f32' else B16)
        x['b32'] = None if x['b16'] is None else x['b16'].to(F32)
        return dict(kind=kind, layer=layer, x=x, out=torch.empty(c['rows'], c['n'], device=DEV))
    if kind == 'step':
        x = _step_inputs(c, seed)
        model = TagenexB200(_step_config(c), x['w'], device=DEV)
        eng = Engine(model, max_tokens=sum(-(-len(t) // PAGE) * PAGE for t in x['toks']), n_slots=c['n_seq'])
        entries = [(i, t, want) for i, (t, want) in enumerate(zip(x['toks'], x['wanted']))]
        return dict(kind=kind, engine=eng, entries=entries, ends=list(range(c['n_seq'])))
    if kind == 'phi':
        x = _phi_inputs(c, seed)
        return dict(kind=kind, model=Phi3B200(_phi_config(c), x['w'], device=DEV), ids=x['ids'])
    x, (cfg, clip) = _clip_inputs(c, seed), _clip_configs(c)
    return dict(kind=kind, model=Phi3B200(cfg, x['w'], device=DEV, clip_cfg=clip), px=x['px'])


def run(s):
    kind = s['kind']
    if kind == 'attention':
        s['layer'].attend(s['w'], s['rows'], s['b'], s['G'], s['key'], s['val'], s['span'], s['kv_bytes'])
        return s['out']
    if kind == 'scan':
        call_struct(s['entry'], s['args'], torch.cuda.current_stream().cuda_stream)
        return [s['out'], s['state']] + ([] if s['extra'] is None else [s['extra']])
    if kind == 'experts':
        x = s['x']
        s['layer'].experts(x['gu'], x['down'], s['unit'], x['xa'], s['y'], x['xa'].shape[0], x['ids'], x['wts'], s['glu'])
        return s['y']
    if kind == 'linear':
        x = s['x']
        left = s['layer'].linear(x['x'], x['w'], s['out'], x['b32'], x['b16'])
        return s['out'] if left is None else [s['out'], left]        # the weight stream of small batches leaves the bias to its consumer
    if kind == 'step':
        return s['engine'].step(s['entries'], end=s['ends'])
    if kind == 'phi':
        logits, cache = s['model'](s['ids'], max_tokens=32, logits_rows='last')
        return [logits, cache.pool]
    return s['model'].clip_features(s['px'])


# ---------------------------------------------------------------------------------------------------------------- accounting
def _pairs(c):
    """(query, key) pairs that are visible, and keys that any query sees"""
    news, pasts = _rows_of(c)
    window, keep, chunk = _mask_of(c)
    pairs = keys = 0
    for n, p in zip(news, pasts):
        i = np.arange(p, p + n)
        lo = np.zeros(n, np.int64)
        if window:
            lo = np.maximum(lo, i - window + 1)
        if chunk:
            lo = np.maximum(lo, i - i % chunk)
        kept = np.minimum(keep, lo)
        pairs += int((i - lo + 1 + kept).sum())
        keys += int(p + n - lo[0] + kept[0])
    return pairs, keys


def work(c):
    k = c['kind']
    if k == 'attention':
        H, G, d = c['heads'], c['kv'], c['dim']
        pairs, keys = _pairs(c)
        T, latent = sum(_rows_of(c)[0]), c['style'] == 'latent'
        dv = 96 if latent else d
        extra = 4 * T * H * dv if c['style'] in ('linear', 'gated') else 0
        return dict(flops=2 * pairs * H * (d + dv), bytes=2 * (T * H * (d + dv) + keys * G * (d + (0 if latent else dv))) + extra)
    if k == 'scan':
        H, G, d, dv, T = c['heads'], c['kv'], c['dim'], c['vdim'], sum(_rows_of(c)[0])
        state = 4 * c['n_seq'] * H * d * dv * (1 if c['fresh'] else 2)
        return dict(flops=T * H * d * dv * (7 if c['mixer'] == 'delta' else 5), bytes=4 * T * (2 * G * d + 2 * H * dv + 2 * H) + state)
    if k == 'experts':
        n, W, F = c['tokens'] * c['top'], c['width'], c['ff']
        return dict(flops=6 * n * W * F, bytes=2 * 3 * W * F * min(c['experts'], n) + c['tokens'] * W * 6)
    if k == 'linear':
        M, N, K, e = c['rows'], c['n'], c['k'], 4 if c['dtype'] == 'f32' else 2
        return dict(flops=2 * M * N * K, bytes=e * (M * K + N * K) + 4 * M * N)
    if k == 'step':
        W, H, G, d, F = c['width'], c['heads'], c['kv'], c['dim'], c['ff']
        T = sum(_rows_of(c)[0])
        per = W * (2 * H * d + 2 * G * d + H) + 3 * W * F
        pairs = sum(min(i + 1, c['window']) for n in _rows_of(c)[0] for i in range(n))
        return dict(flops=c['layers'] * (2 * T * per + 4 * pairs * H * d) + 4 * c['n_seq'] * STEP_VOCAB * W,
                    bytes=2 * (c['layers'] * per + STEP_VOCAB * W) + 2 * T * W)
    if k == 'phi':
        cfg = configs.PHI35_MINI
        H, I, V, T = cfg.hidden_size, cfg.intermediate_size, cfg.vocab_size, c['batch'] * c['tokens']
        per = 4 * H * H + 3 * H * I
        return dict(flops=c['layers'] * (2 * T * per + 2 * T * (c['tokens'] + 1) * H) + 2 * c['batch'] * V * H,
                    bytes=2 * (c['layers'] * (per + 2 * T * H) + V * H + T * H) + 4 * c['batch'] * V)
    T, D, F = c['crops'] * 577, 1024, 4096
    per = 4 * D * D + 2 * D * F
    return dict(flops=c['layers'] * (2 * T * per + 4 * T * 577 * D) + 2 * T * 588 * D, bytes=2 * c['layers'] * per + 4 * (T * D + c['crops'] * 3 * 336 * 336))


def tolerance(c):
    """What the data types give: softmax weights and outputs rounded to bf16, products whose operands pass a bf16 rounding on the way, or
    fp32 arithmetic throughout."""
    k = c['kind']                                                    # about four times the distance from `exact` that was measured:
    if k == 'attention':
        return {'rel': 0.009, 'max': 0.1}                            # 1.9e-3 .. 2.2e-3
    if k == 'scan':
        return {'rel': 1.2e-5, 'max': 3e-4}                          # up to 3.1e-6 after 2048 tokens
    if k == 'experts':
        return {'rel': 0.007, 'max': 0.08}                           # 1.7e-3
    if k == 'linear':
        return {'rel': 1.2e-5 if c['dtype'] == 'bf16' else 3e-6, 'max': 2e-4}    # 3.1e-6 on the tensor cores, 5.7e-7 .. 7.8e-7 in fp32
    if k == 'step':
        return {'rel': 0.012, 'max': 0.15}                           # 2.9e-3
    if k == 'phi':
        return {'rel': 0.023, 'max': 0.3}                            # 5.8e-3
    return {'rel': 0.01, 'max': 0.1}                                 # 2.4e-3


# ---------------------------------------------------------------------------------------------------------------- 64-bit restatement
def _attend64(q, k, v, pos, mask, scale, penalty, sink, sig):
    """q [n, H, d] at positions pos .., k / v [S, G, *] -> [n, H, dv], in blocks of rows"""
    n, H, _ = q.shape
    S, G, _ = k.shape
    window, keep, chunk = mask
    kh, vh = (t.double().repeat_interleave(H // G, 1).transpose(0, 1) for t in (k, v))
    j, out = torch.arange(S, device=DEV), []
    for r in range(0, n, 512):
        i = pos + torch.arange(r, min(n, r + 512), device=DEV)
        dist = i[:, None] - j[None]
        far = torch.zeros_like(dist, dtype=torch.bool)
        if window:
            far |= dist >= window
        if chunk:
            far |= (i[:, None] // chunk) != (j[None] // chunk)
        ok = (dist >= 0) & (~far | (j[None] < keep))
        s = q[r:r + 512].double().transpose(0, 1) @ kh.transpose(1, 2) * scale
        if penalty is not None:
            s = s - penalty.double()[:, dist.clamp(0, penalty.shape[1] - 1)]
        if sig is not None:
            a = torch.sigmoid(s + sig.double()[:, None, None]).masked_fill(~ok, 0.0)
        else:
            s = s.masked_fill(~ok, -math.inf)
            m = s.amax(-1, keepdim=True)
            if sink is not None:
                m = torch.maximum(m, sink.double()[:, None, None])
            e = torch.exp(s - m)
            a = e / (e.sum(-1, keepdim=True) + (0.0 if sink is None else torch.exp(sink.double()[:, None, None] - m)))
        out.append((a @ vh).transpose(0, 1))
    return torch.cat(out)


def _exact_attention(c, seed):
    x, H, outs, r = _attention_inputs(c, seed), c['heads'], [], 0
    for s, (n, p) in enumerate(zip(x['news'], x['pasts'])):
        k = x['k'][s]
        v = k[..., :x['dv']] if x['v'] is None else x['v'][s]
        outs.append(_attend64(x['q'][r:r + n], k, v, p, _mask_of(c), c['dim'] ** -0.5, x['penalty'], x['sink'], x['sig']))
        r += n
    y = torch.cat(outs)
    if x['gate'] is not None:
        y = y * x['gate'].double()[:, :, None]
    y = y.reshape(x['T'], H * x['dv'])
    return y if x['elem'] is None else y * torch.sigmoid(x['elem'].double())


def _exact_scan(c, seed):
    x, H, G, d, dv, m = _scan_inputs(c, seed), c['heads'], c['kv'], c['dim'], c['vdim'], c['mixer']
    rep = H // G
    q, k, v = x['q'].double().repeat_interleave(rep, 1), x['k'].double().repeat_interleave(rep, 1), x['v'].double()
    out, den, states, r = torch.empty(x['T'], H, dv, dtype=F64, device=DEV), None, [], 0
    if m == 'gla':
        z = x['zb'].double() + x['lr'].double() @ x['a2'].double().T
        al = torch.exp(torch.nn.functional.logsigmoid(z) / 16).view(-1, H, d)
    elif m == 'memory':
        cap = lambda t: 15.0 * torch.tanh(t / 15.0)
        ai, bf = cap(x['i'].double() + x['ib'].double()), torch.nn.functional.logsigmoid(cap(x['f'].double() + x['fb'].double()))
        den = torch.empty(x['T'], H, dtype=F64, device=DEV)
    else:
        keep, beta = x['decay'].double(), x['beta'].double()
    for s, n in enumerate(x['news']):
        S = x['s0'][s].double() * (0.0 if c['fresh'] else 1.0)
        if m == 'memory':
            nn, mm = x['n0'][s].double() * (0.0 if c['fresh'] else 1.0), x['m0'][s].double() * (0.0 if c['fresh'] else 1.0)
        for t in range(r, r + n):
            if m == 'gla':
                S = al[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
            elif m == 'delta':
                S = keep[t][:, None, None] * S
                u = beta[t][:, None] * (v[t] - torch.einsum('hdv,hd->hv', S, k[t]))
                S = S + k[t][:, :, None] * u[:, None]
            elif m == 'decay':
                S = keep[t][:, None, None] * S + (beta[t][:, None] * k[t])[:, :, None] * v[t][:, None]
            else:
                m1 = torch.maximum(bf[t] + mm, ai[t])
                f, i = torch.exp(bf[t] + mm - m1), torch.exp(ai[t] - m1)
                S = f[:, None, None] * S + (i[:, None] * k[t])[:, :, None] * v[t][:, None]
                nn, mm = f[:, None] * nn + i[:, None] * k[t], m1
                den[t] = torch.maximum(((nn * q[t]).sum(-1) * d ** -0.5).abs(), torch.exp(-mm)) + 1e-6
            out[t] = (q[t][:, None] @ S)[:, 0]
        r += n
        states.append(S.reshape(H, -1) if m != 'memory' else torch.cat([S.reshape(H, -1), nn, mm[:, None].expand(-1, -(-dv // 32))], 1))
    if m in ('gla', 'memory'):
        out = out * d ** -0.5
    elif m == 'decay':
        out = out + x['skip'].double()[:, None] * v
    state = torch.stack(states) if m == 'memory' else torch.stack(states).view(c['n_seq'], H, d, dv)
    return [out.reshape(x['T'], H * dv), state] + ([] if den is None else [den])


def _glu64(g, u):
    g, u = g.clamp(max=LIMIT), u.clamp(-LIMIT, LIMIT)
    return g * torch.sigmoid(1.702 * g) * (u + 1)


def _exact_experts(c, seed):
    x, F = _experts_inputs(c, seed), c['ff']
    y = torch.zeros(c['tokens'], c['width'], dtype=F64, device=DEV)
    for e in range(c['experts']):
        t, j = torch.nonzero(x['ids'] == e, as_tuple=True)
        if t.numel():
            h = x['xa'][t].double() @ x['gu'][e].double().T
            y.index_add_(0, t, x['wts'][t, j].double()[:, None] * (_glu64(h[:, :F], h[:, F:]) @ x['down'][e].double().T))
    return y


def _exact_linear(c, seed):
    x = _linear_inputs(c, seed)
    y = x['x'].double() @ x['w'].double().T
    if x['b16'] is None:
        return y
    if c['dtype'] == 'bf16' and c['rows'] <= 16 and c['k'] % 64 == 0 and c['n'] % 16 == 0:
        return [y, x['b16'].double()]                                # the bias is left to the consumer
    return y + x['b16'].double()


def _rms64(x, g, eps=1e-5):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * g


def _exact_step(c, seed):
    x, H, G, d, F = _step_inputs(c, seed), c['heads'], c['kv'], c['dim'], c['ff']
    w = {n: t.double() for n, t in x['w'].items()}
    rows = []
    for toks, want in zip(x['toks'], x['wanted']):
        h, first, n = w['embed'][torch.tensor(toks, device=DEV)], None, len(toks)
        dist = torch.arange(n, device=DEV, dtype=F64)
        for i in range(c['layers']):
            p = f'l{i}.mix.'
            q = _rms64((h @ w[p + 'q'].T).view(n, H, d), w[p + 'q.norm'])
            k = _rms64((h @ w[p + 'k'].T).view(n, G, d), w[p + 'k.norm'])
            v = (h @ w[p + 'v'].T).view(n, G, d)
            first, v = (v, v) if first is None else (first, (1 - w[p + 'vmix']) * v + w[p + 'vmix'] * first)
            pen = w[p + 'r1'][:, None] * torch.log1p(w[p + 'r2'][:, None] * dist)
            y = _attend64(q, k, v, 0, (c['window'], 0, 0), d ** -0.5, pen, w[p + 'sink'], None)
            y = (y * torch.sigmoid(h @ w[p + 'g'].T)[:, :, None]).reshape(n, H * d) @ w[p + 'o'].T
            h = h + _rms64(y, w[f'l{i}.norm1'])
            p = f'l{i}.mlp.'
            y = _glu64(h @ w[p + 'gate'].T + w[p + 'gate.b'], h @ w[p + 'up'].T + w[p + 'up.b']) @ w[p + 'down'].T + w[p + 'down.b']
            h = h + _rms64(y, w[f'l{i}.norm2'])
        rows.append(_rms64(h[want], w['final.norm']) @ w['head'].T)
    return torch.cat(rows)


def _exact_phi(c, seed):
    x, cfg = _phi_inputs(c, seed), _phi_config(c)
    B, L, H = c['batch'], c['tokens'], cfg.hidden_size
    nh, hd = cfg.num_attention_heads, H // cfg.num_attention_heads
    w = x['w']
    ratio = cfg.max_position_embeddings / cfg.original_max_position_embeddings
    mag = math.sqrt(1 + math.log(ratio) / math.log(cfg.original_max_position_embeddings))
    inv = 1.0 / (torch.tensor(cfg.rope_scaling['short_factor'], dtype=F64, device=DEV) * cfg.rope_theta ** (torch.arange(0, hd, 2, device=DEV, dtype=F64) / hd))
    ang = torch.arange(L, device=DEV, dtype=F64)[:, None] * inv
    cos, sin = (torch.cat([t, t], -1)[:, None] * mag for t in (ang.cos(), ang.sin()))
    turn = lambda t: t * cos + torch.cat([-t[..., hd // 2:], t[..., :hd // 2]], -1) * sin
    pages = -(-(L + 32) // PAGE)
    pool = torch.zeros(c['layers'], B * pages, 2, nh, PAGE, hd, dtype=F64, device=DEV)
    h = w['model.embed_tokens.weight'][x['ids']].double()
    for i in range(c['layers']):
        p = f'model.layers.{i}.'
        a = _rms64(h, w[p + 'input_layernorm.weight'].double()) @ w[p + 'self_attn.qkv_proj.weight'].double().T
        q, k, v = (t.reshape(B, L, nh, hd) for t in a.split(H, -1))
        q, k = turn(q), turn(k)
        for n, t in enumerate((k, v)):
            full = torch.zeros(B, pages * PAGE, nh, hd, dtype=F64, device=DEV)
            full[:, :L] = t
            pool[i, :, n] = full.view(B * pages, PAGE, nh, hd).transpose(1, 2)
        y = torch.stack([_attend64(q[b], k[b], v[b], 0, (0, 0, 0), hd ** -0.5, None, None, None) for b in range(B)])
        h = h + y.reshape(B, L, H) @ w[p + 'self_attn.o_proj.weight'].double().T
        g, u = (_rms64(h, w[p + 'post_attention_layernorm.weight'].double()) @ w[p + 'mlp.gate_up_proj.weight'].double().T).chunk(2, -1)
        h = h + (torch.nn.functional.silu(g) * u) @ w[p + 'mlp.down_proj.weight'].double().T
    return [_rms64(h[:, -1:], w['model.norm.weight'].double()) @ w['lm_head.weight'].double().T, pool]


def _exact_clip(c, seed):
    x, (_, cc) = _clip_inputs(c, seed), _clip_configs(c)
    w, P = {n: t.double() for n, t in x['w'].items()}, 'model.vision_embed_tokens.img_processor.vision_model.'
    N, D, nh = c['crops'], cc.hidden_size, cc.num_attention_heads
    ln = lambda t, n: torch.nn.functional.layer_norm(t, (D,), w[n + '.weight'], w[n + '.bias'], 1e-5)
    px = x['px'].double().unfold(2, 14, 14).unfold(3, 14, 14).permute(0, 2, 3, 4, 5, 1).reshape(N, 576, 14 * 14 * 3)
    h = px @ w[P + 'embeddings.patch_embedding.weight'].reshape(D, -1).T
    h = torch.cat([w[P + 'embeddings.class_embedding'].expand(N, 1, D), h], 1) + w[P + 'embeddings.position_embedding.weight']
    h = ln(h, P + 'pre_layrnorm')
    for j in range(c['layers']):
        L = P + f'encoder.layers.{j}.'
        lin = lambda t, n: t @ w[L + n + '.weight'].T + w[L + n + '.bias']
        a = ln(h, L + 'layer_norm1')
        q, k, v = (lin(a, f'self_attn.{n}_proj').view(N, 577, nh, D // nh).transpose(1, 2) for n in 'qkv')
        a = (torch.softmax(q @ k.transpose(2, 3) * (D // nh) ** -0.5, -1) @ v).transpose(1, 2).reshape(N, 577, D)
        h = h + lin(a, 'self_attn.out_proj')
        a = lin(ln(h, L + 'layer_norm2'), 'mlp.fc1')
        h = h + lin(a * torch.sigmoid(1.702 * a), 'mlp.fc2')
    return h.reshape(N * 577, D)


def exact(c, seed):
    return {'attention': _exact_attention, 'scan': _exact_scan, 'experts': _exact_experts, 'linear': _exact_linear, 'step': _exact_step,
            'phi': _exact_phi, 'clip': _exact_clip}[c['kind']](c, seed)
