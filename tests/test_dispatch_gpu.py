"""Kernels behind a dispatch by size, at the sizes where each can go wrong: edges of tiles, remainders, the smallest and the largest of
its range. Needs the built library and a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F32, B16 = torch.float32, torch.bfloat16


@pytest.fixture(scope='module')
def dev():
    if not torch.cuda.is_available():
        pytest.skip('needs a GPU')
    import phi3_b200  # noqa: F401
    return torch.device('cuda')


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _gemm_any(x, w, bias=None, rows=None, seg=None, gate=None, out_dtype=F32, batch=None, N=None, K=None):
    from phi3_b200 import _lib
    M, n = (rows.numel() if rows is not None else x.shape[0]), (w.shape[-2] if N is None else N)
    out = torch.full((M, n * (batch[0] if batch else 1)), float('nan'), dtype=out_dtype, device=x.device)
    a = _lib.GemmAnyArgs()
    a.X, a.ldx, a.x_f32, a.x_rows, a.x_row_div = x.data_ptr(), x.stride(0), int(x.dtype == F32), _lib.ptr(rows), 1
    a.W, a.ldw, a.w_f32, a.w_group_stride = w.data_ptr(), w.stride(-2), int(w.dtype == F32), w.stride(0) if w.dim() == 3 and seg is not None else 0
    a.bias, a.out, a.ldo, a.out_f32, a.M, a.N, a.K = _lib.ptr(bias), out.data_ptr(), out.stride(0), int(out_dtype == F32), M, n, w.shape[-1] if K is None else K
    a.seg_offsets, a.n_groups = _lib.ptr(seg), 0 if seg is None else seg.numel() - 1
    if batch:
        a.n_batch, a.x_batch_stride, a.w_batch_stride, a.out_batch_stride = batch
    if gate is not None:
        a.gate, a.ld_gate = gate.data_ptr(), gate.stride(0)
    _lib.call_struct('p3_gemm_any', a, _stream())
    return out


def _odd_pitch(t):
    """the same matrix with a row pitch that is no multiple of 4: the kernel for any alignment takes it"""
    out = torch.zeros(*t.shape[:-1], t.shape[-1] + 1 + t.shape[-1] % 2, dtype=t.dtype, device=t.device)
    out[..., :t.shape[-1]] = t
    return out[..., :t.shape[-1]]


@pytest.mark.parametrize('M,N,K', [(1, 1, 4), (1, 33, 8), (2, 16, 128), (3, 47, 132), (5, 100, 100), (8, 17, 260), (9, 64, 640), (16, 130, 1000),
                                   (17, 31, 16), (31, 33, 20), (33, 64, 12), (63, 129, 36), (65, 65, 260), (130, 1601, 64), (257, 200, 1000),
                                   (700, 1700, 44), (1100, 2050, 16)])
def test_fp32_products_of_aligned_rows_have_the_bits_of_the_general_kernel(dev, M, N, K):
    """every tile (rows 1 .. 16, 32, 64, 128) sums one FMA chain in ascending k: the bits of the kernel that takes any alignment"""
    g = torch.Generator(device=dev).manual_seed(M * 7 + N)
    rn = lambda *s: torch.randn(s, generator=g, device=dev)
    x, w, bias, gate = rn(M, K), rn(N, K), rn(N), rn(M, N)
    for b, gt, dt in ((None, None, F32), (bias, gate, F32), (bias, None, B16)):
        got, ref = _gemm_any(x, w, b, gate=gt, out_dtype=dt), _gemm_any(_odd_pitch(x), _odd_pitch(w), b, gate=gt, out_dtype=dt)
        assert torch.equal(got, ref)
    y = x.double() @ w.double().T
    bound = 2.0 ** -24 * K * (x.double().abs() @ w.double().abs().T) + 1e-30      # rounding of a chain of K additions
    assert ((_gemm_any(x, w).double() - y).abs() <= bound).all()


@pytest.mark.parametrize('cuts', [[0, 0, 1, 1, 40], [0, 64, 65, 200, 200], [0, 500, 500, 501, 1200]])
def test_fp32_grouped_gathered_and_batched_products(dev, cuts):
    g = torch.Generator(device=dev).manual_seed(cuts[-1])
    rn = lambda *s: torch.randn(s, generator=g, device=dev)
    M, N, K = cuts[-1], 72, 52
    x, w = rn(300, K), rn(4, N, K)
    rows = torch.randint(0, 300, (M,), generator=g, device=dev, dtype=torch.int32)
    seg = torch.tensor(cuts, dtype=torch.int32, device=dev)
    got, ref = _gemm_any(x, w, rows=rows, seg=seg), _gemm_any(_odd_pitch(x), _odd_pitch(w), rows=rows, seg=seg)
    assert torch.equal(got, ref) and bool(torch.isfinite(got).all())
    for m in (1, 7, 16, 40, 200):                                   # three products over column blocks, gathered rows
        xb, wb, r = rn(300, 3 * K), rn(3, N, K), rows[:1].repeat(m) if m > M else rows[:m].contiguous()
        got = _gemm_any(xb, wb, rows=r, batch=(3, K, N * K, N), N=N, K=K)
        ref = torch.cat([_gemm_any(_odd_pitch(xb[:, i * K:(i + 1) * K]), _odd_pitch(wb[i]), rows=r) for i in range(3)], 1)
        assert torch.equal(got, ref)


def _attention(dev, H, G, d, dv, lens, window=0, keep=0, chunk=0, sink=True, pen=0, sig=False, gate=False, elem=False, shared=False, scale=None, seed=0,
               offset=0, spread=1.0):
    """ragged prompts [(tokens, position of the first)] through p3_attn_window_prefill, and the same in float64"""
    from phi3_b200 import _lib
    g = torch.Generator(device=dev).manual_seed(seed)
    rn = lambda *s: torch.randn(s, generator=g, device=dev)
    scale = d ** -0.5 if scale is None else scale
    T = sum(n for n, _ in lens)
    q, n_pg = (rn(T, H, d) * spread).to(B16), [-(-(n + p) // 64) for n, p in lens]
    perm, bt = torch.randperm(sum(n_pg) + 2, generator=g, device=dev), torch.zeros(len(lens), max(n_pg), dtype=torch.int32, device=dev)
    kp = torch.full((sum(n_pg) + 2, G, 64, d), 9.0, dtype=B16, device=dev)
    vp = kp if shared else torch.full((sum(n_pg) + 2, G, 64, dv), 9.0, dtype=B16, device=dev)
    sk, pe = (rn(H) if sink else None), (torch.rand(H, 1, generator=g, device=dev) * torch.log1p(torch.arange(pen, device=dev) * 0.3)[None] if pen else None)
    sb, gt, eg = (rn(H) - 1 if sig else None), (torch.rand(T, H, generator=g, device=dev) if gate else None), (rn(T, H * dv + 3)[:, 3:] if elem else None)
    refs, tiles, r, at = [], [], 0, 0
    for s, ((n, p), pages) in enumerate(zip(lens, n_pg)):
        k = rn(n + p, G, d).to(B16)
        v = k[..., :dv] if shared else rn(n + p, G, dv).to(B16)
        ids = perm[at:at + pages]
        bt[s, :pages], at = ids.int(), at + pages
        for pool, t in ((kp, k),) if shared else ((kp, k), (vp, v)):
            full = torch.full((pages * 64, G, t.shape[-1]), 5.0, dtype=B16, device=dev)
            full[:n + p] = t
            pool[ids] = full.view(pages, 64, G, -1).transpose(1, 2)
        tiles += [(r + i, min(64, n - i), s, p + i) for i in range(0, n, 64)]
        i, j = torch.arange(p, p + n, device=dev)[:, None], torch.arange(n + p, device=dev)[None]
        seen, dist = torch.ones(n, n + p, dtype=torch.bool, device=dev), i - j
        if window:
            seen &= dist < window
        if chunk:
            seen &= i // chunk == j // chunk
        seen = (dist >= 0) & (seen | (j < keep))
        sc = torch.einsum('thd,shd->hts', q[r:r + n].double(), k.double().repeat_interleave(H // G, 1)) * scale
        if pen:
            sc = sc - pe.double()[:, dist.clamp(0, pen - 1)]
        if sig:
            a = torch.sigmoid(sc + sb.double()[:, None, None]) * seen
        else:
            sc = sc.masked_fill(~seen, -float('inf'))
            m = sc.amax(-1, keepdim=True)
            m = torch.maximum(m, sk.double()[:, None, None]) if sink else m
            e = torch.exp(sc - m)
            a = e / (e.sum(-1, keepdim=True) + (torch.exp(sk.double()[:, None, None] - m) if sink else 0))
        refs.append(torch.einsum('hts,shd->thd', a, v.double().repeat_interleave(H // G, 1)))
        r += n
    ref = torch.cat(refs)
    if gate:
        ref = ref * gt.double()[..., None]
    ref = ref.reshape(T, H * dv) * (torch.sigmoid(eg.double()) if elem else 1.0)
    td, out = torch.tensor(tiles, dtype=torch.int32, device=dev), torch.full((T, H * dv), float('nan'), dtype=B16, device=dev)
    w = _lib.AttnWindowArgs()
    qf = q.reshape(T, H * d)
    w.q, w.ld_q, w.k_pool, w.v_pool, w.block_table, w.bt_stride = qf.data_ptr(), H * d, kp.data_ptr(), vp.data_ptr(), bt.data_ptr(), bt.stride(0)
    w.sink, w.penalty, w.n_penalty, w.gate, w.out, w.ld_out = _lib.ptr(sk), _lib.ptr(pe), pen, _lib.ptr(gt), out.data_ptr(), H * dv
    w.n_heads, w.n_kv, w.dim, w.vdim, w.scale, w.window, w.keep_first, w.chunk, w.v_ld = H, G, d, dv, scale, window, keep, chunk, d if shared else 0
    w.sig_bias, w.elem_gate, w.ld_elem_gate, w.tiles, w.n_tiles = _lib.ptr(sb), _lib.ptr(eg), H * dv + 3, td.data_ptr(), len(tiles)
    _lib.call_struct('p3_attn_window_prefill', w, _stream())
    torch.cuda.synchronize()
    return out.double(), ref


SHAPES = [  # heads, K/V heads, key size, value size, (tokens, position of the first) of every sequence
    (4, 4, 96, 96, [(2, 0), (64, 0), (65, 63), (130, 1)]), (8, 2, 128, 128, [(300, 0), (63, 640)]), (6, 3, 64, 64, [(129, 0), (2, 700)]),
    (3, 1, 16, 48, [(200, 5)]), (16, 16, 112, 16, [(700, 64), (2, 0), (66, 130)]), (32, 1, 128, 128, [(70, 900)]), (2, 2, 80, 128, [(513, 0)]),
    (64, 64, 64, 64, [(260, 0), (100, 0), (100, 0)]), (16, 4, 128, 96, [(1025, 100), (500, 0), (40, 2000)])]


@pytest.mark.parametrize('shape', range(len(SHAPES)))
@pytest.mark.parametrize('kind', ['plain', 'window', 'keep', 'chunk', 'sigmoid', 'gates', 'far'])
def test_prefill_attention_over_ragged_batches(dev, shape, kind):
    """head groups, sizes of one and two boxes, records of several sequences in one CTA, masks, gates; weights are rounded to bf16 once
    (relative 2^-9 each, averaging out) and so is the output (2^-9)"""
    H, G, d, dv, lens = SHAPES[shape]
    kw = {'plain': dict(sink=False), 'window': dict(window=100, pen=100), 'keep': dict(window=65, keep=70), 'chunk': dict(chunk=96),
          'sigmoid': dict(sink=False, sig=True, window=200), 'gates': dict(gate=True, elem=True, pen=5000),
          'far': dict(sink=False, spread=60.0)}[kind]                  # scores of hundreds: the reference falls 2^64 behind and pages are swept again
    y, ref = _attention(dev, H, G, d, dv, lens, seed=shape, **kw)
    assert bool(torch.isfinite(y).all())
    assert float((y - ref).norm() / ref.norm()) < 6e-3
    assert float((y - ref).abs().max()) < 2.0 ** -6 * float(ref.abs().max())


def test_prefill_attention_with_one_shared_row_per_token(dev):
    for H, lens in ((16, [(700, 100), (300, 0)]), (4, [(33, 0)]), (1, [(200, 64)])):
        y, ref = _attention(dev, H, 1, 128, 96, lens, window=512, shared=True, seed=H)
        assert float((y - ref).norm() / ref.norm()) < 6e-3


@pytest.mark.parametrize('cuts', [[0, 1], [0, 0, 0, 3, 3], [0, 32, 65, 65, 200], [0, 129, 130, 258, 258], [0, 5, 300, 900, 901, 1500], [0] + [7 * i for i in range(1, 71)]])
@pytest.mark.parametrize('N,K', [(128, 64), (200, 72), (72, 136), (384, 520)])
def test_grouped_products_over_ordered_rows(dev, cuts, N, K):
    """few rows per group (boxes of 32 and 128 rows) and many (CTA pairs); rows behind the last group are not written. fp32 sums of K bf16
    products, in another order than float64: 2^-20 of the sum of magnitudes"""
    g = torch.Generator(device=dev).manual_seed(N + cuts[-1])
    M, E = cuts[-1] + 9, len(cuts) - 1
    x, w = torch.randn(M, K, generator=g, device=dev).to(B16), torch.randn(E, N, K, generator=g, device=dev).to(B16)
    seg = torch.tensor(cuts, dtype=torch.int32, device=dev)
    for dt in (F32, B16):
        got = _gemm_any(x, w, seg=seg, out_dtype=dt)
        assert bool(torch.isnan(got[cuts[-1]:]).all())
        for e in range(E):
            a, b = cuts[e], cuts[e + 1]
            y, bound = x[a:b].double() @ w[e].double().T, 2.0 ** -20 * (x[a:b].double().abs() @ w[e].double().abs().T)
            if dt == B16:
                bound = bound + 2.0 ** -8 * y.abs()
            assert ((got[a:b].double() - y).abs() <= bound).all()


@pytest.mark.parametrize('n,E', [(1, 1), (7, 3), (128, 8), (129, 5), (1000, 64), (8192, 8), (30001, 16)])
def test_expert_order_is_stable(dev, n, E):
    from phi3_b200 import _lib
    g = torch.Generator(device=dev).manual_seed(n)
    ids = torch.randint(0, E, (n,), generator=g, device=dev, dtype=torch.int32)
    seg, order, where = (torch.full((k,), -1, dtype=torch.int32, device=dev) for k in (E + 1, n, n))
    _lib.call('p3_moe_sort', ids.data_ptr(), n, E, seg.data_ptr(), order.data_ptr(), where.data_ptr(), _stream())
    ref = torch.sort(ids.long(), stable=True).indices
    assert torch.equal(order.long(), ref) and torch.equal(where[order.long()].long(), torch.arange(n, device=dev))
    assert seg.tolist() == [int((ids < e).sum()) for e in range(E + 1)]
