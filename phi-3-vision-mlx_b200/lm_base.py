"""What the engine models (decoders with an fp32 residual stream that run a ragged token batch against the shared page pool) have in
common: the description of a step, the choice of the matrix-product kernel, the grouped expert products, the attention launches of a
step and the key-slice cost model of the decode attention. A design (tagenex.py, tapalix.py, dugalix.py, danalorn.py, lupusun.py,
gugezen.py) owns its weights and the order of its kernels; it has no cache and no loop of its own.

Matrix products. Dense bf16 products with K % 8 == 0 run on the tcgen05 GEMM (p3_gemm); batches of at most 16 tokens on the
weight-streaming kernel (p3_gemm_skinny); everything else (fp32 = true 32-bit, on the FMA pipes or in three bf16 parts
on tcgen05; grouped expert products, products per attention head over column blocks, odd shapes) on p3_gemm_any.
"""
import ctypes as C
import operator
import os
import torch
from . import _lib
from ._lib import PAGE, call, call_struct, ptr


def _stream():
    """handle of the current stream, without the Stream object that torch.cuda.current_stream() makes for every launch"""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def _page_slices(pairs, pages, slots=2 * 148, merge=0.0):
    """slices of the visible pages per (request, K/V head) for the tensor-core decode attention (two CTAs per SM). Cost model in
    units of the memory latency: a CTA pays one latency to fill its copy ring and half of one per page after that (two pages in
    flight); equal CTAs run in whole rounds of the resident ones. `merge`: what every further slice adds to the merge kernel, which
    walks the slices of a head one after the other (it matters when one K/V head serves many query heads: few CTAs, so the model
    would otherwise cut the keys into very many slices)."""
    best, best_cost = 1, float('inf')
    for ns in range(1, max(1, min(pages, 32)) + 1):
        per = -(-pages // ns)
        cost = -(-pairs * ns // slots) * (1.0 + per / 2.0) + (merge * ns if ns > 1 else 0.0)
        if cost < best_cost - 1e-9:
            best, best_cost = ns, cost
    return best


_last_of = operator.itemgetter(1)


def _shape_of_prompts(w, b, span_of):
    """what the prefill launch shares its work out by: pages that a record of 64 rows sees at most, sequences of the records; span_of(n) = most keys
    a query at position n - 1 sees. A batch that does not say where its prompts lie is taken for one sequence's, or for as many as leave their
    last records half empty where that is more than one can leave"""
    if b.n_pf * w.n_heads > 224 or b.max_pos < 11 * PAGE:        # passes enough, or pages too few to be worth sharing
        w.max_pages = 0
        return
    runs, chunk, pages = b.pf_runs, w.chunk, 0
    if runs is None:
        rows = b.T - b.n_dec
        spare = PAGE * b.n_pf - rows
        w.n_seqs = 1 if spare < PAGE else (spare + PAGE // 4) // (PAGE // 2)
        runs = ((max(0, b.max_pos + 1 - rows), b.max_pos),)
    else:
        w.n_seqs = len(runs)
    if not chunk:
        runs = (max(runs, key=_last_of),)
    for first, last in runs:
        n = last % chunk + 1 if chunk and first // chunk == last // chunk else last + 1
        pages = max(pages, min(last // PAGE + 1, (span_of(n) + 2 * PAGE - 2) // PAGE))
    w.max_pages = pages


class StepBatch:
    """Device-side description of one engine step (built by engine.Engine.step)."""
    __slots__ = ('T', 'ids', 'tok_slot', 'tok_pos', 'pf_tiles', 'n_pf', 'dec_tiles', 'n_dec', 'want_rows', 'R', 'max_pos', 'pf_runs', 'flat',
                 'seqs', 'n_seq', 'slot_seq', 'n_slots')

    def __init__(self):
        self.pf_runs = None                                      # (first, last position) of every prompt, where the batch's maker says so


class PagedLM:
    """base of the engine models: subclasses set self.dev, self.dtype, self.W (width), self.eps and call _init_products()"""
    use_tc = True                # products on tcgen05 where they can be (P3_LM_TC)

    def _init_products(self):
        self.f32 = int(self.dtype == torch.float32)
        self.use_tc = os.environ.get('P3_LM_TC', '1') != '0'
        self.moe_dense_rows = int(os.environ.get('P3_LM_MOE_DENSE_ROWS', '1'))   # (token, choice) pairs from which the experts run on gathered rows (tcgen05)
        self.use_skinny = os.environ.get('P3_LM_SKINNY', '1') != '0' and hasattr(_lib.lib(), 'p3_gemm_skinny')
        self.profile = None      # bench.py: list of (kind, ev0, ev1, flops, bytes) when instrumenting

    def cache_dtype(self):
        return self.dtype

    def _ev(self, start=None, kind=None, flops=0, nbytes=0):
        if self.profile is None:
            return None
        e = torch.cuda.Event(enable_timing=True)
        e.record()
        if start is not None:
            self.profile.append((kind, start, e, flops, nbytes))
        return e

    def rows(self, kind, nbytes, name, *args):
        """a row kernel (norms, rotations, activations, routing) launched through _lib.call, or through _lib.call_struct when
        `args` is (argument struct,); bench.py's instrumentation times it under `kind` with the bytes it moves"""
        ev = self._ev()
        if len(args) == 1 and hasattr(args[0], '_fields_'):
            call_struct(name, args[0], _stream())
        else:
            call(name, *args)
        self._ev(ev, kind, 0, nbytes)

    # ------------------------------------------------------------------ matrix products
    def linear(self, x, w, out, bias32=None, bias16=None, nxt=None):
        """out[M,N] (fp32 or act type, by out.dtype) = x[M,K] w[N,K]^T (+ bias). Returns the bias (fp32) that is STILL TO ADD: None
        when the product added it, bias32 when the kernel has no bias input (the weight-streaming kernel of small batches); the
        consumer kernel (activation / output norm) then adds it. `nxt`: the matrix of the next product; the weight-streaming
        kernel pulls its first megabytes into L2 so that they arrive while the small kernels in between run."""
        M, K = x.shape
        N = w.shape[0]
        ev = self._ev()
        try:
            return self._linear(x, w, out, bias32, bias16, nxt)
        finally:
            self._ev(ev, 'gemm', 2 * M * N * K, w.numel() * w.element_size() + x.numel() * x.element_size() + out.numel() * out.element_size())

    L2_PREFETCH_CAP = int(os.environ.get('P3_LM_PF_CAP_MB', '16')) << 20

    def _linear(self, x, w, out, bias32=None, bias16=None, nxt=None):
        M, K = x.shape
        N = w.shape[0]
        aligned = (not self.f32 and K % 8 == 0 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)
        if (self.use_skinny and aligned and M <= 16 and K % 64 == 0 and N % 16 == 0 and out.dtype == torch.float32
                and w.is_contiguous()):
            # <= 16 tokens: the product is a stream of the weights; the Phi-3 decode kernel does that at HBM speed
            pf = 0 if nxt is None else min(nxt.numel() * nxt.element_size(), self.L2_PREFETCH_CAP)
            call('p3_gemm_skinny', ptr(x), x.stride(0), None, self.eps, ptr(w), ptr(out), out.stride(0), None, M, N, K,
                 _lib.EPI_F32, None, 0, None, ptr(nxt) if pf else None, pf, _stream())
            return bias32
        if self.use_tc and aligned and (bias32 is None or bias16 is not None):
            epi = _lib.EPI_F32 if out.dtype == torch.float32 else _lib.EPI_NONE
            call('p3_gemm', ptr(x), x.stride(0), ptr(w), w.stride(0), ptr(bias16), ptr(out), out.stride(0), None, None,
                 M, N, K, epi, 0, _stream())
            return None
        self.gemm_any(x, w, out, bias32)
        return None

    def gated(self, x, w, act, hid, bias32=None, bias16=None, limit=0.0, alpha=0.0, nxt=None):
        """hid[M,F] = act(g) * u, [g | u] = x w^T (+ bias): one launch where p3_gemm would take CTA pairs for this product (5418
        rows, 2048 -> 8192: 233 us, as two launches 401), else the product into fp32 rows and the activation kernel."""
        (M, K), F = x.shape, w.shape[0] // 2
        if (self.use_tc and not self.f32 and F % 32 == 0 and w.shape[0] == 2 * F and M > 16 and _lib.lib().p3_gemm_pair_width(M, 2 * F)
                and (bias32 is None or bias16 is not None) and not any(t.stride(0) % 8 or t.data_ptr() % 16 for t in (x, w, hid))
                and (bias16 is None or bias16.data_ptr() % 16 == 0)):
            ev = self._ev()
            call('p3_gemm_glu', ptr(x), x.stride(0), ptr(w), w.stride(0), ptr(bias16), ptr(hid), hid.stride(0), M, F, K, act, limit, alpha, _stream())
            self._ev(ev, 'gemm', 4 * M * F * K, w.numel() * 2 + x.numel() * 2 + hid.numel() * 2)
            return
        gu = torch.empty((M, w.shape[0]), dtype=torch.float32, device=self.dev)
        left = self.linear(x, w, gu, bias32, bias16, nxt=nxt)
        nbytes = M * F * (8 + (4 if self.f32 else 2))
        if act == _lib.GLU_CLAMPED:
            self.rows('activation', nbytes, 'p3_glu_clamped', ptr(gu), gu.stride(0), ptr(hid), hid.stride(0), self.f32, M, F, limit, alpha,
                      ptr(left), _stream())
        else:
            if left is not None:                                 # p3_glu_act takes no bias
                gu += left
            self.rows('activation', nbytes, 'p3_glu_act', ptr(gu), ptr(gu[:, F:]), gu.stride(0), ptr(hid), hid.stride(0), self.f32, M, F, act,
                      _stream())

    def gemm_any(self, x, w, out, bias=None, rows=None, row_div=1, seg=None, n_groups=0, M=None, N=None, K=None, ldw=None,
                 batch=None, gate=None):
        """out = x w^T on p3_gemm_any. rows / row_div: gathered activation rows; seg / n_groups: row segments that each take their
        own matrix w[g]. batch = (n, x stride, w stride, out stride): n products over column blocks of x and out (N, K, ldw give the
        shape of one), gate: fp32 logits whose sigmoid multiplies the result."""
        a = _lib.GemmAnyArgs()
        a.X, a.ldx, a.x_f32 = ptr(x), x.stride(0), self.f32
        a.x_rows, a.x_row_div = ptr(rows), row_div
        a.W, a.ldw, a.w_f32 = ptr(w), (w.stride(-2) if ldw is None else ldw), self.f32
        a.w_group_stride = w.stride(0) if (w.dim() == 3 and batch is None) else 0
        a.bias, a.bias_group_stride = ptr(bias), (bias.stride(0) if bias is not None and bias.dim() == 2 else 0)
        a.out, a.ldo, a.out_f32 = ptr(out), out.stride(0), int(out.dtype == torch.float32)
        a.M = x.shape[0] if M is None else M
        a.N, a.K = (w.shape[-2] if N is None else N), (w.shape[-1] if K is None else K)
        a.seg_offsets, a.n_groups, a.force_fma = ptr(seg), n_groups, 0 if self.use_tc else 2
        if batch is not None:
            a.n_batch, a.x_batch_stride, a.w_batch_stride, a.out_batch_stride = batch
        if gate is not None:
            a.gate, a.ld_gate = ptr(gate), gate.stride(0)
        call_struct('p3_gemm_any', a, _stream())
        return out

    def stacked_rows(self, parts):
        """projection matrices over one input as one matrix in the compute type, padded with zero rows to a multiple of 16 (small
        batches keep the weight-streaming kernel)"""
        n = sum(p.shape[0] for p in parts)
        if n % 16:
            parts = parts + [torch.zeros(-n % 16, parts[0].shape[1], dtype=parts[0].dtype, device=parts[0].device)]
        return torch.cat(parts, 0).to(self.dev, self.dtype).contiguous()

    # ------------------------------------------------------------------ attention over the page pool
    def attention_tile_rows(self, H, G, key, val, v_ld, ld_out=None):
        """query rows per prefill tile that the attention launch takes for these sizes (64: its tensor-core kernels); asked of the
        library itself so that the engine's tiles and the kernel's choice cannot disagree. ld_out: pitch of the output rows, when
        they are wider than the heads"""
        a = _lib.AttnWindowArgs()
        a.q = a.out = a.k_pool = a.v_pool = a.block_table = a.tiles = 256              # aligned stand-ins: nothing is launched
        a.ld_q, a.ld_out, a.n_heads, a.n_kv, a.dim, a.vdim, a.v_ld = H * key, ld_out or H * val, H, G, key, val, v_ld
        a.act_f32 = a.cache_f32 = self.f32
        return int(_lib.lib().p3_attn_window_tile_rows(C.byref(a)))

    def attend(self, w, tile_rows, b, G, key, val, span_of, kv_bytes, pf_span=None):
        """the prefill tiles and the single-token requests of the step through p3_attn_window_*; span_of(n) = most keys a query at
        position n - 1 sees, pf_span = mean keys per query of a prompt (accounting only), kv_bytes = cache numbers of one token"""
        st, H = _stream(), w.n_heads
        esz = 4 if self.f32 else 2
        if b.n_pf:
            w.tiles, w.n_tiles = ptr(b.pf_tiles), b.n_pf
            _shape_of_prompts(w, b, span_of)
            ev = self._ev()
            call_struct('p3_attn_window_prefill', w, st)
            if pf_span is None:
                pf_span = span_of(b.max_pos + 1) if w.window else (b.max_pos + 1) // 2
            self._ev(ev, 'attn_prefill', 2 * (b.T - b.n_dec) * H * pf_span * (key + val), 0)
        if b.n_dec:
            w.tiles, w.n_tiles = ptr(b.dec_tiles), b.n_dec
            span = span_of(b.max_pos + 1)
            if tile_rows == 64:
                if G == 1 and H > 1:
                    # one shared K/V head: a request is one CTA per slice (two when the values take two column blocks)
                    w.n_splits = _page_slices(b.n_dec * (-(-val // 128) if key > 128 else 1), 2 * -(-span // 128) + 1, merge=0.4)
                else:
                    w.n_splits = _page_slices(b.n_dec * G, 2 * -(-span // 128) + 1)
            else:
                # one key per lane: enough CTAs for eight per SM, at least 128 keys (one pass of a CTA) per slice
                w.n_splits = max(1, min(-(-8 * 148 // (b.n_dec * G)), -(-span // 128)))
            ws = torch.empty(b.n_dec * H * w.n_splits * (val + 2), dtype=torch.float32, device=self.dev) if w.n_splits > 1 else None
            w.ws = ptr(ws)
            ev = self._ev()
            call_struct('p3_attn_window_decode', w, st)
            self._ev(ev, 'attn_decode', 2 * b.n_dec * H * span * (key + val), b.n_dec * span * kv_bytes * esz)

    # ------------------------------------------------------------------ mixture of experts behind a router
    def experts(self, gu_w, down_w, f, xa, y, T, ids, wts, glu, n_sorted=None, combine=None, meanwhile=None):
        """ids / wts [T, top] from the design's router -> y fp32 [T, W] = sum of the chosen experts' outputs. gu_w [E, 2 ff, W] holds
        every expert's gate rows over its up rows, down_w [E, W, ff]; glu(gu fp32 [n, 2 ff], hid act [n, ff], n) is the design's
        activation. The (token, choice) pairs are sorted by expert and run as two grouped products over the sorted rows.
        A unit without a gate passes its up matrices alone ([E, ff, W]; the activation then gets [n, ff]). n_sorted: the router
        scores this many outputs, of which only the first f.experts have matrices (the pairs of the others are sorted behind them
        and skipped by the products); combine(dn, where) then replaces the plain weighted sum. meanwhile(): work that does not
        depend on the choice (a shared unit), launched behind the sort."""
        st, dev, n = _stream(), self.dev, T * f.top
        n_sorted = f.experts if n_sorted is None else n_sorted
        up, dense, esz = gu_w.shape[1], self.experts_dense(f, T), 4 if self.f32 else 2
        gu = torch.empty((n, up), dtype=torch.float32, device=dev)
        hid = torch.empty((n, f.ff), dtype=self.dtype, device=dev)
        # what only the kernels here see lies in one allocation (a step of few tokens is bound by the host, and an allocation costs it as much
        # as a launch): row outputs, rows in expert order, segment offsets, order and places, each on a 256-byte boundary
        parts = (0 if combine is not None else n * self.W * 4, n * self.W * esz if dense else 0, 4 * (n_sorted + 1), 4 * n, 4 * n)
        at = [0]
        for size in parts:
            at.append(at[-1] + (size + 255 & ~255))
        scratch = torch.empty(at[-1], dtype=torch.uint8, device=dev)
        base = scratch.data_ptr()
        dn, xs, seg, order, where = (base + o for o in at[:5])
        if combine is not None:
            rows_out = torch.empty((n, self.W), dtype=torch.float32, device=dev)
            places, dn = scratch[at[4]:at[4] + 4 * n].view(torch.int32), rows_out.data_ptr()
        self.rows('route', n * 12, 'p3_moe_sort', ptr(ids), n, n_sorted, seg, order, where, st)
        if meanwhile is not None:
            meanwhile()
        # The rows are brought into expert order and run as ONE grouped product per matrix on the tcgen05 GEMM, whose CTAs find their expert
        # from the segment offsets on the device: nothing is read back, whatever the number of rows. What that kernel does not take (fp32,
        # sizes that are no multiples of 8) runs on the grouped kernel for any shape, which gathers the rows itself.
        ev = self._ev()
        if dense:
            call('p3_gather_rows', ptr(xa), xa.stride(0), self.f32, order, f.top, xs, n, self.W, st)
            self._grouped(xs, self.W, None, gu_w, gu.data_ptr(), up, seg, f.experts, n, st)
        else:
            self._grouped(ptr(xa), xa.stride(0), (order, f.top), gu_w, gu.data_ptr(), up, seg, f.experts, n, st)
        self._ev(ev, 'moe_gemm', 2 * n * up * self.W, gu_w.numel() * gu_w.element_size())
        glu(gu, hid, n)
        ev = self._ev()
        self._grouped(hid.data_ptr(), f.ff, None, down_w, dn, self.W, seg, f.experts, n, st)
        self._ev(ev, 'moe_gemm', 2 * n * f.ff * self.W, down_w.numel() * down_w.element_size())
        if combine is not None:
            combine(rows_out, places)
        else:
            self.rows('combine', T * self.W * 4 * (f.top + 1), 'p3_moe_combine', dn, self.W, where, ptr(wts), f.top, ptr(y), T, self.W, st)

    def _grouped(self, x, ldx, gather, w, out, ldo, seg, groups, M, st):
        """a grouped product of the experts, by addresses: out fp32 [M, ldo] = rows of x (gather: the sorted pairs and the choices of a token,
        else row by row), segment by segment, times w[g]^T"""
        rows, div = (None, 1) if gather is None else gather
        call_struct('p3_gemm_any', _lib.GemmAnyArgs(x, ldx, self.f32, rows, div, w.data_ptr(), w.stride(1), self.f32, w.stride(0), None, 0, out, ldo, 1,
                                                    M, w.shape[1], w.shape[2], seg, groups, 0 if self.use_tc else 2), st)

    def experts_dense(self, f, T):
        """do the experts of a step with T tokens run on gathered rows (the tcgen05 GEMM)?"""
        return bool(self.use_tc and not self.f32 and T * f.top >= self.moe_dense_rows and self.W % 8 == 0 and f.ff % 8 == 0)
