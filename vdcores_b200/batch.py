"""Batched greedy decode (2..128 sequences in lock-step) on the tensor cores.

The reference pads every decode batch to 8 request slots and pushes it through
its 64x8 WGMMA GEMV tile (reference include/task/gemv.cuh:13-128,
python/dae/schedule.py:404-570).  Here a step is a list of stage kernels
(csrc/stage_kernels.cu), one per projection and attention, launched back to
back with programmatic dependent launch: the batch sits on the 128 lanes of a
tcgen05 accumulator in tensor memory, blocks of 128 weight rows on its columns,
and activations live in HBM in the k-chunk-major layout the tensor cores read
without swizzling (csrc/isa.h).  Every sequence has its own state block, page
table and length.

The helpers above the engine (`emit_projection` and the layouts it packs) emit
the same projection as tasks of the megakernel.
"""
from __future__ import annotations

from typing import List

import torch

from . import isa, runtime
from .decode import BF16, DecodeConfig, DecodeEngine, kv_page_swizzle
from .program import Program, Src


def pack_kc(x: torch.Tensor) -> torch.Tensor:
    """[R, K] -> flat k-chunk-major [K/8][R/8][8][8] (R, K multiples of 8)."""
    R, K = x.shape
    return x.reshape(R // 8, 8, K // 8, 8).permute(2, 0, 1, 3).contiguous().view(-1)


def unpack_kc(flat: torch.Tensor, R: int, K: int) -> torch.Tensor:
    return flat.view(K // 8, R // 8, 8, 8).permute(1, 2, 0, 3).reshape(R, K)


BLOCK_ROWS = 256    # weight rows per projection block = accumulator columns of one tensor-core task


def projection_blocks(M: int, rows: int = BLOCK_ROWS):
    """[(first row, rows)] of a projection with M output rows (a multiple of 16)."""
    assert M % 16 == 0
    return [(r, min(rows, M - r)) for r in range(0, M, rows)]


def _pack_blocks(rows_of, M: int, bytes_or_elems_per_row: int, out: torch.Tensor, rows: int) -> torch.Tensor:
    """Fills `out` block by block; rows_of(r0, blocks, n) returns the packed rows r0 .. r0 + blocks * n - 1 as `blocks`
    blocks of n rows: all full blocks at once, then the smaller last one."""
    full = M // rows
    if full:
        out[:full * rows * bytes_or_elems_per_row] = rows_of(0, full, rows).reshape(-1)
    if M % rows:
        out[full * rows * bytes_or_elems_per_row:] = rows_of(full * rows, 1, M % rows).reshape(-1)
    return out


def pack_blocks(w: torch.Tensor, rows: int = BLOCK_ROWS) -> torch.Tensor:
    """[M, K] -> flat: every block of `rows` rows (the last one may be smaller) k-chunk-major, so
    that any K-range of a block is one contiguous piece; block (r0, N) starts at element r0 * K."""
    M, K = w.shape
    return _pack_blocks(lambda r0, nb, n: w[r0:r0 + nb * n].reshape(nb, n // 8, 8, K // 8, 8).permute(0, 3, 1, 2, 4),
                        M, K, torch.empty(M * K, dtype=w.dtype, device=w.device), rows)


def pack_blocks_fp8(codes: torch.Tensor, rows: int = BLOCK_ROWS) -> torch.Tensor:
    """[M, K] e4m3 bytes -> flat: per block of `rows` rows the layout [K/16][N/8][8 rows][16 k],
    which a 16-byte load turns into two adjacent bf16 pieces of the tensor-core operand layout."""
    M, K = codes.shape
    return _pack_blocks(lambda r0, nb, n: codes[r0:r0 + nb * n].reshape(nb, n // 8, 8, K // 16, 16).permute(0, 3, 1, 2, 4),
                        M, K, torch.empty(M * K, dtype=codes.dtype, device=codes.device), rows)


def pack_blocks_nvfp4(w: torch.Tensor, K: int, rows: int = BLOCK_ROWS) -> torch.Tensor:
    """[M, K/2 + K/16] NVFP4 rows (e2m1 pairs, then the e4m3 block scales) -> flat: per block of `rows` rows
    and per 16 inputs, the rows' 8 code bytes followed by the rows' scale bytes ([K/16][N x 8 | N]), so that
    any K-range of a block is one contiguous piece of 9 N bytes per 16 inputs."""
    M = w.shape[0]
    codes, bs = w[:, :K // 2].reshape(M, K // 16, 8), w[:, K // 2:]

    def rows_of(r0, nb, n):
        c = codes[r0:r0 + nb * n].reshape(nb, n, K // 16, 8).transpose(1, 2).reshape(nb, K // 16, n * 8)
        return torch.cat((c, bs[r0:r0 + nb * n].reshape(nb, n, K // 16).transpose(1, 2)), dim=2)
    return _pack_blocks(rows_of, M, K * 9 // 16, torch.empty(M * K * 9 // 16, dtype=w.dtype, device=w.device), rows)


def chunk_geometry(N: int, Bpad: int, K: int):
    """(Kc, G): inputs per W chunk (N * Kc * 2 bytes <= 32 KB, Kc divides K) and W chunks per X chunk
    (the X chunk fills at most one 8 KB slot when it can)."""
    kc = 256 if N <= 64 else 128 if N <= 128 else 64
    while K % kc or Bpad * kc * 2 > 16384:
        kc //= 2
    assert kc >= 16
    return kc, max(1, min(4, 8192 // (Bpad * kc * 2)))


def plan_units(blocks, steps: int, sms, load, step_bytes_per_row: int):
    """Deals the (block, W chunk) steps of a projection to the SMs, in `sms` order, as contiguous
    ranges of about equal bytes.  Returns [(sm, block index, first chunk, chunk count)]."""
    remaining = sum(n for _, n in blocks) * steps     # in rows x steps
    units, bi, ci = [], 0, 0
    for i, sm in enumerate(sms):
        quota = -(-remaining // (len(sms) - i))
        got = 0
        while bi < len(blocks) and got < quota:
            n = blocks[bi][1]
            take = min(max(1, round((quota - got) / n)), steps - ci)
            units.append((sm, bi, ci, take))
            got += take * n
            ci += take
            if ci == steps:
                bi, ci = bi + 1, 0
        remaining -= got
        load[sm] += got * step_bytes_per_row
    assert bi == len(blocks) and remaining == 0
    return units


def emit_projection(P: Program, *, sms, load, w_addr, M, K, x_addr, B, Bpad, mode, out_addr, scratch_addr,
                    counter_addr, x_wait=None, release=None, norm_addr=None, eps=0.0, ld=0, keys_addr=0, stats_addr=0,
                    wfmt="bf16", scales_addr=0):
    """Emits every unit of the projection y[B, M] = x[B, K] W^T (W packed by pack_blocks at w_addr,
    x k-chunk-major at x_addr).  scratch_addr: fp32 [blocks][B][256]; counter_addr: int32 [blocks]."""
    blocks = projection_blocks(M)
    Kc, G = chunk_geometry(blocks[0][1], Bpad, K)
    wb16 = {"bf16": 32, "fp8": 16, "nvfp4": 9}[wfmt]       # bytes per 16 weights of one row
    units = plan_units(blocks, K // Kc, sms, load, Kc * wb16 // 16)
    slices = [0] * len(blocks)
    for _, bi, _, _ in units:
        slices[bi] += 1
    if release is not None:
        P.add_releases(release, len(blocks))
    for sm, bi, c0, cnt in units:
        r0, N = blocks[bi]
        k0 = c0 * Kc
        P.gemm_tc(sm, w_addr=w_addr + (r0 * K + k0 * N) * wb16 // 16, N=N, K=K, k_len=cnt * Kc, Kc=Kc, G=G,
                  wfmt=wfmt, scales_addr=scales_addr + 4 * r0 if scales_addr else 0,
                  x_addr=x_addr + k0 * Bpad * 2, B=B, Bpad=Bpad, out_addr=out_addr, mode=mode, x_wait=x_wait,
                  norm_w=Src(norm_addr + k0 * 2, cnt * Kc * 2) if norm_addr is not None else None, eps=eps, n0=r0,
                  ld=ld, keys_addr=keys_addr, stats_addr=stats_addr, release=release,
                  scratch_addr=scratch_addr + bi * B * BLOCK_ROWS * 4, counter_addr=counter_addr + 4 * bi,
                  n_slices=slices[bi])
    return units


class BatchDecodeEngine(DecodeEngine):
    """`batch` sequences decoded together, one list of stage kernels per step.  Dense models; the layer
    projections are bf16, e4m3 with per-row scales (wkind "fp8") or NVFP4 (wkind "nvfp4": e2m1 values, e4m3 block
    scales, fp32 tensor scale), everything else bf16.  num_sms sizes the K-splits of the projections and the page shares of
    the attention; below the device's count it also bounds the CTAs of a step that run at any time, and so the SMs it
    takes."""
    GEMV_PROJECTIONS = False
    SHARED_CACHE = False     # True: the batch rows are consecutive positions of ONE sequence (prefill.PrefillEngine)

    def __init__(self, cfg: DecodeConfig, batch: int, max_seq: int, device="cuda:0", num_sms=None, taps=False,
                 page_perm_seed=None, max_steps: int = 256, timeout_ns: int = 2_000_000_000, wkind: str = "bf16"):
        assert 1 <= batch <= 128 and not cfg.n_experts and wkind in ("bf16", "fp8", "nvfp4")
        self.batch = batch
        self.bpad = next(p for p in (16, 32, 64, 128) if batch <= p)
        super().__init__(cfg, max_seq, device=device, num_sms=num_sms, taps=False, page_perm_seed=None,
                         max_steps=max_steps, timeout_ns=timeout_ns, wkind=wkind)
        B, Bp, L, H, F = batch, self.bpad, cfg.n_layers, cfg.hidden, cfg.ffn
        z = lambda *s, dt=BF16: torch.zeros(*s, dtype=dt, device=self.dev)
        self.hidden = z(Bp * H)                       # k-chunk-major [Bpad, H]
        self.attn_out = z(Bp * cfg.q_width)           # k-chunk-major [Bpad, q_width]
        self.act = z(Bp * F)                          # k-chunk-major [Bpad, F]
        self.normed = z(Bp * H)                       # k-chunk-major: normalised hidden rows
        self.q = z(B, cfg.q_width)                    # rotated query heads
        self.keys = z(B, dt=torch.int64)              # argmax keys (u64), zero between steps
        # per-sequence sums of squares of the hidden matrix after the embedding / each residual add
        # (the RMSNorm statistics of the projection that reads it); zero between steps
        self.stats = z(2 * L + 1, 128, dt=torch.float32)
        self.stages = None
        self.max_ctas = self.num_sms if self.num_sms < torch.cuda.get_device_properties(self.dev).multi_processor_count else 0
        # CTAs that share an attention unit's pages.  A prefill tile's shares are 64 rows each to merge: no more CTAs than are
        # resident at once (8 shares of 64 tiles took 31 us at four pages and 46 at 31 pages); a decode unit's are 4 or 8
        # rows, and two waves of CTAs even out sequences of different lengths
        tile = 64 // cfg.group          # rows of one prefill attention unit
        units = cfg.n_kv_heads * (-(-B // tile) if self.SHARED_CACHE else B)
        self.n_splits = self._splits(units, 2 if self.SHARED_CACHE else 4, self.max_pages)
        self.pages_per_split = -(-self.max_pages // self.n_splits)
        self.state_words = isa.ST_PAGETABLE + self.max_pages
        self.state = z(B, self.state_words, dt=torch.int32)
        self.state_host = torch.zeros(B, self.state_words, dtype=torch.int32).pin_memory()
        self.token_log = z(B, max_steps, dt=torch.int32)
        self._alloc_cache(page_perm_seed)
        self.taps_enabled = taps
        if taps:
            self.taps = z(L, Bp * H)
        self._cur = 0
        self.positions = [0] * B

    def _alloc_cache(self, page_perm_seed):
        """Paged pools and page tables: every sequence owns max_pages pages of one pool."""
        cfg, B, L = self.cfg, self.batch, self.cfg.n_layers
        z = lambda *s: torch.zeros(*s, dtype=BF16, device=self.dev)
        self.kpool = z(L, B * self.max_pages, cfg.n_kv_heads, isa.KV_PAGE, isa.HEAD_DIM)
        self.vpool = z(L, B * self.max_pages, cfg.n_kv_heads, isa.KV_PAGE, isa.HEAD_DIM)
        tables = []
        for b in range(B):
            if page_perm_seed is None:
                t = torch.arange(self.max_pages, dtype=torch.int32)
            else:
                t = torch.randperm(self.max_pages, generator=torch.Generator().manual_seed(page_perm_seed + b)).to(torch.int32)
            tables.append(t + b * self.max_pages)
        self.page_tables = torch.stack(tables)        # [B, max_pages] global page ids

    # ------------------------------------------------------------------ weights
    def load_weights(self, w):
        self._pack_cache = None         # packed copies of the previous weights
        super().load_weights(w)

    def init_random_weights(self, seed: int = 0, std: float = 0.02):
        self._pack_cache = None
        super().init_random_weights(seed, std)

    def weight_bytes(self) -> int:
        ts = [self.lm_head, self.norm_w, self.ln1, self.ln2, self.wqkv, self.wo, self.wgu, self.wd]
        ts += list(self.scales.values())
        return sum(t.numel() * t.element_size() for t in ts)

    def algorithmic_bytes(self, pos: int) -> int:
        """HBM bytes of one step with every sequence at position `pos`: each weight once, one
        embedding row and the KV rows of pos+1 positions per sequence."""
        cfg = self.cfg
        return self.weight_bytes() + self.batch * (cfg.hidden * 2 + 2 * cfg.kv_width * 2 * (pos + 1) * cfg.n_layers)

    # ------------------------------------------------------------------ program
    def _splits(self, units: int, per_sm: int, most: int) -> int:
        """CTAs (one cluster) that share a unit: the largest power of two with at most per_sm CTAs for every SM (one where
        no more CTAs than SMs may run at a time)."""
        s, per_sm = 1, 1 if self.max_ctas else per_sm
        while s < 8 and units * s * 2 <= per_sm * self.num_sms and s * 2 <= most:
            s *= 2
        return s

    def _gemm(self, name, l, w, x, mode, **kw):
        """Projection stage over layer l's matrix `name` ("lm": the vocabulary projection, bf16 in every engine)."""
        wf = self.wkind if name != "lm" else "bf16"
        K = {"wo": self.cfg.q_width, "wd": self.cfg.ffn}.get(name, self.cfg.hidden)
        if (name, l) not in self._pack_cache:     # the programs of one engine share the packed copies
            self._pack_cache[name, l] = {"bf16": lambda: pack_blocks(w, isa.STAGE_BLOCK),
                                         "fp8": lambda: pack_blocks_fp8(w, isa.STAGE_BLOCK),
                                         "nvfp4": lambda: pack_blocks_nvfp4(w, K, isa.STAGE_BLOCK)}[wf]()
        blocks = -(-w.shape[0] // isa.STAGE_BLOCK)
        return runtime.Stage(
            kind=isa.STAGE_GEMM, mode=mode, wfmt={"bf16": 0, "fp8": 1, "nvfp4": 2}[wf], B=self.batch, Bpad=self.bpad,
            M=w.shape[0], K=K, splits=self._splits(blocks, 2, K // 64), w=self._pack_cache[name, l].data_ptr(),
            scales=self.scales[name][l].data_ptr() if wf != "bf16" else 0, x=x.data_ptr(), **kw)

    def _plan(self, vocab: bool = True):
        """The stages of one step; vocab False: it ends after the last layer (prefill chunks before the last)."""
        cfg, B = self.cfg, self.batch
        L, G = cfg.n_layers, cfg.group
        hid = self.hidden.data_ptr()
        norm = lambda i, w: runtime.Stage(kind=isa.STAGE_NORM, B=B, Bpad=self.bpad, K=cfg.hidden, x=hid, out=self.normed.data_ptr(),
                                          stats_in=stat(i), norm_w=w.data_ptr(), eps=cfg.eps)
        stat = lambda i: self.stats[i].data_ptr()
        state = dict(state=self.state.data_ptr(), state_stride=self.state_words)
        heads = dict(group=G, n_kv=cfg.n_kv_heads, **state)
        out = [runtime.Stage(kind=isa.STAGE_EMBED, B=B, Bpad=self.bpad, M=cfg.vocab, K=cfg.hidden, w=self.embed.data_ptr(), hid=hid,
                             stats_out=stat(0), n_stats=2 * L + 1, **state)]
        attn_kind = isa.STAGE_ATTN_PREFILL if self.SHARED_CACHE else isa.STAGE_ATTN
        for l in range(L):
            pools = dict(kpool=self.kpool[l].data_ptr(), vpool=self.vpool[l].data_ptr())
            out.append(norm(2 * l, self.ln1[l]))
            out.append(self._gemm("wqkv", l, self.wqkv[l], self.normed, isa.STAGE_QKV, out=self.q.data_ptr(),
                                  rope=self.rope.data_ptr(), qk_norm=self.qknorm[l].data_ptr() if cfg.qk_norm else 0,
                                  qk_eps=cfg.qk_norm_eps, **heads, **pools))
            out.append(runtime.Stage(kind=attn_kind, B=B, Bpad=self.bpad, splits=self.n_splits, n_pages=self.max_pages,
                                     q=self.q.data_ptr(), out=self.attn_out.data_ptr(), **heads, **pools))
            out.append(self._gemm("wo", l, self.wo[l], self.attn_out, isa.STAGE_RESID, hid=hid,
                                  stats_out=stat(2 * l + 1)))
            out.append(norm(2 * l + 1, self.ln2[l]))
            out.append(self._gemm("wgu", l, self.wgu[l], self.normed, isa.STAGE_SILU, out=self.act.data_ptr()))
            out.append(self._gemm("wd", l, self.wd[l], self.act, isa.STAGE_RESID, hid=hid, stats_out=stat(2 * l + 2)))
            if self.taps_enabled:
                out.append(runtime.Stage(kind=isa.STAGE_COPY, x=hid, out=self.taps[l].data_ptr(), M=self.hidden.numel(), K=2))
        if vocab:
            out.append(norm(2 * L, self.norm_w))
            out.append(self._gemm("lm", 0, self.lm_head, self.normed, isa.STAGE_ARGMAX, keys=self.keys.data_ptr()))
            out.append(runtime.Stage(kind=isa.STAGE_ADVANCE, B=B, Bpad=self.bpad, keys=self.keys.data_ptr(),
                                     log=self.token_log.data_ptr(), log_stride=self.max_steps, **state))
        return (runtime.Stage * len(out))(*out)

    def _build_program(self):
        self._pack_cache = getattr(self, "_pack_cache", None) or {}
        self.stages = self._plan()
        self.launches_per_step = runtime.count_stage_launches(self.stages, self.max_ctas)[0]

    # ------------------------------------------------------------------ state
    def set_state(self, pos: int, token: int, b: int = None):
        """Sequence b (default: the one being prefilled) has positions [0, pos) cached and decodes `token` next."""
        b = self._cur if b is None else b
        assert pos < self.max_seq
        s = self.state_host[b]
        s.zero_()
        page = pos // isa.KV_PAGE
        table = self.page_tables[b]
        s[isa.ST_POS] = pos
        s[isa.ST_NPAGES] = page + 1
        s[isa.ST_TOKEN] = token
        s[isa.ST_NEWROW] = int(table[page]) * isa.KV_PAGE * self.cfg.n_kv_heads + pos % isa.KV_PAGE
        s[isa.ST_NKVH] = self.cfg.n_kv_heads
        s[isa.ST_MAXPAGES] = self.max_pages
        s[isa.ST_PAGETABLE:] = table
        self.state[b].copy_(s, non_blocking=True)
        self.keys.zero_()
        self.stats.zero_()
        self.positions[b] = pos
        self.pos = max(self.positions)
        self.steps_done = 0

    def load_kv(self, k: List[torch.Tensor], v: List[torch.Tensor], b: int = None):
        """Fills sequence b's pages from per-layer contiguous caches [T, n_kv_heads, 128]."""
        b = self._cur if b is None else b
        cfg = self.cfg
        pt = self.page_tables[b].long().to(self.dev)
        for l in range(cfg.n_layers):
            for src, pool in ((k[l], self.kpool[l]), (v[l], self.vpool[l])):
                T = src.shape[0]
                n_pages = (T + isa.KV_PAGE - 1) // isa.KV_PAGE
                pad = torch.zeros(n_pages * isa.KV_PAGE, cfg.n_kv_heads, isa.HEAD_DIM, dtype=BF16, device=self.dev)
                pad[:T] = src.to(self.dev)
                pool[pt[:n_pages]] = kv_page_swizzle(
                    pad.view(n_pages, isa.KV_PAGE, cfg.n_kv_heads, isa.HEAD_DIM).permute(0, 2, 1, 3))

    def read_kv(self, layer: int, T: int, b: int = 0):
        n_pages = (T + isa.KV_PAGE - 1) // isa.KV_PAGE
        pt = self.page_tables[b].long().to(self.dev)[:n_pages]
        out = []
        for pool in (self.kpool[layer], self.vpool[layer]):
            t = kv_page_swizzle(pool[pt]).permute(0, 2, 1, 3).reshape(n_pages * isa.KV_PAGE, self.cfg.n_kv_heads, isa.HEAD_DIM)
            out.append(t[:T])
        return out

    def read_hidden(self, flat: torch.Tensor) -> torch.Tensor:
        """A k-chunk-major [Bpad, hidden] matrix as [batch, hidden] (tests)."""
        return unpack_kc(flat, self.bpad, self.cfg.hidden)[:self.batch]

    @torch.no_grad()
    def prefill(self, tokens: torch.Tensor) -> List[int]:
        """tokens [batch, T]: each prompt goes through the PyTorch prefill; returns the first greedy tokens."""
        assert tokens.shape[0] == self.batch
        out = []
        for b in range(self.batch):
            self._cur = b
            out.append(DecodeEngine.prefill(self, tokens[b]))
        return out

    # ------------------------------------------------------------------ decode
    def step_async(self):
        """Enqueues one decode step (its stages, one kernel each); no synchronisation."""
        assert self.stages is not None, "load weights first"
        if self.pos >= self.max_seq or self.steps_done >= self.max_steps:
            raise RuntimeError("out of KV pages or token-log space")
        runtime.launch_stages(self.stages, self.stream.cuda_stream, self.timeout_ns, self.max_ctas)
        self.pos += 1
        self.steps_done += 1

    def generate(self, n_steps: int) -> List[List[int]]:
        """n_steps greedy steps, device resident; returns [n_steps][batch] token ids."""
        first = self.steps_done
        for _ in range(n_steps):
            self.step_async()
        runtime.read_status(self.stream.cuda_stream)
        self.positions = [p + n_steps for p in self.positions]
        return self.token_log[:, first:first + n_steps].t().tolist()

    def step_host(self, tokens: List[int]) -> List[int]:
        """One step driven from host buffers: batch token ids go up, the next ids come back."""
        if not hasattr(self, "_tok_in"):
            self._tok_in = torch.zeros(self.batch, dtype=torch.int32).pin_memory()
            self._tok_out = torch.zeros(self.batch, dtype=torch.int32).pin_memory()
        self._tok_in.copy_(torch.as_tensor(tokens, dtype=torch.int32))
        self.state[:, isa.ST_TOKEN].copy_(self._tok_in, non_blocking=True)
        idx = self.steps_done
        self.step_async()
        self._tok_out.copy_(self.token_log[:, idx], non_blocking=True)
        runtime.read_status(self.stream.cuda_stream)
        self.positions = [p + 1 for p in self.positions]
        return self._tok_out.tolist()
