"""Prefill on the device: the prompt's positions as rows of stage kernels.

A prompt longer than a chunk goes through a layer with all its rows together, up to isa.WIDE_ROWS of them
(csrc/wide_kernels.cu): the weights are read once and the tensor cores are the bound.  On a part of the SMs (num_sms below the
device's), or without room for those rows' buffers, it goes chunk by chunk through the batched step's stages instead.

The chunks: the batched decode step (batch.BatchDecodeEngine) already computes, for every row of its batch, exactly what a prompt
position needs; what differs in a prefill is that the rows are consecutive positions of ONE sequence.  PrefillEngine
therefore gives every row the same page table and position pos0 + b.  The QKV projection's epilogue writes the normed,
rotated key rows and the value rows of all the chunk's positions to the paged pools, so the attention behind it finds
the rows of every earlier position of its own chunk in HBM; its units are tiles of 64 query rows (64 / G positions times
the G heads of a KV head) that share one walk over the pages, with the causal mask applied in the pages at the diagonal.
The pools and the page table are those of the decode engine the prompt is prefilled for: nothing is copied when decode
takes over.

The reference has no prefill of its own on the device either side of its decode schedules: its correctness runs
take the prompt's cache from a HuggingFace forward (app/python/llama3/sched.py:574-622 in the reference); this
engine replaces the PyTorch prefill of decode.DecodeEngine.prefill on the product path."""
import numpy as np
import torch

from . import isa, runtime
from .batch import BatchDecodeEngine
from .decode import BF16, DecodeEngine

STAGE = np.dtype(runtime.Stage)


class PrefillEngine(BatchDecodeEngine):
    """Prompts into the KV pools of `target` (a DecodeEngine of the same model).  `chunk` rows at most go through the batched
    step's stages at a time; it bounds neither the rows of a longer prompt's launches nor what the engine holds for them, which
    is the buffers of WideStages: for an 8B shape 176 MB, when max_seq is 2048 or more."""
    SHARED_CACHE = True
    BLOCKS = 4          # chunks whose state blocks may wait in host memory

    def __init__(self, target: DecodeEngine, chunk: int = 64, timeout_ns: int = 2_000_000_000):
        assert not isinstance(target, BatchDecodeEngine) and not target.cfg.n_experts
        self.target = target
        super().__init__(target.cfg, chunk, target.max_seq, device=target.dev, num_sms=target.num_sms,
                         max_steps=1, timeout_ns=timeout_ns, wkind=target.wkind)
        self.rope = target.rope

    def _alloc_cache(self, page_perm_seed):
        t = self.target
        self.kpool, self.vpool = t.kpool, t.vpool
        self.page_table = t.page_table
        self.page_tables = t.page_table[None, :].expand(self.batch, -1).contiguous()

    def adopt_weights(self):
        """Takes the target's tensors (embedding, norms, vocabulary projection, the layer projections in their
        stored form: bf16 rows, e4m3 codes or NVFP4 rows, with their scales) and packs the projections for the
        tensor-core tasks; both engines store a projection the same way, only the packing differs."""
        t = self.target
        for name in ("embed", "lm_head", "norm_w", "ln1", "ln2", "qknorm", "wqkv", "wo", "wgu", "wd"):
            setattr(self, name, getattr(t, name))
        self.router, self.scales, self.w = None, dict(t.scales), True
        self._pack_cache = None
        self._build_program()
        return self

    def _build_program(self):
        """Two lists of stages over the same packed weights: chunks before the prompt's last end after the last layer,
        the last chunk adds the final norm, the vocabulary projection and the argmax (the first generated id)."""
        super()._build_program()
        self._body = self._plan(vocab=False)
        self._wide = None
        if not self.max_ctas and self.max_seq - 1 > self.batch:      # otherwise no prompt is longer than a chunk
            try:
                self._wide = WideStages(self)
            except torch.cuda.OutOfMemoryError:
                pass                                                 # prompts go chunk by chunk
        self._first = torch.zeros(1, dtype=torch.int32).pin_memory()

    def launches(self, T: int) -> int:
        """Kernels a prompt of T tokens takes."""
        if self._goes_wide(T):
            return self._wide.launches(T)
        body, last = (runtime.count_stage_launches(s, self.max_ctas)[0] for s in (self._body, self.stages))
        return (T - 1) // self.batch * body + last

    # ------------------------------------------------------------------ chunks
    def _fill_states(self, s, tokens, c: int):
        """State blocks of chunk c into the int32 array s [chunk, state_words]: row b is position c * chunk + b (rows past
        the prompt's end repeat its last position; the first of them writes the cache row)."""
        pos = np.minimum(np.arange(c * self.batch, (c + 1) * self.batch), len(tokens) - 1)
        page = pos // isa.KV_PAGE
        table = self.page_table.numpy()
        s[:, :isa.ST_PAGETABLE] = 0
        s[:, isa.ST_POS] = pos
        s[:, isa.ST_NPAGES] = page + 1
        s[:, isa.ST_TOKEN] = tokens[pos]
        s[:, isa.ST_NEWROW] = table[page] * (isa.KV_PAGE * self.cfg.n_kv_heads) + pos % isa.KV_PAGE
        s[:, isa.ST_NKVH] = self.cfg.n_kv_heads
        s[:, isa.ST_MAXPAGES] = self.max_pages
        s[:, isa.ST_PAGETABLE:] = table

    def _goes_wide(self, T: int) -> bool:
        return self._wide is not None and T > self.batch

    @torch.no_grad()
    def prefill(self, tokens: torch.Tensor, set_target_state: bool = True) -> int:
        """Runs the prompt and returns the first generated (greedy) id.  What the host sends (ids, state blocks) is prepared in
        pinned memory while the GPU runs what was sent before it, in BLOCKS blocks at most: every row of a chunk's block carries
        the page table, and a place per chunk would grow with the square of the prompt."""
        T, B = int(tokens.numel()), self.batch
        assert 1 <= T < self.max_seq and self.stages is not None
        n = (T + B - 1) // B
        wide = self._goes_wide(T)
        ids = tokens.cpu().to(torch.int32).numpy().reshape(-1)
        blocks = torch.empty(min(n, self.BLOCKS), B, self.state_words, dtype=torch.int32, pin_memory=True)
        k, sent = len(blocks), 0
        # a block's place is waited for only where it is used a second time
        copied = [torch.cuda.Event() for _ in blocks] if (self._wide.sends(T) + 1 if wide else n) > k else None

        def send(fill, dst):
            """The next block, filled by fill(numpy view), into dst; its place is free again when it has been copied."""
            nonlocal sent
            if sent >= k:
                copied[sent % k].synchronize()
            block = blocks[sent % k]
            fill(block.numpy())
            dst.copy_(block.view(-1)[:dst.numel()].view(dst.shape), non_blocking=True)
            if copied:
                copied[sent % k].record(self.stream)
            sent += 1
        launch = lambda stages: runtime.launch_stages(stages, self.stream.cuda_stream, self.timeout_ns, self.max_ctas)
        with torch.cuda.stream(self.stream):
            if wide:
                self._wide.run(ids, send, launch)
            self.keys.zero_()
            for c in range(n - 1 if wide else 0, n):
                send(lambda s: self._fill_states(s, ids, c), self.state)
                launch(self._wide.last if wide else self.stages if c == n - 1 else self._body)
            self._first.copy_(self.token_log[(T - 1) % B, :1], non_blocking=True)
        runtime.read_status(self.stream.cuda_stream)
        first = int(self._first)
        if set_target_state:
            self.target.set_state(T, first)
        return first


def batched_projection(name: str, M: int, K: int, fmt: int, splits: int) -> bool:
    """Whether 128 rows of a prompt go through a layer's M x K projection as a stage of the batched step (`splits` CTAs to a block
    of its rows) and not as wide tiles.  What bounds 128 rows of a large projection is the weights, and the stage's two CTAs per SM
    bring them faster than a wide tile's one; where there are few of them it is its cluster's exchange and its longer prologue.
    What a layer of 100 rows gains from the one in place of the other (us, B200, weights from HBM; from L2 within 1 us of it):
      bf16   wo 4096 x 4096  6.2, wd 4096 x 14336  8.1, 2048 x 1024  1.2, 1024 x 3072  0.1, 1024 x 1024  -0.3, 512 x 1024  -0.8
             gate/up 8192 x 4096  12.7, 12288 x 2048  2.3, 6144 x 1024  0.2, 8192 x 512  -1.9
      e4m3   wo 4096 x 4096  13.4, wd 4096 x 14336  20.9, wo 2048 x 2048  5.1, wd 2048 x 1024  -0.7, 1024 x 3072  -1.0, 512 x 1024  -1.1
             gate/up 28672 x 4096  12.1, 12288 x 2048  5.1, 6144 x 1024  0.6, 2048 x 512  -3.9     (NVFP4 up to 4 us more, 28672 x 4096
             18.8)
    A bf16 gate/up of more blocks than SMs leaves some SMs two CTAs of whole rows (24576 x 4096  -5.3, 28672 x 4096  -3.8).  QKV sums
    come from wide tiles as fast or faster everywhere (6144 x 4096 bf16 -1.7, e4m3 -2.0, NVFP4 -0.4; 1536 x 1024  -3.1, -3.7, -3.7): the
    tiles' K ranges leave several sums of a value, for each of which heads take 0.1 us more and a norm 0.5."""
    return name != "wqkv" and M >= 2048 and (K >= 1024 and splits > 1 if fmt == 0 else K >= 2048)


class WideStages:
    """Buffers and stages of a prompt whose rows go through a layer together.  Rows are taken in passes of `rows` (whole chunks
    of the engine, at most isa.WIDE_ROWS); a pass over R rows (a multiple of 128) has a list of stages of its own."""
    HEADER = isa.ST_PAGETABLE       # words in front of the page table

    def __init__(self, e: PrefillEngine):
        self.e, cfg, dev = e, e.cfg, e.dev
        B, H, F, Q = e.batch, cfg.hidden, cfg.ffn, cfg.q_width
        self.rows = min(isa.WIDE_ROWS, -(-e.max_seq // B) * B) // B * B
        self.sms = torch.cuda.get_device_properties(dev).multi_processor_count
        self.fmt = {"bf16": 0, "fp8": 1, "nvfp4": 2}[e.wkind]
        R = -(-self.rows // 128) * 128
        z = lambda n, dt=BF16: torch.empty(n, dtype=dt, device=dev)
        self.hidden, self.normed, self.attn, self.act, self.q = z(R * H), z(R * H), z(R * Q), z(R * F), z(R * Q)
        # every K-split leaves sums of its own: at most 8, and no more than make 2048 rows of them (runtime.wide_tiles)
        self.sums = z(max(R, min(8 * R, 2048)) * max(e.qkv_rows, H), torch.float32)
        self.block = z(self.HEADER + e.max_pages + self.rows, torch.int32)       # header, page table, ids
        self.table = e.page_table.numpy()
        self.template, self.places = self._plan()
        self.lists = {r: self._stages(r) for r in range(128, R + 1, 128)}
        # what follows the last layer: the last chunk's rows, then the chunk's own final stages
        tail = runtime.Stage(kind=isa.STAGE_WIDE_TAIL, B=B, Bpad=e.bpad, K=H, x=self.hidden.data_ptr(), hid=e.hidden.data_ptr(),
                             stats_out=e.stats[2 * cfg.n_layers].data_ptr(), state=self.block.data_ptr())
        final = list(e.stages)[-3:]
        self.last = (runtime.Stage * 4)(tail, *final)

    def launches(self, T: int) -> int:
        passes = -(-T // self.rows)
        return passes * len(self.template) + len(self.last)

    def _plan(self):
        """The stages of a pass without what depends on its rows, and the places of each projection and of its sums' reader."""
        e, cfg = self.e, self.e.cfg
        H, F, Q = cfg.hidden, cfg.ffn, cfg.q_width
        hid, normed, sums, state, attn, act = (t.data_ptr() for t in (self.hidden, self.normed, self.sums, self.block, self.attn, self.act))
        S = runtime.Stage
        heads = dict(group=cfg.group, n_kv=cfg.n_kv_heads, state=state)

        def gemm(name, l, M, K, x, out):
            return S(kind=isa.STAGE_WIDE_GEMM, mode=isa.STAGE_SILU if name == "wgu" else isa.STAGE_SUMS, wfmt=self.fmt, M=M, K=K,
                     w=e._pack_cache[name, l].data_ptr(), x=x, out=out, scales=e.scales[name][l].data_ptr() if self.fmt else 0)
        norm = lambda w, out, x: S(kind=isa.STAGE_WIDE_NORM, K=H, hid=hid, out=out, norm_w=w.data_ptr(), eps=cfg.eps, x=x, splits=1)
        out = [S(kind=isa.STAGE_WIDE_EMBED, M=cfg.vocab, K=H, w=e.embed.data_ptr(), hid=hid, state=state,
                 log=state + 4 * (self.HEADER + e.max_pages))]
        for l in range(cfg.n_layers):
            pools = dict(kpool=e.kpool[l].data_ptr(), vpool=e.vpool[l].data_ptr())
            out += [norm(e.ln1[l], normed, sums if l else 0),
                    gemm("wqkv", l, e.qkv_rows, H, normed, sums),
                    S(kind=isa.STAGE_WIDE_HEADS, M=e.qkv_rows, x=sums, out=self.q.data_ptr(), rope=e.rope.data_ptr(),
                      qk_norm=e.qknorm[l].data_ptr() if cfg.qk_norm else 0, qk_eps=cfg.qk_norm_eps, **heads, **pools),
                    S(kind=isa.STAGE_WIDE_ATTN, n_pages=e.max_pages, q=self.q.data_ptr(), out=attn, **heads, **pools),
                    gemm("wo", l, H, Q, attn, sums),
                    norm(e.ln2[l], normed, sums),
                    gemm("wgu", l, 2 * F, H, normed, act),
                    gemm("wd", l, H, F, act, sums)]
        out.append(norm(e.norm_w, 0, sums))
        # place of a layer's first stage, then of the projection and the reader of its sums (0: none) from there
        places = {"wqkv": (1, 2, e.qkv_rows, H), "wo": (4, 5, H, Q), "wgu": (6, 0, 2 * F, H), "wd": (7, 8, H, F)}
        return (S * len(out))(*out), places

    def _stages(self, R: int):
        """The stages of a pass over R rows."""
        e, cfg = self.e, self.e.cfg
        arr = type(self.template).from_buffer_copy(self.template)
        v = np.frombuffer(arr, dtype=STAGE)
        v["Bpad"] = R
        n = 8 * cfg.n_layers
        v["splits"][1 + 3:1 + n:8] = e._splits(cfg.n_kv_heads * (R // (64 // cfg.group)), 2, e.max_pages)
        for name, (at, reader, M, K) in self.places.items():
            splits, ks = e._splits(-(-M // isa.STAGE_BLOCK), 2, K // 64), 1
            if R == 128 and batched_projection(name, M, K, self.fmt, splits):
                v["kind"][1 + at:1 + n:8], v["B"][1 + at:1 + n:8], v["splits"][1 + at:1 + n:8] = isa.STAGE_GEMM, R, splits
            else:
                subs, cols, ks = runtime.wide_tiles(R, M, K, self.fmt, self.sms, name == "wgu")
                v["group"][1 + at:1 + n:8], v["n_kv"][1 + at:1 + n:8], v["splits"][1 + at:1 + n:8] = subs, cols, ks
            if reader:
                v["splits"][1 + reader:2 + n:8] = ks
        return arr

    def sends(self, T: int) -> int:
        """Blocks of the engine's pinned memory that a prompt's ids and page tables take."""
        at, piece = self.HEADER + self.e.max_pages, self.e.batch * self.e.state_words
        return sum(-(-(at + min(self.rows, T - p0)) // piece) for p0 in range(0, T, self.rows))

    def run(self, ids, send, launch):
        """All layers over the prompt's ids; send and launch are PrefillEngine.prefill's."""
        at = self.HEADER + self.e.max_pages
        for p0 in range(0, len(ids), self.rows):
            part = ids[p0:p0 + self.rows]
            words = np.zeros(at + len(part), dtype=np.int32)
            words[isa.WIDE_POS], words[isa.WIDE_N] = p0, len(part)
            words[isa.ST_PAGETABLE:at] = self.table
            words[at:] = part
            piece = self.e.batch * self.e.state_words       # a block of the engine's pinned memory
            for w0 in range(0, len(words), piece):
                w = words[w0:w0 + piece]

                def fill(s, w=w):
                    s.reshape(-1)[:len(w)] = w
                send(fill, self.block[w0:w0 + len(w)])
            launch(self.lists[-(-len(part) // 128) * 128])
        n = len(ids)
        self.last[0].M = (n - 1) // self.e.batch * self.e.batch % self.rows      # the last chunk's first row in its pass
