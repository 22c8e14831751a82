"""Prefill on the device: a chunk of consecutive prompt positions per list of stage kernels.

The batched decode step (batch.BatchDecodeEngine) already computes, for every row of its batch, exactly what a prompt
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
from .decode import DecodeEngine


class PrefillEngine(BatchDecodeEngine):
    """`chunk` prompt positions per list of stages into the KV pools of `target` (a DecodeEngine of the same model)."""
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

    def launches(self, T: int) -> int:
        """Kernels a prompt of T tokens takes."""
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

    @torch.no_grad()
    def prefill(self, tokens: torch.Tensor, set_target_state: bool = True) -> int:
        """Runs the prompt, ceil(T / chunk) lists of stages, and returns the first generated (greedy) id.  A chunk's state
        blocks are prepared in pinned memory while the GPU runs the chunks before it, BLOCKS of them at most: every row of a
        block carries the page table, and a place per chunk would grow with the square of the prompt."""
        T, B = int(tokens.numel()), self.batch
        assert 1 <= T < self.max_seq and self.stages is not None
        n = (T + B - 1) // B
        ids = tokens.cpu().to(torch.int32).numpy().reshape(-1)
        blocks = torch.empty(min(n, self.BLOCKS), B, self.state_words, dtype=torch.int32, pin_memory=True)
        k = len(blocks)
        copied = [torch.cuda.Event() for _ in blocks] if n > k else None
        self.keys.zero_()
        with torch.cuda.stream(self.stream):
            for c in range(n):
                if c >= k:
                    copied[c % k].synchronize()         # the chunk that had this block has been copied
                self._fill_states(blocks[c % k].numpy(), ids, c)
                self.state.copy_(blocks[c % k], non_blocking=True)
                if copied:
                    copied[c % k].record(self.stream)
                runtime.launch_stages(self.stages if c == n - 1 else self._body, self.stream.cuda_stream, self.timeout_ns,
                                      self.max_ctas)
        runtime.read_status(self.stream.cuda_stream)
        first = int(self.token_log[(T - 1) % B, 0])
        if set_target_state:
            self.target.set_state(T, first)
        return first
