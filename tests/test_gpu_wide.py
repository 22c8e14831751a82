"""The stages of a whole prompt (csrc/wide_kernels.cu): the projection at the edges of its tiles against an fp32 matmul, and
prompts whose rows go through a layer together against the same prompts chunk by chunk."""
import pytest
import torch

from tests.test_gpu_stages import rel, seeded, weights

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _rows(x):
    """[R, K] -> sub-matrices of 128 rows, each k-chunk-major"""
    from vdcores_b200.batch import pack_kc
    return torch.cat([pack_kc(x[r:r + 128]) for r in range(0, x.shape[0], 128)])


@pytest.mark.parametrize("fmt", ["bf16", "fp8", "nvfp4"])
@pytest.mark.parametrize("R,M,K,subs,cols,splits", [
    (128, 16, 64, 1, 16, 1),            # the smallest tile, one chunk
    (128, 272, 1024, 1, 48, 3),         # tiles across a block's edge, the last block and tile smaller, uneven K ranges
    (384, 400, 512, 2, 240, 2),         # a last row tile of one sub-matrix; tiles over three blocks
    (256, 4096, 1024, 2, 256, 1),
    (640, 6144, 2048, 2, 176, 1),       # several tiles per CTA
    (2048, 1024, 4096, 1, 80, 8)])      # both accumulators of one-sub-matrix tiles in turn, many times
def test_prompt_projection(cuda_device, fmt, R, M, K, subs, cols, splits):
    from vdcores_b200 import isa, runtime
    dev = cuda_device
    x = seeded((R, K), 1).to(dev)
    w, sc, ref = weights(M, K, fmt, dev)
    xd = _rows(x)
    sums = torch.full((splits, M // 4, R, 4), float("nan"), device=dev)
    act = torch.full((R * M // 2,), float("nan"), device=dev, dtype=BF16)
    kw = dict(kind=isa.STAGE_WIDE_GEMM, wfmt={"bf16": 0, "fp8": 1, "nvfp4": 2}[fmt], Bpad=R, M=M, K=K, group=subs, n_kv=cols,
              w=w.data_ptr(), scales=sc.data_ptr() if sc is not None else 0, x=xd.data_ptr())
    arr = (runtime.Stage * 2)(runtime.Stage(mode=isa.STAGE_SUMS, splits=splits, out=sums.data_ptr(), **kw),
                              runtime.Stage(mode=isa.STAGE_SILU, splits=1, out=act.data_ptr(), **kw))
    s = torch.cuda.current_stream(dev).cuda_stream
    runtime.launch_stages(arr, s, 500_000_000)
    runtime.read_status(s)
    y = x.double() @ ref.to(dev).double().t()
    got = sums.sum(0).permute(1, 0, 2).reshape(R, M)
    # the tensor cores add K / 16 products of 16 to an fp32 sum, each addition exact to 2^-23 of it (twice that where cut off)
    assert rel(got, y) < 2 * K / 16 * 2.0 ** -23 + 1e-6
    g, u = y[:, 0::2].float().to(BF16).float(), y[:, 1::2].float().to(BF16).float()
    want = torch.nn.functional.silu(g).to(BF16).float() * u
    rows = torch.cat([a.view(M // 16, 16, 8, 8).permute(1, 2, 0, 3).reshape(128, M // 2) for a in act.view(R // 128, -1)])
    assert rel(rows, want) < 4e-3       # three bf16 roundings of 2^-9 each


@pytest.mark.parametrize("kind,fmt,T,chunk,perm", [("llama", "bf16", 77, 64, 3), ("llama", "bf16", 129, 128, None),
                                                   ("qwen3", "bf16", 300, 48, 5), ("llama", "fp8", 257, 16, None),
                                                   ("qwen3_1k", "nvfp4", 515, 128, 1), ("llama", "bf16", 2200, 120, 2)])
def test_prompt_in_one_pass_agrees_with_its_chunks(cuda_device, kind, fmt, T, chunk, perm):
    """Ragged prompts, shuffled pages, chunks that do not divide 128, prompts of two passes: cache rows of every layer, the last
    chunk's hidden rows (its repeated ones too) and the first id."""
    from tests.helpers import engine_config, small_cfg
    _one_pass_against_chunks(cuda_device, engine_config(small_cfg(kind)), fmt, T, chunk, perm)


def _one_pass_against_chunks(dev, cfg, fmt, T, chunk, perm):
    """The prompt's stages of one pass, when it has agreed."""
    from vdcores_b200.decode import DecodeEngine
    from vdcores_b200.prefill import PrefillEngine
    eng = DecodeEngine(cfg, (T + 70) // 64 * 64, device=dev, wkind=fmt, page_perm_seed=perm)
    eng.init_random_weights(3)
    prompt = torch.randint(0, cfg.vocab, (T,), generator=torch.Generator().manual_seed(T))
    pre = PrefillEngine(eng, chunk=chunk, timeout_ns=500_000_000).adopt_weights()
    lists = dict(pre._wide.lists)
    got = []
    for wide in (True, False):
        if not wide:
            pre._wide = None
        assert pre._goes_wide(T) == wide
        eng.kpool.zero_()
        eng.vpool.zero_()
        first = pre.prefill(prompt)
        assert not wide or pre._wide.lists == lists          # the first prompt of a length plans nothing
        hidden = pre.read_hidden(pre.hidden)
        # the id: the largest logit of the last row, where the next one is further off than roundings (2^-9 of the row's size)
        x = hidden[(T - 1) % chunk].float()
        x = (x * torch.rsqrt(x.pow(2).mean() + cfg.eps)).to(BF16) * eng.norm_w
        logits = x.float() @ eng.lm_head.float().t()
        top = torch.topk(logits, 2)
        clear = float(top.values[0] - top.values[1]) > 2.0 ** -7 * float(top.values[0].abs())
        assert first == int(top.indices[0]) or not clear
        got.append((first, hidden.clone(), eng.kpool.clone(), eng.vpool.clone(), clear))
    (f1, h1, k1, v1, clear1), (f0, h0, k0, v0, clear0) = got
    assert f1 == f0 or not (clear1 and clear0)
    assert bool(torch.isfinite(h1.float()).all())
    for a, b in ((h1, h0), (k1[1:], k0[1:]), (v1[1:], v0[1:])):
        assert rel(a, b) < 1e-2          # sums in other orders, rounded to bf16 through two or three layers
    for a, b in ((k1[0], k0[0]), (v1[0], v0[0])):
        assert rel(a, b) < 2e-3          # one projection behind exact inputs: a rounding here and there
        rows = (a.float() - b.float()).flatten(0, 2).norm(dim=1) / b.float().flatten(0, 2).norm(dim=1).clamp_min(1e-6)
        assert float(rows.max()) < 1e-2
    assert bool(((k1 == 0) == (k0 == 0)).float().mean() > 0.999)     # nothing written past the prompt
    return lists[-(-min(T, 2048) // 128) * 128]


@pytest.mark.parametrize("fmt,hidden,kv,ffn,T,chunk,batched", [
    ("fp8", 2048, 4, 2048, 77, 64, ("wo", "wgu", "wd")),
    ("nvfp4", 2048, 4, 2048, 128, 48, ("wo", "wgu", "wd")),
    ("fp8", 2048, 4, 1536, 65, 64, ("wo", "wgu")),      # inputs shorter than 2048; rows shorter than that
    ("fp8", 1024, 2, 3072, 70, 64, ()),
    ("nvfp4", 1024, 2, 3072, 120, 100, ()),
    ("bf16", 512, 1, 4096, 65, 64, ()),
    ("bf16", 1024, 2, 9472, 101, 64, ("wgu",)),         # 148 blocks of gate/up, 152
    ("bf16", 1024, 2, 9728, 128, 100, ()),
    ("bf16", 2048, 4, 1024, 90, 32, ("wo", "wgu", "wd"))])
def test_a_prompt_of_up_to_128_rows(cuda_device, fmt, hidden, kv, ffn, T, chunk, batched):
    """Projections as stages of the batched step and as wide tiles, on either side of what decides between them."""
    from vdcores_b200 import isa
    from vdcores_b200.decode import DecodeConfig
    cfg = DecodeConfig(hidden=hidden, n_heads=4 * kv, n_kv_heads=kv, head_dim=128, ffn=ffn, vocab=1024, n_layers=2, eps=1e-5, theta=5e5)
    stages = _one_pass_against_chunks(cuda_device, cfg, fmt, T, chunk, 3)
    for layer in range(2):
        for name, at in (("wqkv", 1), ("wo", 4), ("wgu", 6), ("wd", 7)):
            assert (stages[1 + 8 * layer + at].kind == isa.STAGE_GEMM) == (name in batched), name


def test_prompts_go_chunk_by_chunk_without_the_wide_buffers(cuda_device, monkeypatch):
    """No buffers are taken where no prompt is longer than a chunk, and none are needed where there is no room for them."""
    from tests.helpers import engine_config, small_cfg
    from vdcores_b200 import prefill
    from vdcores_b200.decode import DecodeEngine
    eng = DecodeEngine(engine_config(small_cfg("llama")), 65, device=cuda_device)
    eng.init_random_weights(3)
    prompt = torch.arange(3, 53)
    assert prefill.PrefillEngine(eng, chunk=64).adopt_weights()._wide is None
    wide = prefill.PrefillEngine(eng, chunk=32).adopt_weights()
    assert wide._goes_wide(50)
    want = wide.prefill(prompt), eng.kpool.clone()

    def no_room(self, e):
        raise torch.cuda.OutOfMemoryError
    monkeypatch.setattr(prefill.WideStages, "__init__", no_room)
    pre = prefill.PrefillEngine(eng, chunk=32).adopt_weights()
    assert not pre._goes_wide(50)
    eng.kpool.zero_()
    pre.prefill(prompt)
    assert rel(eng.kpool, want[1]) < 1e-2


def test_an_id_outside_the_vocabulary_ends_a_prompt_with_an_error(cuda_device):
    from tests.helpers import engine_config, small_cfg
    from vdcores_b200 import isa, runtime
    from vdcores_b200.decode import DecodeEngine
    from vdcores_b200.prefill import PrefillEngine
    eng = DecodeEngine(engine_config(small_cfg("llama")), 320, device=cuda_device)
    eng.init_random_weights(3)
    pre = PrefillEngine(eng, chunk=64, timeout_ns=500_000_000).adopt_weights()
    prompt = torch.randint(0, eng.cfg.vocab, (200,), generator=torch.Generator().manual_seed(5))
    first, keys = pre.prefill(prompt), eng.kpool.clone()
    for bad in (-1, eng.cfg.vocab, 2 ** 31 - 1):
        wrong = prompt.clone()
        wrong[130] = bad
        eng.set_state(7, 3)
        state = eng.state.clone()
        with pytest.raises(runtime.VdcError) as e:
            pre.prefill(wrong)
        assert e.value.code == 5 and e.value.status["pc"] == 130 and e.value.status["opcode"] == isa.STAGE_WIDE_EMBED
        assert e.value.status["aux"] == bad and torch.equal(eng.state, state)
    eng.kpool.zero_()
    assert pre.prefill(prompt) == first and torch.equal(eng.kpool, keys)


@pytest.mark.parametrize("fmt", ["bf16", "fp8"])
def test_a_wait_that_runs_out_ends_with_an_error(cuda_device, fmt):
    """Waits limited to a nanosecond: a projection ends as it should or with the timeout in the status block; the next launch
    with a proper limit is right."""
    from vdcores_b200 import isa, runtime
    dev, R, M, K = cuda_device, 256, 4096, 2048
    w, sc, _ = weights(M, K, fmt, dev)
    xd = _rows(seeded((R, K), 1).to(dev))
    out = torch.zeros(M // 4, R, 4, device=dev)
    s = runtime.Stage(kind=isa.STAGE_WIDE_GEMM, mode=isa.STAGE_SUMS, wfmt=int(fmt == "fp8"), Bpad=R, M=M, K=K, group=2, n_kv=128,
                      splits=1, w=w.data_ptr(), scales=sc.data_ptr() if sc is not None else 0, x=xd.data_ptr(), out=out.data_ptr())
    stream, want = torch.cuda.current_stream(dev).cuda_stream, None
    for i in range(21):
        out.zero_()
        runtime.launch_stages((runtime.Stage * 1)(s), stream, 1 if i % 2 else 500_000_000)
        try:
            runtime.read_status(stream)
        except runtime.VdcError as e:
            assert i % 2 and e.code == 1 and e.status["opcode"] == isa.STAGE_WIDE_GEMM
            continue
        want = out.clone() if want is None else want
        assert torch.equal(out, want)


@pytest.mark.parametrize("K,splits", [(512, 0), (4096, 1), (4096, 3), (5120, 2), (8192, 8)])
def test_norm_of_a_prompts_rows(cuda_device, K, splits):
    """Fewer pieces than threads, as many as stay in registers, more than those: the hidden state is the bf16 sum to the bit, its
    norm two bf16 roundings (2^-9 each) from fp32's."""
    from vdcores_b200 import isa, runtime
    dev, R = cuda_device, 128
    h, parts, w = seeded((R, K), 4).to(BF16).to(dev), seeded((max(splits, 1), R, K), 5).float().to(dev), (1 + 0.1 * seeded((K,), 6).float()).to(BF16).to(dev)
    hd, out = _rows(h), torch.zeros(R * K, dtype=BF16, device=dev)
    x = parts.permute(0, 2, 1).reshape(max(splits, 1), K // 4, 4, R).transpose(2, 3).contiguous()
    s = runtime.Stage(kind=isa.STAGE_WIDE_NORM, Bpad=R, K=K, hid=hd.data_ptr(), out=out.data_ptr(), norm_w=w.data_ptr(), eps=1e-5,
                      x=x.data_ptr() if splits else 0, splits=max(splits, 1))
    stream = torch.cuda.current_stream(dev).cuda_stream
    runtime.launch_stages((runtime.Stage * 1)(s), stream, 500_000_000)
    runtime.read_status(stream)
    want = h
    if splits:
        total = parts[0].clone()
        for p in parts[1:]:
            total += p
        want = (h.float() + total.to(BF16).float()).to(BF16)
    assert torch.equal(hd, _rows(want))
    norm = want.double() * torch.rsqrt(want.double().pow(2).mean(1, keepdim=True) + 1e-5) * w.double()
    assert rel(out.double(), _rows(norm.to(BF16)).double()) < 2 * 2.0 ** -9
