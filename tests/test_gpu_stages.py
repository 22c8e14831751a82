"""The stage kernels of a batched step one by one (runtime.launch_stages), at the sizes where a tile, a K-split or a page
walk can go wrong, against plain fp32 matmuls and softmaxes of the same bf16 inputs.

Bounds: a result rounded once to bf16 is within 2^-8 of the exact one per element, 2^-9 rms and less in the 2-norm; the
fp32 accumulation adds about 1e-6.  Rounding twice (bf16 product, then bf16 sum or norm weight) doubles that.  Attention
rounds the probabilities to bf16 as well (another 2^-9).  4e-3 covers each of them."""
import math

import pytest
import torch

from tests.test_gpu_ops import seeded

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
REL = 4e-3


def rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-20))


def bpad(B):
    return next(p for p in (16, 32, 64, 128) if B <= p)


def packed_rows(x, dev):
    from vdcores_b200.batch import pack_kc
    full = torch.zeros(bpad(x.shape[0]), x.shape[1], dtype=BF16)
    full[:x.shape[0]] = x
    return pack_kc(full.to(dev))


def run(dev, *stages):
    from vdcores_b200 import runtime
    arr = (runtime.Stage * len(stages))(*stages)
    runtime.launch_stages(arr, torch.cuda.current_stream(dev).cuda_stream, 500_000_000)
    runtime.read_status(torch.cuda.current_stream(dev).cuda_stream)


def weights(M, K, fmt, dev, seed=2):
    """(device tensor in the stages' layout, scales or None, the fp32 matrix it stands for)"""
    from vdcores_b200 import isa
    from vdcores_b200.batch import pack_blocks, pack_blocks_fp8, pack_blocks_nvfp4
    from vdcores_b200.decode import quantize_fp8_rows, quantize_nvfp4_rows
    w = seeded((M, K), seed, 0.05)
    if fmt == "bf16":
        return pack_blocks(w.to(dev), isa.STAGE_BLOCK), None, w.float()
    if fmt == "fp8":
        codes, sc = quantize_fp8_rows(w)
        return (pack_blocks_fp8(codes.to(dev), isa.STAGE_BLOCK), sc.to(dev),
                codes.view(torch.float8_e4m3fn).float() * sc[:, None])
    rows, ts = quantize_nvfp4_rows(w)
    grid = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
    grid = torch.cat((grid, -grid))
    codes, bs = rows[:, :K // 2], rows[:, K // 2:].contiguous().view(torch.float8_e4m3fn).float()
    vals = torch.stack((grid[(codes & 15).long()], grid[(codes >> 4).long()]), -1).view(M, K // 16, 16) * bs[..., None]
    return (pack_blocks_nvfp4(rows.to(dev), K, isa.STAGE_BLOCK), ts.expand(M).contiguous().to(dev), vals.view(M, K) * ts)


CASES = [(1, 256, 16, 4, "bf16"), (3, 512, 144, 8, "bf16"), (16, 4096, 256, 8, "bf16"), (40, 768, 400, 2, "bf16"),
         (128, 1024, 128, 1, "bf16"), (100, 14336, 128, 8, "bf16"), (2, 512, 48, 1, "fp8"), (33, 1024, 272, 4, "fp8"),
         (128, 4096, 128, 2, "fp8"), (5, 1024, 16, 8, "nvfp4"), (64, 2048, 272, 1, "nvfp4"), (128, 1024, 112, 2, "nvfp4")]


def gemm(dev, fmt, B, M, K, splits, w, sc, x, **kw):
    from vdcores_b200 import isa, runtime
    return runtime.Stage(kind=isa.STAGE_GEMM, wfmt={"bf16": 0, "fp8": 1, "nvfp4": 2}[fmt], B=B, Bpad=bpad(B), M=M, K=K,
                         splits=splits, w=w.data_ptr(), scales=sc.data_ptr() if sc is not None else 0, x=x.data_ptr(), **kw)


@pytest.mark.parametrize("B,K,M,splits,fmt", CASES)
def test_projection_with_residual(cuda_device, B, K, M, splits, fmt):
    from vdcores_b200 import isa
    from vdcores_b200.batch import unpack_kc
    dev, Bp = cuda_device, bpad(B)
    x, h = seeded((B, K), 1), seeded((B, M), 3)
    w, sc, wf = weights(M, K, fmt, dev)
    xd, hd = packed_rows(x, dev), packed_rows(h, dev)
    stats = torch.zeros(128, device=dev)
    run(dev, gemm(dev, fmt, B, M, K, splits, w, sc, xd, mode=isa.STAGE_RESID, hid=hd.data_ptr(), stats_out=stats.data_ptr()))
    ref = h.float() + x.float() @ wf.t()
    got = unpack_kc(hd.cpu(), Bp, M)
    assert rel(got[:B], ref) < REL and float(got[B:].abs().max() if B < Bp else 0) == 0
    assert torch.allclose(stats.cpu()[:B], got[:B].float().pow(2).sum(1), rtol=1e-4) and float(stats[B:].abs().sum()) == 0


@pytest.mark.parametrize("B,K,M,splits,fmt", CASES)
def test_projection_gate_up_and_argmax(cuda_device, B, K, M, splits, fmt):
    from vdcores_b200 import isa, runtime
    from vdcores_b200.batch import unpack_kc
    dev, Bp = cuda_device, bpad(B)
    x = seeded((B, K), 5)
    w, sc, wf = weights(M, K, fmt, dev, seed=6)
    stats = torch.zeros(128)
    stats[:B] = seeded((B,), 7).float().abs() * K + 1
    xd, sd, out = packed_rows(x, dev), stats.to(dev), torch.zeros(Bp * M // 2, dtype=BF16, device=dev)
    keys = torch.zeros(B, dtype=torch.int64, device=dev)
    nw = (1 + 0.1 * seeded((K,), 4).float()).to(BF16)
    nwd = nw.to(dev)
    xnd = torch.zeros_like(xd)
    norm = runtime.Stage(kind=isa.STAGE_NORM, B=B, Bpad=Bp, K=K, x=xd.data_ptr(), out=xnd.data_ptr(), stats_in=sd.data_ptr(),
                         norm_w=nwd.data_ptr(), eps=1e-5)
    run(dev, norm, gemm(dev, fmt, B, M, K, splits, w, sc, xnd, mode=isa.STAGE_SILU, out=out.data_ptr()))
    xn = (x.float() * torch.rsqrt(stats[:B, None] / K + 1e-5)).to(BF16).float() * nw.float()
    assert rel(unpack_kc(xnd.cpu(), Bp, K)[:B], xn) < REL
    y = xn.to(BF16).float() @ wf.t()
    yb = y.to(BF16).float()
    ref = torch.nn.functional.silu(yb[:, 0::2]) * yb[:, 1::2]
    assert rel(unpack_kc(out.cpu(), Bp, M // 2)[:B], ref) < 2 * REL
    if sc is not None:      # rows whose scales differ by more than their logits: the winner is the scaled one
        f = torch.where(torch.arange(M) % 3 == 0, 8.0, 1.0)
        sc, y = (sc.cpu() * f).to(dev), y * f
    run(dev, gemm(dev, fmt, B, M, K, splits, w, sc, xnd, mode=isa.STAGE_ARGMAX, keys=keys.data_ptr()))
    rows = 0xFFFFFFFF - (keys.cpu() & 0xFFFFFFFF)
    top = y.max(1).values
    assert bool((y[torch.arange(B), rows] >= top - 2.0 ** -7 * top.abs()).all())


@pytest.mark.parametrize("B,fmt", [(3, "bf16"), (16, "nvfp4"), (128, "bf16"), (128, "fp8"), (16, "fp8")])
def test_many_blocks_stream_in_order(cuda_device, B, fmt):
    """More CTAs than SMs, so that two stream side by side, and rings of 3 to 8 stages behind 64 chunks: every pass gives
    the same bits (each CTA alone owns its block's sums), and the sums of the inputs."""
    from vdcores_b200 import isa
    from vdcores_b200.batch import unpack_kc
    dev, Bp, K, M = cuda_device, bpad(B), 4096, 28672
    x = seeded((B, K), 11)
    w, sc, wf = weights(M, K, fmt, dev, seed=12)
    xd, outs = packed_rows(x, dev), []
    for _ in range(12):
        out = torch.zeros(Bp * M // 2, dtype=BF16, device=dev)
        run(dev, gemm(dev, fmt, B, M, K, 1, w, sc, xd, mode=isa.STAGE_SILU, out=out.data_ptr()))
        outs.append(out)
    assert all(torch.equal(o, outs[0]) for o in outs)
    yb = (x.to(dev).double() @ wf.to(dev).double().t()).to(BF16).float()
    ref = torch.nn.functional.silu(yb[:, 0::2]) * yb[:, 1::2]
    assert rel(unpack_kc(outs[0].cpu(), Bp, M // 2)[:B], ref.cpu()) < 2 * REL


def test_quantised_codes_widen_exactly(cuda_device):
    """Every e4m3 code, and every e2m1 code under every block scale, against one-hot rows: the stored value itself, the
    codes that are no numbers included."""
    from vdcores_b200 import isa
    from vdcores_b200.batch import pack_blocks_fp8, pack_blocks_nvfp4, unpack_kc
    dev, K, M, B = cuda_device, 64, 256, 64
    x = torch.eye(B, K).to(BF16)
    codes = torch.zeros(M, K, dtype=torch.uint8)
    codes[torch.arange(M), torch.arange(M) % K] = torch.arange(M, dtype=torch.uint8)
    rows = torch.zeros(M, K // 2 + K // 16, dtype=torch.uint8)
    pairs = torch.tensor([(2 * j) | ((2 * j + 1) << 4) for j in range(8)], dtype=torch.uint8)
    rows[:, :8], rows[:, K // 2] = pairs, torch.arange(M, dtype=torch.uint8)
    ones = torch.ones(M, device=dev)
    grid = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
    e4m3 = torch.arange(256, dtype=torch.uint8).view(torch.float8_e4m3fn).float()
    want8 = torch.zeros(B, M)
    want8[torch.arange(M) % K, torch.arange(M)] = e4m3
    want4 = torch.zeros(B, M)
    want4[:16] = torch.cat((grid, -grid))[:, None] * e4m3[None]
    for fmt, w, want in (("fp8", pack_blocks_fp8(codes.to(dev), isa.STAGE_BLOCK), want8),
                         ("nvfp4", pack_blocks_nvfp4(rows.to(dev), K, isa.STAGE_BLOCK), want4)):
        xd, hd, st = packed_rows(x, dev), torch.zeros(64 * M, dtype=BF16, device=dev), torch.zeros(128, device=dev)
        run(dev, gemm(dev, fmt, B, M, K, 1, w, ones, xd, mode=isa.STAGE_RESID, hid=hd.data_ptr(), stats_out=st.data_ptr()))
        got = unpack_kc(hd.cpu(), 64, M).float()
        nan = torch.isnan(e4m3)[None].expand(B, -1)     # a row with a code that is no number is one in every sum
        assert torch.equal(got[~nan], want[~nan]) and bool(torch.isnan(got[nan]).all())


@pytest.mark.parametrize("kind", ["decode", "prefill"])
@pytest.mark.parametrize("G,n_kv,B,splits,lens", [(4, 2, 3, 8, [1, 64, 65]), (8, 1, 2, 2, [700, 129]), (4, 1, 17, 1, None),
                                                  (8, 2, 9, 4, None), (4, 2, 128, 2, None)])
def test_attention(cuda_device, kind, G, n_kv, B, splits, lens):
    """decode: every row over its own pages (lengths of one row, whole pages, one row more; more CTAs than pages).
    prefill: rows are consecutive positions of one sequence, the last ones repeated, tiles that end past the rows."""
    from vdcores_b200 import isa, runtime
    from vdcores_b200.batch import unpack_kc
    from vdcores_b200.decode import kv_page_swizzle
    dev, Bp, D = cuda_device, bpad(B), 128
    if kind == "prefill":
        pos = torch.arange(90, 90 + B).clamp_(max=90 + max(0, B - 3))
        n_tab, tables = 5, torch.randperm(5, generator=torch.Generator().manual_seed(1))[None].expand(B, -1)
    else:
        pos = torch.tensor([l - 1 for l in lens]) if lens else torch.randint(0, 300, (B,), generator=torch.Generator().manual_seed(3))
        n_tab = int(pos.max()) // 64 + 2
        tables = torch.randperm(B * n_tab, generator=torch.Generator().manual_seed(2)).view(B, n_tab)
    k, v = seeded((int(tables.max()) + 1, n_kv, 64, D), 8), seeded((int(tables.max()) + 1, n_kv, 64, D), 9)
    for b in range(B):          # rows past a sequence's last position: whatever an earlier request left
        last = int(pos.max()) if kind == "prefill" else int(pos[b])
        for t in (k, v):
            t[tables[b, last // 64], :, last % 64 + 1:] = float("nan")
    q = seeded((B, n_kv * G, D), 10, 2.0)
    state = torch.zeros(B, isa.ST_PAGETABLE + n_tab, dtype=torch.int32)
    state[:, isa.ST_POS] = pos
    state[:, isa.ST_PAGETABLE:] = tables
    kd, vd, qd, sd = kv_page_swizzle(k).to(dev), kv_page_swizzle(v).to(dev), q.to(dev), state.to(dev)
    out = torch.zeros(Bp * n_kv * G * D, dtype=BF16, device=dev)
    run(dev, runtime.Stage(kind=isa.STAGE_ATTN if kind == "decode" else isa.STAGE_ATTN_PREFILL, B=B, Bpad=Bp, splits=splits,
                           group=G, n_kv=n_kv, n_pages=n_tab, state_stride=state.shape[1], state=sd.data_ptr(),
                           q=qd.data_ptr(), out=out.data_ptr(), kpool=kd.data_ptr(), vpool=vd.data_ptr()))
    got = unpack_kc(out.cpu(), Bp, n_kv * G * D).view(Bp, n_kv, G, D)
    for b in range(B):
        T = int(pos[b]) + 1
        kk = k[tables[b]].transpose(0, 1).reshape(n_kv, -1, D)[:, :T].float()
        vv = v[tables[b]].transpose(0, 1).reshape(n_kv, -1, D)[:, :T].float()
        p = torch.softmax(q[b].view(n_kv, G, D).float() @ kk.transpose(1, 2) / math.sqrt(D), -1)
        assert rel(got[b], p @ vv) < REL, f"row {b}"
    assert float(got[B:].abs().max() if B < Bp else 0) == 0


def _walk(dev, kind, B, n_kv, G, splits, pos, seed):
    """One attention stage over random pages: (run() -> fresh output rows [B, heads, 128], the same in fp32)."""
    from vdcores_b200 import isa, runtime
    from vdcores_b200.batch import unpack_kc
    from vdcores_b200.decode import kv_page_swizzle
    g = torch.Generator(device=dev).manual_seed(seed)
    rnd = lambda *s: torch.empty(*s, device=dev).normal_(generator=g).to(BF16)
    n_tab, seqs, D = int(max(pos)) // 64 + 1, (B if kind == "decode" else 1), 128
    tables = torch.randperm(seqs * n_tab, generator=torch.Generator().manual_seed(seed)).view(seqs, n_tab).expand(B, -1)
    k, v, q = rnd(seqs * n_tab, n_kv, 64, D), rnd(seqs * n_tab, n_kv, 64, D), rnd(B, n_kv * G, D)
    state = torch.zeros(B, isa.ST_PAGETABLE + n_tab, dtype=torch.int32)
    state[:, isa.ST_POS] = torch.tensor(pos, dtype=torch.int32)
    state[:, isa.ST_PAGETABLE:] = tables
    kd, vd, sd = kv_page_swizzle(k), kv_page_swizzle(v), state.to(dev)

    def once():
        out = torch.full((bpad(B) * n_kv * G * D,), float("nan"), dtype=BF16, device=dev)
        run(dev, runtime.Stage(kind=isa.STAGE_ATTN if kind == "decode" else isa.STAGE_ATTN_PREFILL, B=B, Bpad=bpad(B),
                               splits=splits, group=G, n_kv=n_kv, n_pages=n_tab, state_stride=state.shape[1],
                               state=sd.data_ptr(), q=q.data_ptr(), out=out.data_ptr(), kpool=kd.data_ptr(),
                               vpool=vd.data_ptr()))
        return unpack_kc(out, bpad(B), n_kv * G * D)[:B].view(B, n_kv * G, D)

    ref = torch.empty(B, n_kv, G, D, device=dev)
    for b in range(B):
        T, rows = int(pos[b]) + 1, tables[b].to(dev)
        kk, vv = (t[rows].transpose(0, 1).reshape(n_kv, -1, D)[:, :T].float() for t in (k, v))
        ref[b] = torch.softmax(q[b].view(n_kv, G, D).float() @ kk.transpose(1, 2) / math.sqrt(D), -1) @ vv
    return once, ref.view(B, n_kv * G, D)


@pytest.mark.parametrize("kind,B,n_kv,G,splits,lo,hi", [
    ("decode", 128, 8, 4, 1, 351, 700), ("decode", 64, 8, 4, 1, 1051, 2100), ("decode", 24, 4, 8, 1, 2050, 2300),
    ("decode", 32, 8, 4, 2, 751, 1500), ("prefill", 128, 8, 4, 1, 1037, 1164), ("prefill", 40, 2, 8, 2, 2100, 2139)])
def test_long_walks_give_the_same_bits_every_time(cuda_device, kind, B, n_kv, G, splits, lo, hi):
    """Up to 36 pages per CTA (the ring many times over, a second read of the page ids), more units than fit the GPU at
    once, with one CTA per unit and with several: the sums are ordered, so that every head of every row has the same bits
    in every pass, and each is the fp32 softmax's within the bound of the attention."""
    dev = cuda_device
    pos = list(range(lo, lo + B)) if kind == "prefill" else [hi - (b * 37) % (hi - lo + 1) for b in range(B)]
    once, ref = _walk(dev, kind, B, n_kv, G, splits, pos, seed=B + G)
    first = once()
    err = (first.float() - ref).norm(dim=2) / ref.norm(dim=2)
    assert float(err.max()) < 2 * REL, f"(row, head) {divmod(int(err.argmax()), n_kv * G)}"
    for i in range(150):
        differs = (once() != first).any(2).nonzero()
        assert not len(differs), f"pass {i}: (row, head) {differs[:8].tolist()}"


@pytest.mark.parametrize("batch,ctx", [(128, 700), (64, 2100)])
def test_every_step_of_a_large_batch_has_the_same_bits(cuda_device, batch, ctx):
    """One layer, one step from the same state again and again: queries, appended cache rows and attention outputs depend on
    ordered sums only and repeat bit for bit; the hidden rows behind them repeat within the rounding of their statistics'
    order."""
    from vdcores_b200.batch import BatchDecodeEngine
    from vdcores_b200.decode import DecodeConfig
    cfg = DecodeConfig(hidden=1024, n_heads=32, n_kv_heads=8, ffn=2048, vocab=2048, n_layers=1)
    eng = BatchDecodeEngine(cfg, batch, max_seq=ctx + 64, device=cuda_device, page_perm_seed=3)
    eng.init_random_weights(1)
    assert eng.n_splits == 1
    g = torch.Generator(device=cuda_device).manual_seed(2)
    for t in (eng.kpool, eng.vpool):
        t.normal_(generator=g)
    for b in range(batch):
        eng.set_state(ctx - (b * 37) % (ctx // 2), (b * 29) % cfg.vocab, b=b)
    torch.cuda.synchronize()
    state, pos, first = eng.state.clone(), eng.pos, None
    k_rows, v_rows = (t.view(-1, 128) for t in (eng.kpool, eng.vpool))
    from vdcores_b200 import isa
    new = (state[:, isa.ST_NEWROW, None] + 64 * torch.arange(8, device=cuda_device)).long()     # [batch, kv heads]
    for i in range(200):
        for t in (k_rows, v_rows):
            t[new] = 0
        eng.q.zero_()
        eng.attn_out.zero_()
        eng.state.copy_(state)
        eng.pos, eng.steps_done = pos, 0
        eng.generate(1)
        got = [eng.q.clone(), k_rows[new], v_rows[new], eng.attn_out.clone(), eng.read_hidden(eng.hidden).float()]
        if first is None:
            first = got
            continue
        for name, a, b in zip(("q", "k", "v", "attention"), got, first):
            assert torch.equal(a, b), f"pass {i}: {name} differs at {(a != b).nonzero()[:8].tolist()}"
        rows = (got[4] - first[4]).norm(dim=1) / first[4].norm(dim=1)
        assert float(rows.max()) < 1e-2, f"pass {i}: hidden row {int(rows.argmax())}"


@pytest.mark.parametrize("splits", [1, 8])
def test_qkv_stage_writes_a_repeated_position_once(cuda_device, splits):
    """Query rows and cache rows against plain matmuls (no rotation at position 0's angles); rows with the cache row of the
    row in front of them leave it to that one, whatever their own values are."""
    from vdcores_b200 import isa, runtime
    from vdcores_b200.decode import kv_page_swizzle
    dev, B, G, n_kv, K, D = cuda_device, 24, 4, 2, 1024, 128
    M = n_kv * (G + 2) * D
    x = seeded((B, K), 31)
    w, _, wf = weights(M, K, "bf16", dev, seed=32)
    xd = packed_rows(x, dev)
    rope = torch.cat((torch.ones(128, 64), torch.zeros(128, 64)), 1).to(dev)
    pos = torch.arange(60, 60 + B).clamp_(max=60 + 9)
    table = torch.tensor([2, 0])
    state = torch.zeros(B, isa.ST_PAGETABLE + 2, dtype=torch.int32)
    state[:, isa.ST_POS] = pos
    state[:, isa.ST_NEWROW] = table[pos // 64] * 64 * n_kv + pos % 64
    sd, q = state.to(dev), torch.zeros(B, n_kv * G, D, dtype=BF16, device=dev)
    for _ in range(20):
        pools = [torch.zeros(3, n_kv, 64, D, dtype=BF16, device=dev) for _ in range(2)]
        run(dev, gemm(dev, "bf16", B, M, K, splits, w, None, xd, mode=isa.STAGE_QKV, out=q.data_ptr(), rope=rope.data_ptr(),
                      kpool=pools[0].data_ptr(), vpool=pools[1].data_ptr(), group=G, n_kv=n_kv, state=sd.data_ptr(),
                      state_stride=state.shape[1]))
        y = (x.float() @ wf.t()).view(B, n_kv, G + 2, D)
        assert rel(q.cpu().view(B, n_kv, G, D), y[:, :, :G]) < REL
        for i, pool in enumerate(pools):
            rows = kv_page_swizzle(pool.cpu()).float()
            want = torch.zeros_like(rows)
            for b in range(10):
                want[table[pos[b] // 64], :, pos[b] % 64] = y[b, :, G + i]
            assert rel(rows, want) < REL and bool((rows[want.abs().sum(-1) == 0] == 0).all())
            last = rows[table[pos[9] // 64], :, pos[9] % 64]
            assert rel(last, y[9, :, G + i]) < REL


@pytest.mark.parametrize("num_sms", [1, 7, 61, 140])
def test_a_step_and_a_prompt_on_fewer_sms(cuda_device, num_sms):
    """num_sms below the device's count: slices of at most that many CTAs, and the results of the whole device."""
    from vdcores_b200 import runtime
    from vdcores_b200.batch import BatchDecodeEngine
    from vdcores_b200.decode import DecodeConfig, DecodeEngine
    from vdcores_b200.prefill import PrefillEngine
    cfg = DecodeConfig(hidden=512, n_heads=8, n_kv_heads=2, ffn=1024, vocab=512, n_layers=2)
    prompt = torch.randint(0, cfg.vocab, (100,), generator=torch.Generator().manual_seed(4))
    got = {}
    for n in (None, num_sms):
        eng = BatchDecodeEngine(cfg, 20, max_seq=192, device=cuda_device, num_sms=n)
        eng.init_random_weights(1)
        g = torch.Generator(device=cuda_device).manual_seed(2)
        for t in (eng.kpool, eng.vpool):
            t.normal_(generator=g)
        for b in range(20):
            eng.set_state(150 - 7 * b, 10 + b, b=b)
        torch.cuda.synchronize()
        eng.generate(1)
        dec = DecodeEngine(cfg, 192, device=cuda_device, num_sms=n)
        dec.init_random_weights(1)
        pre = PrefillEngine(dec, chunk=64).adopt_weights()
        pre.prefill(prompt)
        got[n] = eng.read_hidden(eng.hidden), pre.read_hidden(pre.hidden), dec.kpool[:, :2]
        assert n is None or all(runtime.count_stage_launches(e.stages, e.max_ctas)[1] <= n for e in (eng, pre))
    for a, b in zip(got[None], got[num_sms]):
        assert rel(a, b) < 2e-2          # other K-splits: other orders of the sums, in bf16 through two layers


@pytest.mark.parametrize("fmt", ["bf16", "fp8", "nvfp4"])
def test_a_budget_of_one_nanosecond_ends_every_wait(cuda_device, fmt):
    """Waits that may give up at their first look at the clock: the launch ends, either with the right result (nothing had
    to wait that long) or with the timeout in the status block; the context stays usable and the next launch is right."""
    from vdcores_b200 import isa, runtime
    dev, B, K, M, G, n_kv, n_tab = cuda_device, 40, 4096, 4096, 4, 2, 16
    x = seeded((B, K), 1)
    w, sc, _ = weights(M, K, fmt, dev)
    xd = packed_rows(x, dev)
    pools = [torch.randn(B * n_tab, n_kv, 64, 128, device=dev).to(BF16) for _ in range(2)]
    state = torch.zeros(B, isa.ST_PAGETABLE + n_tab, dtype=torch.int32)
    state[:, isa.ST_POS] = 64 * n_tab - 1
    state[:, isa.ST_PAGETABLE:] = torch.arange(B * n_tab).view(B, n_tab)
    sd, q = state.to(dev), seeded((B, n_kv * G, 128), 10, 2.0).to(dev)
    stream = torch.cuda.current_stream(dev).cuda_stream

    def both(timeout_ns):
        act = torch.zeros(bpad(B) * M // 2, dtype=BF16, device=dev)
        out = torch.zeros(bpad(B) * n_kv * G * 128, dtype=BF16, device=dev)
        stages = [gemm(dev, fmt, B, M, K, 2, w, sc, xd, mode=isa.STAGE_SILU, out=act.data_ptr()),
                  runtime.Stage(kind=isa.STAGE_ATTN, B=B, Bpad=bpad(B), splits=2, group=G, n_kv=n_kv, n_pages=n_tab,
                                state_stride=state.shape[1], state=sd.data_ptr(), q=q.data_ptr(), out=out.data_ptr(),
                                kpool=pools[0].data_ptr(), vpool=pools[1].data_ptr())]
        for s in stages:
            runtime.launch_stages((runtime.Stage * 1)(s), stream, timeout_ns)
        try:
            runtime.read_status(stream)
            ok = True
        except runtime.VdcError as e:
            assert e.code == 1 and e.status["opcode"] in (isa.STAGE_GEMM, isa.STAGE_ATTN)
            ok = False
        return ok, act, out

    ok, act, out = both(500_000_000)
    assert ok
    for _ in range(20):
        ok, a, o = both(1)
        assert not ok or (torch.equal(a, act) and torch.equal(o, out))
    ok, a, o = both(500_000_000)
    assert ok and torch.equal(a, act) and torch.equal(o, out)


def test_a_row_without_a_token_is_reported_and_nothing_runs_on(cuda_device):
    """A key of 0 (no number among the logits) at the advance, ids outside the table at the embedding: an error in the status
    block, a valid id in the state; stages behind an unread error leave hidden rows, keys and states as they were."""
    from vdcores_b200 import isa, runtime
    from vdcores_b200.batch import unpack_kc
    dev, B, H, V = cuda_device, 3, 256, 32
    stream = torch.cuda.current_stream(dev).cuda_stream
    state = torch.zeros(B, isa.ST_PAGETABLE + 2, dtype=torch.int32, device=dev)
    state[:, isa.ST_POS], state[:, isa.ST_MAXPAGES], state[:, isa.ST_NKVH] = 5, 2, 1
    log = torch.full((B, 4), -9, dtype=torch.int32, device=dev)
    keys = torch.tensor([(1 << 40) | (0xFFFFFFFF - 7), 0, (1 << 40) | (0xFFFFFFFF - 9)], device=dev)
    advance = runtime.Stage(kind=isa.STAGE_ADVANCE, B=B, Bpad=16, keys=keys.data_ptr(), log=log.data_ptr(), log_stride=4,
                            state=state.data_ptr(), state_stride=state.shape[1])
    table = seeded((V, H), 1).to(dev)
    hid, stats = torch.zeros(16 * H, dtype=BF16, device=dev), torch.zeros(128, device=dev)
    embed = runtime.Stage(kind=isa.STAGE_EMBED, B=B, Bpad=16, M=V, K=H, w=table.data_ptr(), hid=hid.data_ptr(),
                          stats_out=stats.data_ptr(), n_stats=1, state=state.data_ptr(), state_stride=state.shape[1])
    w, sc, _ = weights(H, H, "bf16", dev)
    xd = packed_rows(seeded((B, H), 2), dev)
    add = gemm(dev, "bf16", B, H, H, 2, w, sc, xd, mode=isa.STAGE_RESID, hid=hid.data_ptr(), stats_out=stats.data_ptr())

    def launch(*stages):
        runtime.launch_stages((runtime.Stage * len(stages))(*stages), stream, 500_000_000)

    launch(advance)
    kept = state.clone(), log.clone(), keys.clone(), hid.clone(), stats.clone()
    launch(embed, add, advance)
    with pytest.raises(runtime.VdcError) as e:
        runtime.read_status(stream)
    assert e.value.code == 5 and e.value.status["pc"] == 1 and e.value.status["opcode"] == isa.STAGE_ADVANCE
    assert all(torch.equal(a, b) for a, b in zip(kept, (state, log, keys, hid, stats)))
    assert state[:, isa.ST_TOKEN].tolist() == [7, 0, 9] and state[:, isa.ST_ERR].tolist() == [0, 1, 0]
    assert log[:, 0].tolist() == [7, 0, 9] and state[:, isa.ST_POS].tolist() == [6, 6, 6] and not keys.any()
    for bad in (-1, V, 2 ** 31 - 1, -2 ** 31):
        state[1, isa.ST_TOKEN] = bad
        launch(embed)
        with pytest.raises(runtime.VdcError) as e:
            runtime.read_status(stream)
        assert e.value.code == 5 and e.value.status["aux"] == bad
        assert torch.equal(unpack_kc(hid, 16, H)[1], table[0])
    state[1, isa.ST_TOKEN] = V - 1
    run(dev, embed)
    assert torch.equal(unpack_kc(hid, 16, H)[:B], table[[7, V - 1, 9]])


def test_logits_without_a_number_end_a_generation_with_an_error(cuda_device):
    """Weights with a NaN: the steps already enqueued behind the first one stop at it, and the engine can be used again."""
    from vdcores_b200 import isa, runtime
    from vdcores_b200.batch import BatchDecodeEngine
    from vdcores_b200.decode import DecodeConfig
    cfg = DecodeConfig(hidden=512, n_heads=8, n_kv_heads=2, ffn=1024, vocab=256, n_layers=1)
    eng = BatchDecodeEngine(cfg, 3, max_seq=128, device=cuda_device)
    eng.init_random_weights(1)

    def start():
        for b in range(3):
            eng.set_state(4, 10 + b, b=b)
        torch.cuda.synchronize()
    start()
    good = eng.generate(4)
    eng.norm_w.fill_(float("nan"))
    start()
    with pytest.raises(runtime.VdcError) as e:
        eng.generate(4)
    assert e.value.code == 5
    assert eng.state[:, isa.ST_POS].tolist() == [5, 5, 5] and eng.state[:, isa.ST_TOKEN].tolist() == [0, 0, 0]
    eng.norm_w.fill_(1.0)
    start()
    assert eng.generate(4) == good


@pytest.mark.parametrize("fmt", ["bf16", "fp8", "nvfp4"])
@pytest.mark.parametrize("M,K,splits,B", [(48, 1024, 1, 128), (1040, 2048, 2, 128), (4096, 4096, 8, 77), (256, 1024, 4, 16), (400, 1024, 1, 33)])
def test_projection_leaves_fp32_sums(cuda_device, fmt, M, K, splits, B):
    """A block of 48, 16 or 128 weight rows, K whole and shared, rows that do not fill the accumulator: fp32 sums of bf16 products,
    so only the order of the additions differs from the matmul's (1e-5 of the result's norm)."""
    from vdcores_b200 import isa
    dev = cuda_device
    w, sc, wd = weights(M, K, fmt, dev)
    x = seeded((B, K), 9).to(BF16)
    xd = packed_rows(x, dev)
    Bp = next(p for p in (16, 32, 64, 128) if B <= p)
    out = torch.full((M // 4, Bp, 4), -7.0, device=dev)
    run(dev, gemm(dev, fmt, B, M, K, splits, w, sc, xd, mode=isa.STAGE_SUMS, out=out.data_ptr()))
    got = out.permute(1, 0, 2).reshape(Bp, M)
    want = x.double().to(dev) @ wd.double().to(dev).t()
    assert rel(got[:B].double(), want) < 1e-5
    assert bool((got[B:] == -7.0).all())
