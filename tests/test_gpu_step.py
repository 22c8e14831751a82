"""A token at batch 1 as one persistent kernel (csrc/step_kernel.cu) against the megakernel's program over the same weights and
caches, at the places where shares, chunks, K-splits and page walks can go wrong."""
import pytest
import torch

from tests.test_gpu_stages import rel

pytestmark = pytest.mark.gpu


def _engine(dev, max_seq, seed=3, **kw):
    from vdcores_b200.decode import DecodeConfig, DecodeEngine
    num_sms, wkind = kw.pop("num_sms", None), kw.pop("wkind", "bf16")
    cfg = DecodeConfig(eps=1e-5, theta=5e5, **kw)
    eng = DecodeEngine(cfg, max_seq, device=dev, wkind=wkind, num_sms=num_sms, taps=True, page_perm_seed=7, timeout_ns=500_000_000)
    eng.init_random_weights(seed)
    eng.step_kernel = eng._plan_step()
    g = torch.Generator(device=dev).manual_seed(seed)
    for t in (eng.kpool, eng.vpool):
        t.normal_(generator=g)
    return eng


def _steps(eng, pos, n, step_kernel, caches):
    """n steps from position pos, every step's layer outputs, logits and token; the ids are forced."""
    saved, eng.step_kernel = eng.step_kernel, eng.step_kernel if step_kernel else None
    eng.kpool.copy_(caches[0])
    eng.vpool.copy_(caches[1])
    eng.set_state(pos, 5)
    out = []
    for i in range(n):
        tok = eng.generate(1)[0]
        out.append((eng.taps.clone(), eng.logits.clone(), eng.hidden.clone(), tok))
        eng.state[2:3].fill_(6 + i)
    eng.step_kernel = saved
    return out, eng.state.clone(), eng.kpool.clone(), eng.vpool.clone()


CASES = [
    # fewer rows than SMs, one unit per head; the first position; a page that holds the new row only
    (dict(hidden=256, n_heads=4, n_kv_heads=1, ffn=256, vocab=34, n_layers=2), (0, 63, 64), None),
    (dict(hidden=512, n_heads=8, n_kv_heads=2, ffn=1024, vocab=2048, n_layers=3), (199, 255, 256, 257), None),
    # splits of several pages, the last ones empty; a head group of 8; q/k norms
    (dict(hidden=1024, n_heads=16, n_kv_heads=2, ffn=1280, vocab=530, n_layers=2, qk_norm=True), (1200, 4095), None),
    # K ranges that do not divide among the warps (7, 5 and 3 steps), rows over 28 KB, an odd number of SMs
    (dict(hidden=1280, n_heads=8, n_kv_heads=2, ffn=14336, vocab=1000, n_layers=1), (300,), 61),
    (dict(hidden=1792, n_heads=16, n_kv_heads=4, ffn=768, vocab=4096, n_layers=2), (70,), 17),
    (dict(hidden=1024, n_heads=8, n_kv_heads=1, ffn=3072, vocab=256, n_layers=2, wkind="fp8"), (130, 2500), None),
    (dict(hidden=2048, n_heads=32, n_kv_heads=8, ffn=1536, vocab=1024, n_layers=2, wkind="fp8"), (77,), 132),
    (dict(hidden=1024, n_heads=8, n_kv_heads=2, ffn=3072, vocab=256, n_layers=2, wkind="nvfp4"), (130,), None),
    (dict(hidden=4096, n_heads=32, n_kv_heads=8, ffn=12288, vocab=512, n_layers=1, wkind="nvfp4", qk_norm=True), (333,), None),
    (dict(hidden=512, n_heads=8, n_kv_heads=2, ffn=256, vocab=512, n_layers=2, n_experts=16, top_k=4), (100,), None),
    (dict(hidden=2048, n_heads=32, n_kv_heads=4, ffn=768, vocab=512, n_layers=1, n_experts=128, top_k=8, qk_norm=True), (64,), None)]


@pytest.mark.parametrize("kw,positions,num_sms", CASES)
def test_step_kernel_against_the_megakernels_program(cuda_device, kw, positions, num_sms):
    eng = _engine(cuda_device, (max(positions) + 70) // 64 * 64, num_sms=num_sms, **dict(kw))
    assert eng.step_kernel is not None
    caches = eng.kpool.clone(), eng.vpool.clone()
    for pos in positions:
        n = 1 if pos + 3 > eng.max_seq else 3
        a, sa, ka, va = _steps(eng, pos, n, True, caches)
        b, sb, kb, vb = _steps(eng, pos, n, False, caches)
        assert torch.equal(sa, sb)
        for (ta, la, ha, na), (tb, lb, hb, nb) in zip(a, b):
            assert bool(torch.isfinite(ta.float()).all()) and torch.equal(ta[-1], ha)
            # each is within the oracle tests' 1e-2 of the exact result, so the two are within sqrt(2) of that of each other;
            # random experts' weights hang on logits that the roundings move
            bound = 2e-2 if kw.get("n_experts") else 1.5e-2
            assert rel(ta, tb) < bound, pos
            # the logits of this hidden state (the program's own cover whole chunks of rows only): one bf16 rounding, 2^-9
            x = ha.float() * torch.rsqrt(ha.float().pow(2).mean() + eng.cfg.eps)
            assert rel(la, (x.to(torch.bfloat16) * eng.norm_w).float() @ eng.lm_head.float().t()) < 4e-3, pos
            top = torch.topk(la.float(), 2).values
            assert na == int(la.float().argmax())
            if float(top[0] - top[1]) > 5e-2 * float(top[0].abs()):
                assert na == nb
        for x, y, c in ((ka, kb, caches[0]), (va, vb, caches[1])):
            changed = (x != c).flatten(0, 3).any(-1)
            assert int(changed.sum()) <= n * eng.cfg.n_kv_heads * eng.cfg.n_layers        # one row per step, head and layer
            assert rel(x[x != c], y[x != c]) < 2e-2


def test_steps_repeat_bit_for_bit_and_under_a_graph(cuda_device):
    """Nothing is added up with atomics: the same step gives the same bits, fifty times over, also replayed from a graph."""
    eng = _engine(cuda_device, 1024, hidden=1024, n_heads=32, n_kv_heads=8, ffn=2048, vocab=2048, n_layers=3)
    eng.set_state(777, 9)
    torch.cuda.synchronize()
    state = eng.state.clone()
    want = None
    graph = torch.cuda.CUDAGraph()
    for i in range(50):
        eng.state.copy_(state)
        eng.pos, eng.steps_done = 777, 0
        if i == 25:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            own, eng.stream = eng.stream, side
            with torch.cuda.graph(graph, stream=side):
                eng.step_async()
            eng.stream = own
        if i < 25:
            eng.step_async()
        else:
            graph.replay()
        got = eng.logits.clone(), eng.taps.clone()
        want = want or got
        assert all(torch.equal(a, b) for a, b in zip(got, want)), i
    from vdcores_b200 import runtime
    runtime.read_status(eng.stream.cuda_stream)


def test_a_token_outside_the_vocabulary_is_reported(cuda_device):
    """The step ends with an error and leaves state and log as they were; what is enqueued behind it does not run; after the
    error is read the engine goes on."""
    from vdcores_b200 import runtime
    eng = _engine(cuda_device, 128, hidden=512, n_heads=8, n_kv_heads=2, ffn=512, vocab=64, n_layers=1)
    want = _steps(eng, 20, 1, True, (eng.kpool.clone(), eng.vpool.clone()))[0][0]
    eng.set_state(20, 64)
    eng.token_log.fill_(-7)
    before = eng.state.clone()
    eng.step_async()
    eng.step_async()
    with pytest.raises(runtime.VdcError):
        runtime.read_status(eng.stream.cuda_stream)
    assert torch.equal(eng.state, before) and bool((eng.token_log == -7).all())
    eng.set_state(20, 5)
    assert eng.generate(1)[0] == want[3] and torch.equal(eng.logits, want[1])
