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
    # more splits of a head than a warp has lanes: 32 of four pages, 33, 119 of five, the last one smaller
    (dict(hidden=512, n_heads=4, n_kv_heads=1, ffn=512, vocab=64, n_layers=1), (8191, 8192, 37900), None),
    (dict(hidden=512, n_heads=16, n_kv_heads=2, ffn=512, vocab=64, n_layers=1), (9000, 23000), 132),
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
    assert eng.step_kernel.n_splits == min(eng.num_sms // eng.cfg.n_kv_heads, eng.max_pages)
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
            rows = [(t != c).any(-1) for t in (x, y)]              # by both, one row per step, head and layer
            assert torch.equal(*rows) and int(rows[0].sum()) == n * eng.cfg.n_kv_heads * eng.cfg.n_layers
            assert rel(x[rows[0]], y[rows[0]]) < 2e-2


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


def test_a_wait_that_runs_out_ends_with_an_error(cuda_device):
    """Two SMs busy with another engine's step for some milliseconds: the SMs that have started wait for those two, to a limit of a
    nanosecond.  The step ends with the timeout in the status block, nothing moved on and nothing left that the next one takes
    for its own: that one, with a proper limit, is right."""
    from vdcores_b200 import isa, runtime
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        busy = _engine(cuda_device, 64, hidden=1024, n_heads=4, n_kv_heads=1, ffn=1024, vocab=131072, n_layers=1, num_sms=2)
    eng = _engine(cuda_device, 1024, hidden=1024, n_heads=16, n_kv_heads=4, ffn=2048, vocab=512, n_layers=3)
    assert busy.step_kernel is not None and busy.stream == side

    def start(token):
        eng.set_state(700, token)
        busy.set_state(0, 1)
        torch.cuda.synchronize()
    start(5)
    want = eng.generate(1), eng.logits.clone()
    ended = 0
    for i in range(8):
        start(6 + i)              # another token: entries it leaves are not those of the next step
        state = eng.state.clone()
        eng.timeout_ns = 1
        busy.step_async()
        eng.step_async()
        torch.cuda.synchronize()
        try:
            runtime.read_status(eng.stream.cuda_stream)
        except runtime.VdcError as e:
            assert e.code == 1 and e.status["opcode"] == isa.STEP_KIND and torch.equal(eng.state, state)
            ended += 1
        eng.timeout_ns = 500_000_000
        start(5)
        assert eng.generate(1) == want[0] and torch.equal(eng.logits, want[1])
    assert ended > 0


@pytest.mark.parametrize("pos", [100, 1500])         # one SM walks a head's pages; several do, and merge
def test_queries_without_a_number_attend_to_nothing(cuda_device, pos):
    eng = _engine(cuda_device, 1600, hidden=512, n_heads=8, n_kv_heads=2, ffn=512, vocab=640, n_layers=1, qk_norm=True)
    eng.qknorm[:, :128] = float("nan")
    caches = eng.kpool.clone(), eng.vpool.clone()
    (a, la, _, _), = _steps(eng, pos, 1, True, caches)[0]
    (b, _, _, _), = _steps(eng, pos, 1, False, caches)[0]
    assert bool(torch.isfinite(la.float()).all()) and rel(a, b) < 1.5e-2


def test_logits_without_a_number_are_reported(cuda_device):
    """The step itself ends with the error and leaves state and log; one logit that is a number is enough for a token."""
    from vdcores_b200 import runtime
    eng = _engine(cuda_device, 128, hidden=512, n_heads=8, n_kv_heads=2, ffn=512, vocab=640, n_layers=1)
    head = eng.lm_head.clone()
    eng.set_state(20, 5)
    want = eng.generate(1)[0]
    eng.lm_head.fill_(float("nan"))
    eng.set_state(20, 5)
    eng.token_log.fill_(-7)
    before = eng.state.clone()
    with pytest.raises(runtime.VdcError, match="no number among"):
        eng.generate(1)
    assert torch.equal(eng.state, before) and bool((eng.token_log == -7).all())
    eng.lm_head[601] = head[601]
    eng.set_state(20, 5)
    assert eng.generate(1) == [601]
    eng.lm_head.copy_(head)
    eng.set_state(20, 5)
    assert eng.generate(1)[0] == want


@pytest.mark.parametrize("wkind", ["bf16", "fp8"])
def test_sums_lose_no_more_bits_than_fp32_fmas(cuda_device, wkind):
    """Sums of 8192 products, two of them large and cancelling, so that every addition's rounding shows in the result: values of
    the cache rows (a layer's projection) and logits that are not the bf16 rounding of the sum in 64 bits.  The program adds with
    FMAs; the step kernel may miss no more of them than it, up to five standard deviations of the two counts."""
    from vdcores_b200.decode import DecodeConfig, DecodeEngine
    H, L = 8192, 4
    cfg = DecodeConfig(hidden=H, n_heads=32, n_kv_heads=8, ffn=512, vocab=16384, n_layers=L, eps=0.0, theta=1e4)
    eng = DecodeEngine(cfg, 64, device=cuda_device, wkind=wkind, timeout_ns=500_000_000)
    eng.init_random_weights(1)
    g = torch.Generator(device=cuda_device).manual_seed(2)
    # a hidden state of ones that no layer adds to: the norms' weights are the inputs
    eng.embed.fill_(1.0)
    for n in ("wo", "wd"):
        (eng.scales[n] if wkind == "fp8" else getattr(eng, n)).zero_()
    x = torch.randn(L + 1, H, generator=g, device=cuda_device).to(torch.bfloat16)
    x[:, 0] = x[:, -1] = 2.0 ** 14
    eng.ln1.copy_(x[:L])
    eng.norm_w.copy_(x[L])

    def matrix(rows):
        w = 0.02 * torch.randn(rows, H, generator=g, device=cuda_device)
        w[:, 0], w[:, -1] = 0.02, -0.02
        return w.to(torch.bfloat16)
    eng.lm_head.copy_(matrix(cfg.vocab))
    exact_l, exact_v = eng.lm_head.double() @ x[L].double(), []
    for l in range(L):
        rows, sc = eng._encode(matrix(eng.qkv_rows))
        eng.wqkv[l].copy_(rows)
        if sc is not None:
            eng.scales["wqkv"][l].copy_(sc)
            rows = rows.view(torch.float8_e4m3fn).double() * sc.double()[:, None]
        exact_v.append((rows.double() @ x[l].double()).view(cfg.n_kv_heads, cfg.group + 2, 128)[:, -1].reshape(-1))
    missed = []
    for step in (eng.step_kernel, None):
        eng.step_kernel = step
        eng.set_state(0, 3)
        eng.generate(1)
        v = torch.stack([eng.read_kv(l, 1)[1][0].reshape(-1) for l in range(L)])
        missed.append([int((got != want.float().to(torch.bfloat16)).sum())
                       for got, want in ((v, torch.stack(exact_v)), (eng.logits, exact_l))])
    for a, b in zip(*missed):
        assert a <= b + 5 * (a + b) ** 0.5, missed


# rows of which four make more than a copy: K of 18, 32, 33 and 56 steps, groups that end with two rows; an SM's gate/up rows too many
# for the sums of slices (544 and 540 of 4608 inputs), and on 16 of 28 SMs only (532, and 528 in slices); the vocabulary projection
# of quantised models
SLICED = [
    (dict(hidden=8192, n_heads=64, n_kv_heads=8, ffn=8448, vocab=1002, n_layers=1), (70,), None),
    (dict(hidden=4608, n_heads=32, n_kv_heads=8, ffn=4608, vocab=700, n_layers=2), (64,), 17),
    (dict(hidden=4608, n_heads=32, n_kv_heads=8, ffn=7424, vocab=700, n_layers=1), (64,), 28),
    (dict(hidden=4096, n_heads=32, n_kv_heads=8, ffn=14336, vocab=512, n_layers=1), (130,), 132),
    (dict(hidden=8192, n_heads=64, n_kv_heads=8, ffn=14336, vocab=1000, n_layers=1, wkind="fp8"), (70,), None),
    (dict(hidden=8192, n_heads=64, n_kv_heads=8, ffn=1024, vocab=4098, n_layers=1, wkind="nvfp4"), (70,), None)]


@pytest.mark.parametrize("kw,positions,num_sms", SLICED)
def test_rows_that_come_in_slices(cuda_device, kw, positions, num_sms):
    test_step_kernel_against_the_megakernels_program(cuda_device, kw, positions, num_sms)


# sums of rows that nobody else adds to, as many as there is room for: 1088 and 4172 gate/up rows, 302 rows of 13 experts' sums
CROWDED = [
    (dict(hidden=1024, n_heads=4, n_kv_heads=1, ffn=4352, vocab=66, n_layers=1), (70,), 8),
    (dict(hidden=1024, n_heads=4, n_kv_heads=1, ffn=14592, vocab=66, n_layers=1), (70,), 7),
    (dict(hidden=6912, n_heads=4, n_kv_heads=1, ffn=512, vocab=66, n_layers=1, n_experts=16, top_k=13), (70,), 23)]


@pytest.mark.parametrize("kw,positions,num_sms", CROWDED)
def test_many_rows_per_sm(cuda_device, kw, positions, num_sms):
    test_step_kernel_against_the_megakernels_program(cuda_device, kw, positions, num_sms)


def test_widest_quantised_rows(cuda_device, monkeypatch):
    """Inputs of 96 KB: the scales' place leaves the ring a little less than three copies of 32 KB, pages of the cache among them.
    Longer than what the program's tasks take, so against PyTorch: the second layer's cache rows hang on all that stands in front."""
    from vdcores_b200.decode import DecodeEngine
    monkeypatch.setattr(DecodeEngine, "_build_program", lambda self: setattr(self, "program", True))
    eng = _engine(cuda_device, 768, hidden=4096, n_heads=32, n_kv_heads=8, ffn=49152, vocab=512, n_layers=2, wkind="nvfp4")
    assert eng.step_kernel is not None
    tokens = torch.randint(0, 512, (701,), generator=torch.Generator().manual_seed(2))
    eng.prefill(tokens)
    want = [t[-1].clone() for t in eng.read_kv(1, 701)]
    page, row = int(eng.page_table[700 // 64]), 700 % 64
    eng.kpool[1, page, :, row] = eng.vpool[1, page, :, row] = 0.0
    eng.set_state(700, int(tokens[-1]))
    eng.generate(1)
    for got, w in zip(eng.read_kv(1, 701), want):
        assert rel(got[-1], w) < 1.5e-2


def test_of_equal_experts_the_lowest_are_chosen(cuda_device):
    """Router rows that are copies of one another give equal logits; two rows are the others' negative, so either all that are not
    chosen last or the first two."""
    eng = _engine(cuda_device, 128, hidden=512, n_heads=8, n_kv_heads=2, ffn=256, vocab=512, n_layers=1, n_experts=96, top_k=6)
    row = eng.router[0][0].clone()
    for odd in ((), (3, 64), (40, 95)):
        eng.router[0].copy_(row)
        for i in odd:
            eng.router[0][i].neg_()
        eng.set_state(70, 5)
        eng.generate(1)
        ids, weights = eng.route[:6].tolist(), eng.route[16:22].view(torch.float32)
        rest = [i for i in range(96) if i not in odd]
        assert ids in (rest[:6], list(odd) + rest[:6 - len(odd)])
        if ids == rest[:6]:
            assert torch.equal(weights, torch.full_like(weights, 1 / 6).to(torch.bfloat16).float())


@pytest.mark.parametrize("expert", [8, 40, 95])
@pytest.mark.parametrize("value", ["nan", "-nan", "inf"])
def test_a_router_logit_without_a_number_ends_a_step(cuda_device, expert, value):
    """The softmax's sum carries it into every expert's weight, wherever among a lane's logits it stands: the step ends with an error
    and no token.  An infinite logit leaves the softmax without a number too."""
    from vdcores_b200 import runtime
    eng = _engine(cuda_device, 128, hidden=512, n_heads=8, n_kv_heads=2, ffn=256, vocab=512, n_layers=1, n_experts=96, top_k=6)
    eng.set_state(70, 5)
    want, router = eng.generate(1), eng.router.clone()
    eng.router[0][expert].fill_(0.0)
    if value == "inf":      # of an input whose sign is not known: two rows, one of which gets +inf
        eng.router[0][expert, 0] = float("inf")
        eng.router[0][expert - 1].fill_(0.0)
        eng.router[0][expert - 1, 0] = float("-inf")
    else:
        eng.router[0][expert] = float(value)
    eng.set_state(70, 5)
    before = eng.state.clone()
    with pytest.raises(runtime.VdcError, match="no number among"):
        eng.generate(1)
    assert torch.equal(eng.state, before)
    weights = eng.route[16:22].view(torch.float32)
    assert bool(torch.isnan(weights).all())
    eng.router.copy_(router)
    eng.set_state(70, 5)
    assert eng.generate(1) == want


def test_silu_of_gates_whose_exponentials_are_close_to_infinity(cuda_device):
    """exp(88) is 1.65e38, and 1 / (1 + exp(88)) below the smallest normal number: the quotient -88 / (1 + exp(88)) is not."""
    eng = _engine(cuda_device, 64, hidden=512, n_heads=8, n_kv_heads=2, ffn=256, vocab=64, n_layers=1)
    eng.embed.fill_(1.0)
    eng.ln2.fill_(1.0)
    for w in (eng.wo, eng.wgu, eng.wd):
        w.zero_()
    eng.wgu[0][0::2, 0], eng.wgu[0][1::2, 0] = -88.0, 2.0 ** 120
    eng.wd[0][:, 7] = 1.0
    caches = eng.kpool.clone(), eng.vpool.clone()
    (a, _, _, _), = _steps(eng, 20, 1, True, caches)[0]
    (b, _, _, _), = _steps(eng, 20, 1, False, caches)[0]
    want = 1 - 88 / (1 + torch.tensor(88.0).double().exp()) * 2.0 ** 120
    for got in (a, b):      # bf16: the SiLU, its product, the sum; __expf has 2 + 1.16 * 88 ulp at 88
        assert bool(((got.double().cpu() - want).abs() < 3 * 2.0 ** -8).all()), (float(got.flatten()[0]), float(want))
