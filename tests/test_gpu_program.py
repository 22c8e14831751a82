"""What runs where the step kernel and the wide stages do not, against the oracle: the megakernel's program of a batch-1 step
(the decode engine's oracle tests once more, and steps that only it can run) and prompts chunk by chunk."""
import pytest
import torch

from oracle import decode_oracle as O
from tests import test_gpu_decode, test_gpu_prefill
from tests.helpers import dense_weights, engine_config, perturb_norms, small_cfg

pytestmark = pytest.mark.gpu


@pytest.fixture
def program(monkeypatch):
    from vdcores_b200.decode import DecodeEngine
    monkeypatch.setattr(DecodeEngine, "_plan_step", lambda self: None)


@pytest.mark.parametrize("kind,prompt_len,n_steps,num_sms", [("llama", 70, 4, None), ("qwen3", 130, 2, 61), ("moe", 70, 3, None)])
def test_program_matches_oracle(cuda_device, program, kind, prompt_len, n_steps, num_sms):
    test_gpu_decode.test_decode_matches_oracle(cuda_device, kind, prompt_len, n_steps, num_sms)


@pytest.mark.parametrize("wkind,tol,base", [("fp8", 3e-2, "llama"), ("nvfp4", 6e-2, "qwen3_1k")])
def test_quantised_program_matches_oracle(cuda_device, program, wkind, tol, base):
    test_gpu_decode.test_decode_quantised_matches_oracle(cuda_device, wkind, tol, base)


def test_full_size_layer_of_the_program_matches_hf_fixture(cuda_device, program):
    test_gpu_decode.test_full_size_llama_layer_matches_hf_fixture(cuda_device)


@pytest.mark.parametrize("cfg_kw,eng_kw", [
    (dict(), dict(num_sms=1)),                              # fewer SMs than KV heads
    (dict(ffn=16896, n_layers=1), dict(split_down=True)),   # rows of 33 KB, as two halves
    (dict(), dict(split_down=True)), (dict(), dict(shared_counters=True)), (dict(), dict(interleave=False))])
def test_steps_the_step_kernel_does_not_take(cuda_device, cfg_kw, eng_kw):
    """The engine runs them as a program of its own accord, and follows the oracle."""
    import dataclasses
    from vdcores_b200.decode import DecodeEngine
    cfg = dataclasses.replace(small_cfg("llama"), **cfg_kw)
    w = perturb_norms(O.ModelWeights.random(cfg, seed=9))
    prompt = torch.randint(0, cfg.vocab, (70,), generator=torch.Generator().manual_seed(4)).tolist()
    orc = O.DecodeOracle(w, 128)
    orc.prefill(prompt[:-1])
    eng = DecodeEngine(engine_config(cfg), max_seq=128, device=cuda_device, taps=True, timeout_ns=500_000_000, **eng_kw)
    eng.load_weights(dense_weights(w))
    assert eng.step_kernel is None
    eng.load_kv([k[:69] for k in orc.k], [v[:69] for v in orc.v])
    eng.set_state(69, prompt[-1])
    tok = prompt[-1]
    for _ in range(2):
        caps = []
        logits, nxt, gap = orc.step(tok, caps)
        got = eng.step_host(tok)
        for l in range(cfg.n_layers):
            assert O.rel_l2(eng.taps[l].cpu(), caps[l]["hidden_state_out"]) < test_gpu_decode.REL_L2_BF16
        assert O.rel_l2(eng.logits.cpu(), logits) < test_gpu_decode.REL_L2_BF16
        assert got == nxt or gap <= test_gpu_decode.GAP
        tok = nxt


@pytest.mark.parametrize("kind,prompt_len", [("llama", 70), ("moe", 40)])
def test_prefill_by_the_program_matches_oracle(cuda_device, program, kind, prompt_len):
    cfg, prompt, orc, nxt, gap, eng = test_gpu_prefill._setup(kind, prompt_len, cuda_device, seed=31)
    first = eng.prefill_device(prompt)
    test_gpu_prefill._check_cache_and_continue(cfg, prompt_len, orc, nxt, gap, eng, first)


@pytest.mark.parametrize("kind,prompt_len,chunk,perm", [("llama", 150, 16, None), ("qwen3", 100, 32, 3), ("llama", 200, 128, 9)])
def test_prefill_chunk_by_chunk_matches_oracle(cuda_device, monkeypatch, kind, prompt_len, chunk, perm):
    from vdcores_b200.prefill import PrefillEngine
    monkeypatch.setattr(PrefillEngine, "_goes_wide", lambda self, T: False)
    test_gpu_prefill.test_chunked_prefill_matches_oracle(cuda_device, kind, prompt_len, chunk, perm)


@pytest.mark.parametrize("kw,eng_kw", [(dict(vocab=2051), dict()), (dict(vocab=2058), dict(shared_counters=True)), (dict(vocab=5), dict()),
                                       (dict(vocab=64, hidden=2048, n_experts=76, top_k=4, ffn=256), dict())])
def test_rows_behind_the_last_whole_chunk(cuda_device, program, kw, eng_kw):
    """Vocabularies and experts that whole copies of a router's or a head's rows do not make up: every logit, and the largest."""
    from vdcores_b200.decode import DecodeConfig, DecodeEngine
    cfg = DecodeConfig(**{**dict(hidden=512, n_heads=8, n_kv_heads=2, ffn=512, n_layers=1, eps=1e-5, theta=5e5), **kw})
    eng = DecodeEngine(cfg, 128, device=cuda_device, timeout_ns=500_000_000, **eng_kw)
    eng.init_random_weights(3)
    for last in (False, True):
        if last:                # the last row is the largest for whatever the hidden state is then
            eng.lm_head[-1] = eng.norm_w * (20 * x)
        eng.set_state(20, 4)
        tok = eng.generate(1)[0]
        h = eng.hidden.float()
        x = (h * torch.rsqrt(h.pow(2).mean() + cfg.eps)).to(torch.bfloat16)
        want = (x * eng.norm_w).float() @ eng.lm_head.float().t()
        assert O.rel_l2(eng.logits.cpu(), want.cpu()) < 4e-3          # one rounding to bf16, 2^-9
        assert tok == int(eng.logits.float().argmax()) and (tok == cfg.vocab - 1 or not last)
    if cfg.n_experts:
        eng.router[0][:-4] = 0.0                                          # logits of zero and four that are not
        eng.router[0][-4:] = 0.1
        eng.set_state(20, 4)
        eng.generate(1)
        logits = eng.router_logits
        assert torch.equal(torch.topk(logits, 4).indices.sort().values, eng.route[:4].sort().values.to(torch.int64))
        assert not bool((logits[-4:] == 0).any())
