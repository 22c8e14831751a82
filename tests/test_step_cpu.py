"""Which steps the step kernel takes (csrc/step_kernel.cu): its limits are checked on the host, without a GPU."""
import pytest


def step(hidden, ffn, num_sms, n_kv=1, group=4, vocab=64, experts=0, top_k=0, wfmt=0, splits=1):
    from vdcores_b200 import runtime
    return runtime.Step(num_sms=num_sms, n_layers=1, hidden=hidden, ffn=ffn, vocab=vocab, n_kv=n_kv, group=group, wfmt=wfmt,
                        max_pages=4, n_splits=splits, n_experts=experts, top_k=top_k, eps=1e-5, qk_eps=1e-5)


def division(K, n, experts, wfmt=0):
    """Warps that keep a sum of every one of an SM's n rows of K inputs.  Four dense bf16 rows that are longer than a copy of 32 KB
    come in slices, which all eight warps divide, while 4224 floats hold eight sums of each; otherwise two teams of warps take the
    chunks in turn (four for NVFP4 rows and experts), and a team's warps divide the inputs as far as they would have fewer than
    four rows of a chunk each."""
    steps, row = K // (256 << wfmt), (2 * K, K, K // 2 + K // 16)[wfmt]
    if wfmt == 0 and not experts and steps > 16 and 4 <= n <= 528:
        return 8
    per = max(1, min(32, 32768 // row) // 2 * 2)
    teams = 4 if (experts or wfmt == 2) and n // per >= 4 else 2 if n // per >= 2 else 1
    warps, kw = 8 // teams, 1
    while kw < warps and 2 * kw <= steps and min(n, per) < 4 * (warps // kw):
        kw *= 2
    return kw


def sums_and_room(rows, unit, K, num_sms, slots, experts):
    """Partial sums of the SMs with the most rows and of those with a unit less, and the room for them."""
    most = -(-(rows // unit) // num_sms) * unit
    return [(n * slots, 4224 // division(K, n * slots, experts)) for n in (most, most - unit) if n]


@pytest.mark.parametrize("hidden,ffn,num_sms,experts,top_k,taken", [
    (6912, 512, 23, 8, 7, True),         # the down projection of 7 experts: 302 rows of 7 sums, of 13 and of 14; room for 4224
    (6912, 512, 23, 16, 13, True),
    (6912, 512, 23, 16, 14, False),
    (2560, 768, 79, 64, 16, True),       # 34 rows of 16 sums
    (1024, 4352, 8, 0, 0, True),         # gate and up: 1088 rows that no two warps divide
    (1024, 14592, 7, 0, 0, True),        # 4172 rows
    (1024, 14848, 7, 0, 0, False),       # 4244
    (4608, 4608, 17, 0, 0, True),        # rows of 9 KB: 544 whole, 540 of them
    (5120, 2048, 16, 0, 0, True),        # 256 in slices
    (8192, 1024, 2, 0, 0, True),         # two rows to a chunk, inputs divided by four: 1024 rows, room for 1056
    (8192, 1280, 2, 0, 0, False)])
def test_partial_sums_of_a_taken_step_fit(hidden, ffn, num_sms, experts, top_k, taken):
    from vdcores_b200 import runtime
    k = top_k or 1
    stages = [(768, 2, hidden, 1), (hidden, 2, 512, 1), (2 * ffn * k, 4, hidden, 1), (hidden, 2, ffn, k)]
    room = all(need <= have for rows, unit, K, slots in stages
               for need, have in sums_and_room(rows, unit, K, num_sms, slots, experts > 0))
    assert room == taken
    assert (runtime.step_workspace(step(hidden, ffn, num_sms, experts=experts, top_k=top_k)) is not None) == taken


@pytest.mark.parametrize("hidden,ffn,taken", [
    (4096, 49152, True),         # inputs and hidden state leave 96 KB, of which the scales take 4
    (8192, 45056, True),
    (4096, 50176, False),
    (8192, 46080, False)])
def test_scales_take_nothing_from_what_a_wide_step_needs(hidden, ffn, taken):
    """NVFP4 rows of the widest projections: 2-byte inputs and hidden state, 26496 bytes of sums, heads and probabilities, and a ring
    of three copies of 32 KB share 231296 bytes."""
    from vdcores_b200 import runtime
    assert (2 * (hidden + ffn) + 26496 + 3 * 32768 <= 231296) == taken
    assert (runtime.step_workspace(step(hidden, ffn, 148, n_kv=8, wfmt=2, splits=4)) is not None) == taken
