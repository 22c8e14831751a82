"""Host-side logic of the batched (tensor-core) decode path, without a GPU: operand layouts,
the dealing of projection work to SMs, and the memory streams the program builder emits
(expanded here by a small interpreter of REPEAT loops)."""
import pytest
import torch

from vdcores_b200 import isa
from vdcores_b200.batch import (BLOCK_ROWS, chunk_geometry, emit_projection, pack_blocks, pack_blocks_fp8, pack_kc,
                                plan_units, projection_blocks, unpack_kc)
from vdcores_b200.program import Program


def test_k_chunk_major_layout():
    x = torch.arange(32 * 64, dtype=torch.float32).view(32, 64)
    p = pack_kc(x)
    bp = 32
    for b, k in [(0, 0), (3, 9), (31, 63), (8, 8), (17, 40)]:
        off = ((k // 8) * (bp // 8) + b // 8) * 128 + (b % 8) * 16 + (k % 8) * 2       # bytes, as isa.h states it
        assert p[off // 2] == x[b, k]
    assert torch.equal(unpack_kc(p, 32, 64), x)
    # a K-range of the matrix is one contiguous piece
    assert torch.equal(p[16 * bp:48 * bp], pack_kc(x[:, 16:48].contiguous()))


def test_block_packing_keeps_k_ranges_contiguous():
    M, K = 256 + 256 + 96, 512
    w = torch.arange(M * K, dtype=torch.float32).view(M, K)
    pk = pack_blocks(w)
    for r0, n in projection_blocks(M):
        blk = pk[r0 * K:(r0 + n) * K]
        assert torch.equal(unpack_kc(blk, n, K), w[r0:r0 + n])
        kc = 64
        for c in (0, 3, K // kc - 1):
            assert torch.equal(blk[c * kc * n:(c + 1) * kc * n], pack_kc(w[r0:r0 + n, c * kc:(c + 1) * kc].contiguous()))


def test_fp8_block_packing_matches_the_in_kernel_conversion():
    """A 16-byte piece (16 k of one row) becomes the two adjacent 8-k pieces of the bf16 operand layout."""
    M, K, kc = 256, 256, 64
    codes = torch.randint(0, 256, (M, K), dtype=torch.uint8)
    pk = pack_blocks_fp8(codes)
    chunk = pk[0:M * kc]                                    # first W chunk of the block: [kc/16][M/8][8][16]
    out = torch.zeros(M * kc, dtype=torch.uint8)            # what the converting warps write (here: bytes, not bf16)
    pieces = chunk.view(-1, 16)
    for p in range(pieces.shape[0]):
        i16, row = divmod(p, M)
        out.view(-1, 8)[(2 * i16) * M + row] = pieces[p, :8]
        out.view(-1, 8)[(2 * i16 + 1) * M + row] = pieces[p, 8:]
    assert torch.equal(out, pack_kc(codes[:, :kc].contiguous()))


def test_plan_units_covers_every_step_once_and_balances():
    for M, K, S in [(6144, 4096, 148), (4096, 14336, 148), (28672, 4096, 148), (128256, 4096, 148), (640, 4096, 5),
                    (96, 512, 2)]:
        blocks = projection_blocks(M)
        kc, _ = chunk_geometry(blocks[0][1], 16, K)
        steps = K // kc
        load = [0] * S
        units = plan_units(blocks, steps, list(range(S)), load, kc * 2)
        seen = {}
        for sm, bi, c0, cnt in units:
            assert cnt > 0 and 0 <= c0 and c0 + cnt <= steps
            for c in range(c0, c0 + cnt):
                assert (bi, c) not in seen
                seen[(bi, c)] = sm
        assert len(seen) == len(blocks) * steps
        assert sum(load) == M * K * 2
        if S == 148:
            assert max(load) <= 1.15 * (sum(load) / S)


def expand_loads(minsts):
    """(address, bytes) of every 1-D load of one SM's memory stream, REPEAT loops unrolled."""
    out, i = [], 0
    deltas, count = {}, None
    while i < len(minsts):
        op, size, num_slots, arg, addr = minsts[i]
        opid = op >> isa.FLAG_BITS
        if opid == isa.op_id(isa.OP_REPEAT):
            lo, hi = num_slots & 0xFF, num_slots >> 8
            for lane in range(lo, hi):
                deltas[lane] = addr
            if size:
                count = size
            i += 1
            if count is not None and size:
                body = []
                while True:
                    body.append(minsts[i])
                    i += 1
                    if body[-1][0] & isa.F_JUMP:
                        break
                for it in range(count):
                    for j, (bop, bsize, _, _, baddr) in enumerate(body):
                        if bop >> isa.FLAG_BITS == isa.op_id(isa.OP_ALLOC_TMA_LOAD_1D):
                            out.append((baddr + it * deltas.get(j, 0), bsize))
                deltas, count = {}, None
            continue
        if opid == isa.op_id(isa.OP_ALLOC_TMA_LOAD_1D):
            out.append((addr, size))
        i += 1
    return out


def test_emitted_streams_read_every_weight_byte_once_and_the_right_activations():
    M, K, B, Bp, S = 1280, 2048, 12, 16, 7
    W_ADDR, X_ADDR, NORM = 1 << 30, 1 << 28, 1 << 27
    P = Program(S)
    bar = P.new_barrier()
    units = emit_projection(P, sms=list(range(S)), load=[0] * S, w_addr=W_ADDR, M=M, K=K, x_addr=X_ADDR, B=B, Bpad=Bp,
                            mode=isa.GEMM_MODE_STORE_ROWS, out_addr=1 << 26, scratch_addr=1 << 25, counter_addr=1 << 24,
                            release=bar, norm_addr=NORM, eps=1e-5, ld=M, stats_addr=1 << 23)
    assert P.bar_counts[bar] == len(projection_blocks(M))          # one release per block (its last arriver)
    w_bytes, x_total, n_total = [], 0, 0
    for sm in range(S):
        for addr, n in expand_loads(P.m[sm]):
            if W_ADDR <= addr < W_ADDR + M * K * 2:
                w_bytes.append((addr, n))
            elif X_ADDR <= addr < X_ADDR + Bp * K * 2:
                x_total += n
            elif NORM <= addr < NORM + K * 2:
                n_total += n
            else:
                raise AssertionError(hex(addr))
    w_bytes.sort()
    pos = W_ADDR
    for addr, n in w_bytes:                                        # contiguous, no gap, no overlap
        assert addr == pos
        pos += n
    assert pos == W_ADDR + M * K * 2
    k_streamed = sum(cnt for _, _, _, cnt in units) * chunk_geometry(BLOCK_ROWS, Bp, K)[0]
    assert x_total == Bp * k_streamed * 2                          # every unit reads the activations of its K-range
    assert n_total == k_streamed * 2                               # and the matching slice of the norm weights
    # compute side: one task per unit, eleven words each
    assert sum(1 for sm in range(S) for c in P.c[sm] if c[0] == isa.OP_GEMM_TC_BF16) == len(units)
    assert all(len(P.c[sm]) % 11 == 0 for sm in range(S))


def test_prefill_state_blocks_of_a_chunk():
    """Row b of chunk c: its position, page count, token, cache row and page table; rows past the prompt repeat the last."""
    import types
    import numpy as np
    from vdcores_b200.prefill import PrefillEngine
    table = torch.tensor([3, 0, 4, 1, 2], dtype=torch.int32)
    e = types.SimpleNamespace(batch=48, page_table=table, max_pages=5, cfg=types.SimpleNamespace(n_kv_heads=2))
    tokens = np.arange(1000, 1130, dtype=np.int32)      # 130 positions: chunks of 48, 48 and 34
    for c in range(3):
        s = np.full((48, isa.ST_PAGETABLE + 5), -7, dtype=np.int32)
        PrefillEngine._fill_states(e, s, tokens, c)
        for b in range(48):
            pos = min(c * 48 + b, 129)
            assert s[b, isa.ST_POS] == pos and s[b, isa.ST_TOKEN] == 1000 + pos and s[b, isa.ST_NPAGES] == pos // 64 + 1
            assert s[b, isa.ST_NEWROW] == int(table[pos // 64]) * 64 * 2 + pos % 64
            assert s[b, isa.ST_NKVH] == 2 and s[b, isa.ST_MAXPAGES] == 5 and s[b, isa.ST_STEP] == 0 and s[b, isa.ST_ERR] == 0
            assert (s[b, isa.ST_PAGETABLE:] == table.numpy()).all()


def test_stages_refuse_bad_arguments():
    """The check that a launch runs over its whole list first; no GPU is needed for it."""
    from vdcores_b200 import isa, runtime
    a = 1 << 20         # aligned; never read
    heads = dict(group=4, n_kv=1, state=a, state_stride=isa.ST_PAGETABLE + 3, kpool=a, vpool=a)
    proj = dict(kind=isa.STAGE_GEMM, B=2, Bpad=16, K=128, splits=1, w=a, x=a)
    kinds = [
        (dict(proj, mode=isa.STAGE_SILU, M=64, out=a),
         [dict(K=96), dict(M=8), dict(splits=3), dict(splits=4), dict(Bpad=24), dict(B=17), dict(w=0), dict(x=a + 8), dict(wfmt=1),
          dict(kind=9), dict(mode=7), dict(out=a + 8), dict(wfmt=1, scales=a + 4)]),
        (dict(proj, mode=isa.STAGE_RESID, M=64, hid=a, stats_out=a), [dict(hid=a + 8), dict(hid=0), dict(stats_out=a + 2)]),
        (dict(proj, mode=isa.STAGE_ARGMAX, M=64, keys=a), [dict(keys=a + 4), dict(keys=0)]),
        (dict(proj, mode=isa.STAGE_QKV, M=768, out=a, rope=a, **heads),
         [dict(M=896), dict(out=a + 2), dict(rope=a + 4), dict(qk_norm=a + 2), dict(kpool=a + 8), dict(vpool=a + 8), dict(state=0),
          dict(state=a + 2), dict(state_stride=4)]),
        (dict(kind=isa.STAGE_ATTN, B=2, Bpad=16, splits=1, n_pages=3, q=a, out=a, **heads),
         [dict(group=5), dict(q=a + 8), dict(out=a + 8), dict(kpool=0), dict(vpool=a + 8), dict(n_pages=0), dict(n_pages=4), dict(splits=16)]),
        (dict(kind=isa.STAGE_ATTN_PREFILL, B=2, Bpad=16, splits=1, n_pages=3, q=a, out=a, **heads), [dict(n_pages=4), dict(group=2)]),
        (dict(kind=isa.STAGE_EMBED, B=2, Bpad=16, M=8, K=64, w=a, hid=a, stats_out=a, n_stats=1, state=a, state_stride=64),
         [dict(K=0), dict(K=60), dict(w=a + 8), dict(hid=a + 8), dict(n_stats=0), dict(M=-1), dict(state=0), dict(state_stride=1)]),
        (dict(kind=isa.STAGE_NORM, B=2, Bpad=16, K=64, x=a, out=a, stats_in=a, norm_w=a),
         [dict(K=0), dict(x=a + 8), dict(out=0), dict(norm_w=a + 2), dict(stats_in=a + 1)]),
        (dict(kind=isa.STAGE_ADVANCE, B=2, Bpad=16, keys=a, log=a, state=a, state_stride=64),
         [dict(keys=a + 4), dict(log=a + 2), dict(state=0), dict(state_stride=isa.ST_PAGETABLE)])]
    for good, bads in kinds:
        runtime.count_stage_launches((runtime.Stage * 1)(runtime.Stage(**good)))
        for bad in bads:
            with pytest.raises(runtime.VdcError):
                runtime.count_stage_launches((runtime.Stage * 1)(runtime.Stage(**{**good, **bad})))


@pytest.mark.parametrize("limit", [1, 7, 61, 147])
def test_slices_of_a_limited_launch(limit):
    """Whole clusters, never more than the limit, all units once: per kind the number of launches and the largest."""
    from vdcores_b200 import isa, runtime
    a = 1 << 20
    common = dict(B=100, Bpad=128, w=a, x=a, out=a, hid=a, stats_out=a, stats_in=a, norm_w=a, keys=a, log=a, state=a, q=a, kpool=a,
                  vpool=a, n_stats=1, state_stride=64, group=4, n_kv=8, n_pages=9, K=4096)
    for kind, units, splits, more in ((isa.STAGE_GEMM, 113, 4, dict(M=14400, mode=isa.STAGE_SILU)),
                                      (isa.STAGE_GEMM, 32, 1, dict(M=4096, mode=isa.STAGE_RESID)), (isa.STAGE_ATTN, 800, 1, {}),
                                      (isa.STAGE_ATTN_PREFILL, 56, 2, {}), (isa.STAGE_NORM, 256, 1, {}), (isa.STAGE_EMBED, 100, 1, {}),
                                      (isa.STAGE_ADVANCE, 1, 1, {})):
        st = (runtime.Stage * 1)(runtime.Stage(kind=kind, splits=splits, **{**common, **more}))
        assert runtime.count_stage_launches(st) == (1, units * splits)
        if splits > limit:
            with pytest.raises(runtime.VdcError, match="splits"):
                runtime.count_stage_launches(st, limit)
            continue
        launches, largest = runtime.count_stage_launches(st, limit)
        per = limit // splits
        assert launches == -(-units // per) and largest == min(units, per) * splits <= limit
