"""Batched decode: the batched glue kernels against their single-sequence forms on identical inputs
(bit for bit), and the whole batched step against single-sequence engines on the same weights."""

import ctypes

import pytest
import torch

from conftest import rel_l2
from gpu_util import RawPool
from leankv_b200 import _native
from leankv_b200.batch_engine import BatchDecodeEngine
from leankv_b200.engine import DecodeEngine, DecoderConfig

pytestmark = pytest.mark.gpu

CFG = DecoderConfig(vocab_size=1024, hidden_size=512, intermediate_size=1024, num_layers=2, num_q_heads=8,
                    num_kv_heads=2)


def _dev():
    return torch.device("cuda:0")


def _st():
    return torch.cuda.current_stream().cuda_stream


def test_rmsnorm_rows_equals_single_row_kernel():
    lib = _native.lib()
    g = torch.Generator(device=_dev()).manual_seed(0)
    rows, n = 5, 4096
    x = torch.randn(rows, n, device=_dev(), generator=g).half()
    d = torch.randn(rows, n, device=_dev(), generator=g).half()
    w = torch.randn(n, device=_dev(), generator=g).half()
    xa, ya = x.clone(), torch.empty_like(x)
    _native.check(lib.leankv_rmsnorm_rows_f16(xa.data_ptr(), d.data_ptr(), w.data_ptr(), ya.data_ptr(), rows, n,
                                              1e-5, _st()), "rows")
    for r in range(rows):
        xb, yb = x[r].clone(), torch.empty(n, dtype=torch.float16, device=_dev())
        _native.check(lib.leankv_rmsnorm_f16(xb.data_ptr(), d[r].data_ptr(), w.data_ptr(), yb.data_ptr(), n, 1e-5,
                                             _st()), "row")
        torch.cuda.synchronize()
        assert torch.equal(xa[r], xb) and torch.equal(ya[r], yb)


def test_silu_mul_rounding_points():
    lib = _native.lib()
    g = torch.Generator(device=_dev()).manual_seed(1)
    rows, inter = 7, 1024
    gu = (torch.randn(rows, 2 * inter, device=_dev(), generator=g) * 3).half()
    out = torch.empty(rows, inter, dtype=torch.float16, device=_dev())
    _native.check(lib.leankv_silu_mul_f16(gu.data_ptr(), out.data_ptr(), rows, inter, _st()), "silu_mul")
    torch.cuda.synchronize()
    gate, up = gu[:, :inter].float(), gu[:, inter:]
    want = (gate * torch.sigmoid(gate)).half() * up
    # __expf differs from torch's exp in the last bits: allow one fp16 ulp on the activation
    err = (out.float() - want.float()).abs()
    assert float((err / (want.float().abs() + 1e-3)).max()) < 3e-3
    assert rel_l2(out, want) < 1e-3


def test_batch_begin_builds_the_flat_page_table():
    lib = _native.lib()
    B, pps, hidden, vocab = 6, 9, 256, 50
    g = torch.Generator().manual_seed(2)
    table = torch.randn(vocab, hidden, generator=g).half().to(_dev())
    tokens = torch.tensor([3, 49, 0, 7, 7, 21], device=_dev())
    pos = torch.tensor([0, 15, 16, 47, 100, 143], dtype=torch.int32, device=_dev())
    bt = torch.randperm(B * pps, generator=g).to(torch.int32).reshape(B, pps).to(_dev())
    h = torch.zeros(B, hidden, dtype=torch.float16, device=_dev())
    indptr = torch.zeros(B + 1, dtype=torch.int32, device=_dev())
    flat = torch.full((B * pps,), -1, dtype=torch.int32, device=_dev())
    last = torch.zeros(B, dtype=torch.int32, device=_dev())
    _native.check(lib.leankv_batch_decode_begin(table.data_ptr(), tokens.data_ptr(), h.data_ptr(), hidden, vocab, B,
                                                pos.data_ptr(), bt.data_ptr(), pps, indptr.data_ptr(),
                                                flat.data_ptr(), last.data_ptr(), _st()), "begin")
    torch.cuda.synchronize()
    assert torch.equal(h, table[tokens])
    used = [int(p) // 16 + 1 for p in pos.tolist()]
    want_indptr = [0]
    for u in used:
        want_indptr.append(want_indptr[-1] + u)
    assert indptr.tolist() == want_indptr
    assert last.tolist() == [int(p) % 16 + 1 for p in pos.tolist()]
    want_flat = torch.cat([bt[b, :used[b]] for b in range(B)])
    assert torch.equal(flat[:want_indptr[-1]], want_flat)


def test_batch_decode_end_is_rowwise_argmax():
    lib = _native.lib()
    B, vocab, cap = 5, 4096, 12
    g = torch.Generator(device=_dev()).manual_seed(3)
    logits = torch.randn(B, vocab, device=_dev(), generator=g).half()
    logits[2, 100] = logits[2, 3000] = 9.0          # tie: lowest index wins
    tokens = torch.zeros(B, dtype=torch.int64, device=_dev())
    hist = torch.zeros(B, cap, dtype=torch.int64, device=_dev())
    pos = torch.arange(10, 10 + B, dtype=torch.int32, device=_dev())
    steps = torch.tensor([0, 1, 2, 3, 11], dtype=torch.int32, device=_dev())
    _native.check(lib.leankv_batch_decode_end(logits.data_ptr(), vocab, B, tokens.data_ptr(), hist.data_ptr(), cap,
                                              pos.data_ptr(), steps.data_ptr(), _st()), "end")
    torch.cuda.synchronize()
    want = logits.float().argmax(dim=-1)
    want[2] = 100
    assert torch.equal(tokens, want)
    assert pos.tolist() == list(range(11, 11 + B)) and steps.tolist() == [1, 2, 3, 4, 12]
    for b, s in enumerate([0, 1, 2, 3, 11]):
        assert int(hist[b, s]) == int(want[b])


@pytest.mark.parametrize("vocab", [1, 7, 8, 31, 64, 4093, 32768, 50001])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_decode_end_over_the_shares_of_a_cluster(vocab, dtype):
    """Best value in every share of the vocabulary and in the remainder, ties (the lowest index), NaN beside numbers, no number at all."""
    lib = _native.lib() if dtype == torch.float16 else _native.mixers()
    end = lib.leankv_decode_end if dtype == torch.float16 else lib.leankv_greedy_end
    rows = []
    for at in sorted({0, vocab // 2, vocab - 1, *(vocab * r // 8 for r in range(8))}):
        row = torch.linspace(-1, 1, vocab).to(dtype)
        row[at] = 5.0
        rows.append(row.clone())
        row[vocab - 1] = 5.0
        row[vocab // 3] = float("nan") if vocab // 3 != at and vocab > 1 else row[vocab // 3]
        rows.append(row)
    rows.append(torch.full((vocab,), float("nan"), dtype=dtype))
    for row in rows:
        want = int(row.float().nan_to_num(nan=-10.0).argmax()) if not bool(row.isnan().all()) else 0
        want = int((row == row[want]).nonzero()[0]) if not bool(row.isnan().all()) else 0
        dev, token = row.to(_dev()), torch.full((1,), -1, dtype=torch.int64, device=_dev())
        hist, state = torch.zeros(4, dtype=torch.int64, device=_dev()), torch.zeros(8, dtype=torch.int32, device=_dev())
        state[:2] = torch.tensor([10, 2])
        _native.check(end(dev.data_ptr(), vocab, token.data_ptr(), hist.data_ptr(), 4, state.data_ptr(), _st()), "end")
        torch.cuda.synchronize()
        assert int(token) == want == int(hist[2]) and state[:2].tolist() == [11, 3]


@pytest.mark.parametrize("B", [1, 48, 49, 64, 65, 200])
@pytest.mark.parametrize("vocab", [8, 4096, 32776])
def test_batch_decode_end_of_few_and_many_sequences(B, vocab):
    """Either side of the line between a cluster and a CTA for each: ties (the lowest index), rows of NaN, a full history."""
    g = torch.Generator(device=_dev()).manual_seed(B)
    logits = torch.randint(-40, 40, (B, vocab), device=_dev(), generator=g).half()
    logits[B // 2, vocab // 2:] = float("nan")
    logits[B - 1] = float("nan") if B > 1 else logits[B - 1]
    tok, hist = torch.full((B,), -1, dtype=torch.int64, device=_dev()), torch.full((B, 3), -1, dtype=torch.int64, device=_dev())
    pos, steps = torch.arange(B, dtype=torch.int32, device=_dev()), (torch.arange(B, device=_dev()) % 4).to(torch.int32)
    p0, s0 = pos.clone(), steps.clone()
    _native.check(_native.lib().leankv_batch_decode_end(logits.data_ptr(), vocab, B, tok.data_ptr(), hist.data_ptr(), 3, pos.data_ptr(),
                                                        steps.data_ptr(), _st()), "end")
    x = logits.float().nan_to_num(nan=-1e9)
    want = (x == x.amax(1, keepdim=True)).int().argmax(1)
    assert torch.equal(tok, want) and torch.equal(pos, p0 + 1) and torch.equal(steps, s0 + 1)
    for b in range(B):
        assert hist[b].tolist() == [int(want[b]) if s == int(s0[b]) else -1 for s in range(3)]


@pytest.mark.parametrize("rows", [1, 15, 17, 48, 80, 128])
@pytest.mark.parametrize("k,n", [(8, 8), (64, 128), (72, 136), (1000, 520), (3584, 1024), (520, 8192), (128, 40000)])
def test_skinny_gemm_edges(rows, k, n):
    """Rows beyond a product's sixteen, K and N with remainders, one to eight CTAs a column block, more blocks than CTAs at once:
    against float64. The sums are fp32 (below 1e-5 of the result), so the fp16 rounding of the outputs, 2^-11 a value, bounds it."""
    lib = _native.lib()
    g = torch.Generator(device=_dev()).manual_seed(rows + k)
    x = torch.randn(rows, k, device=_dev(), generator=g).half()
    w = (torch.randn(k, n, device=_dev(), generator=g) * k ** -0.5).half()
    y = torch.full((rows + 1, n), 7.0, dtype=torch.float16, device=_dev())
    want = x.double() @ w.double()
    for early in (0, 1):
        _native.check(lib.leankv_skinny_gemm_f16(x.data_ptr(), w.data_ptr(), y.data_ptr(), rows, k, n, early, _st()), "skinny_gemm")
        torch.cuda.synchronize()
        assert bool((y[rows] == 7.0).all())
        assert float((y[:rows].double() - want).norm()) <= 2 ** -11 * float(want.norm())


@pytest.mark.parametrize("flags", [2, 3])
def test_skinny_gemm_that_takes_its_tensor_memory_first(flags):
    """Behind a launch of CUDA cores, in a row of both: the bits of a launch in plain order."""
    lib, rows, k, n = _native.lib(), 33, 520, 2056
    g = torch.Generator(device=_dev()).manual_seed(3)
    x = torch.randn(rows, k, device=_dev(), generator=g).half()
    w = (torch.randn(k, n, device=_dev(), generator=g) * k ** -0.5).half()
    gain = torch.ones(k, dtype=torch.float16, device=_dev())
    outs = [torch.empty(rows, n, dtype=torch.float16, device=_dev()) for _ in range(21)]
    for i, y in enumerate(outs):
        h = torch.empty_like(x)
        _native.check(lib.leankv_rmsnorm_rows_f16(x.data_ptr(), None, gain.data_ptr(), h.data_ptr(), rows, k, 1e-5, _st()), "norm")
        _native.check(lib.leankv_skinny_gemm_f16(h.data_ptr(), w.data_ptr(), y.data_ptr(), rows, k, n, flags if i else 0, _st()), "gemm")
    torch.cuda.synchronize()
    assert all(torch.equal(y, outs[0]) for y in outs[1:])


@pytest.mark.parametrize("early", [0, 1])
def test_skinny_gemm_next_to_kernels_with_tensor_memory(early):
    """Prompt attention holds all of an SM's tensor memory: a projection right behind it, and it right behind a projection, without the
    host in between, give the bits that each gives alone."""
    lib, T, H, rows, k, n = _native.lib(), 333, 2, 40, 1032, 1544
    g = torch.Generator(device=_dev()).manual_seed(8)
    rp = RawPool(64, H, _dev())
    kv = [torch.randn(1, H, T, 128, device=_dev(), generator=g).half() for _ in range(2)]
    rp.append(*kv, [0, 21], range(21), [0])
    q = torch.randn(T, 4 * H, 128, device=_dev(), generator=g).half()
    pages, attended = rp.i32(range(21)), rp.prefill_attention(q, range(21), 0)
    x = torch.randn(rows, k, device=_dev(), generator=g).half()
    w = (torch.randn(k, n, device=_dev(), generator=g) * k ** -0.5).half()
    ws = torch.zeros(lib.leankv_tq_prefill_attn_workspace_bytes(T, 0, 4 * H, H), dtype=torch.uint8, device=_dev())
    outs = [(torch.empty_like(q), torch.empty(rows, n, dtype=torch.float16, device=_dev())) for _ in range(20)]

    def project(y):
        _native.check(lib.leankv_skinny_gemm_f16(x.data_ptr(), w.data_ptr(), y.data_ptr(), rows, k, n, early, _st()), "skinny_gemm")

    alone = torch.empty(rows, n, dtype=torch.float16, device=_dev())
    project(alone)
    torch.cuda.synchronize()
    for out, y in outs:
        _native.check(lib.leankv_tq_prefill_attn(q.data_ptr(), out.data_ptr(), T, 0, 4 * H, H, rp.pool.data_ptr(), rp.n_pages,
                                                 pages.data_ptr(), rp.Pi_k.data_ptr(), rp.Pi_v.data_ptr(), rp.centroids_host.data_ptr(),
                                                 128 ** -0.5, ws.data_ptr(), ws.numel(), _st()), "prefill_attn")
        project(y)
    torch.cuda.synchronize()
    assert all(torch.equal(out, attended) and torch.equal(y, alone) for out, y in outs)


@pytest.mark.parametrize("rows,k,n,own", [(48, 512, 1024, True), (48, 512, 1032, False), (49, 512, 512, False), (3, 4096, 8192, True),
                                          (3, 4200, 8200, False), (2, 20000, 4000, True), (2, 20000, 4008, False), (2, 516, 512, False)])
def test_which_projections_are_this_library_s(rows, k, n, own):
    """Either side of each line; both give the product to one fp16 rounding."""
    eng = BatchDecodeEngine.random_init(CFG, _dev(), 2, seed=1, max_seq_len=64)
    g = torch.Generator(device=_dev()).manual_seed(rows + n)
    x = torch.randn(rows, k, device=_dev(), generator=g).half()
    w = (torch.randn(k, n, device=_dev(), generator=g) * k ** -0.5).half()
    y, before = torch.empty(rows, n, dtype=torch.float16, device=_dev()), eng.own_gemms_per_step
    eng._mm(x, w, y)
    assert eng.own_gemms_per_step - before == int(own)
    want = x.double() @ w.double()
    assert float((y.double() - want).norm()) <= 2 ** -11 * float(want.norm())


def test_a_projection_that_gave_up_is_reported():
    """The word that the kernels set is the one that the engine reads: untouched by steps that end well, an error once it is set."""
    eng = BatchDecodeEngine.random_init(CFG, _dev(), 3, seed=1, max_seq_len=64)
    prompts = torch.arange(3 * 20).reshape(3, 20)
    eng.generate(prompts, 4)
    assert eng.own_gemms_per_step > 0 and eng.status_words() == (0, 0)
    eng.ws_attn[:4].view(torch.int32).fill_(8)
    with pytest.raises(RuntimeError, match="projection"):
        eng.check_status()
    with pytest.raises(RuntimeError, match="projection"):
        eng.generate(prompts, 4)


def test_batch_qkv_post_is_bit_identical_to_single_sequence_kernel():
    """Same qkv rows, positions and pages through the batched launch and through one launch per sequence."""
    lib = _native.lib()
    B = 11
    eng = BatchDecodeEngine.random_init(CFG, _dev(), B, seed=1, max_seq_len=160)
    g = torch.Generator(device=_dev()).manual_seed(4)
    qkv = torch.randn(B, eng.n_qkv, device=_dev(), generator=g).half()
    pos = torch.tensor([0, 1, 15, 16, 17, 31, 32, 77, 100, 158, 159], dtype=torch.int32, device=_dev())
    eng.pos.copy_(pos)
    # page table of this step
    _native.check(lib.leankv_batch_decode_begin(eng.w["embed"].data_ptr(), eng.tokens.data_ptr(), eng.h.data_ptr(),
                                                CFG.hidden_size, CFG.vocab_size, B, eng.pos.data_ptr(),
                                                eng.block_table.data_ptr(), eng.pps, eng.kv_indptr.data_ptr(),
                                                eng.kv_page_indices.data_ptr(), eng.kv_last.data_ptr(), _st()), "begin")
    base = torch.randint(0, 256, eng.pools[0].shape, dtype=torch.uint8, device=_dev(), generator=g)
    pool_a, pool_b = base.clone(), base.clone()
    q_a = torch.zeros(B, eng.nq, 128, dtype=torch.float32, device=_dev())
    q_b = torch.zeros_like(q_a)
    _native.check(lib.leankv_batch_qkv_post(qkv.data_ptr(), B, eng.inv_freq.data_ptr(), eng.pos.data_ptr(),
                                            eng.kv_indptr.data_ptr(), eng.Pi_k_t[0].data_ptr(),
                                            eng.Pi_v_t[0].data_ptr(), eng.bounds.data_ptr(), pool_a.data_ptr(),
                                            eng.max_pages, eng.kv_page_indices.data_ptr(), eng.nq, eng.nkv,
                                            q_a.data_ptr(), _st()), "batch post")
    state = torch.zeros(8, dtype=torch.int32, device=_dev())
    for b in range(B):
        state[0] = pos[b]
        pages = eng.block_table[b].contiguous()
        _native.check(lib.leankv_decode_qkv_post(qkv[b].data_ptr(), eng.inv_freq.data_ptr(), state.data_ptr(),
                                                 eng.Pi_k_t[0].data_ptr(), eng.Pi_v_t[0].data_ptr(),
                                                 eng.bounds.data_ptr(), pool_b.data_ptr(), eng.max_pages,
                                                 pages.data_ptr(), eng.nq, eng.nkv, q_b[b].data_ptr(), _st()), "post")
        torch.cuda.synchronize()
    assert torch.equal(q_a, q_b)
    assert torch.equal(pool_a, pool_b)
    assert not torch.equal(pool_a, base)


@pytest.mark.parametrize("B,n_q,n_kv", [(1, 8, 2), (11, 8, 2), (48, 32, 8)])
def test_qkv_post_with_the_early_flag_writes_the_same_bits(B, n_q, n_kv):
    """One sequence, a CTA for every four sequences, and CTAs that walk several groups; behind a launch that writes the projections only."""
    lib, g, pages = _native.lib(), torch.Generator(device=_dev()).manual_seed(B), 4
    rp = RawPool(pages * B, n_kv, _dev())
    n, Pk, Pv = (n_q + 2 * n_kv) * 128, rp.Pi_k.t().contiguous(), rp.Pi_v.t().contiguous()
    src, qkv = torch.randn(B, n, device=_dev(), generator=g).half(), torch.empty(B, n, dtype=torch.float16, device=_dev())
    ones, inv = torch.ones(n, dtype=torch.float16, device=_dev()), 10000.0 ** (-torch.arange(64, device=_dev()) / 64)
    pos = torch.randint(0, 16 * pages, (B,), device=_dev(), generator=g).to(torch.int32)
    state = torch.zeros(8, dtype=torch.int32, device=_dev())
    state[0] = pos[0]
    indptr, pages_of = rp.i32(range(0, pages * B + 1, pages)), rp.i32(reversed(range(pages * B)))
    base = torch.randint(0, 256, rp.pool.shape, dtype=torch.uint8, device=_dev(), generator=g)
    got = []
    for flags in (0, _native.POST_EARLY):
        for _ in range(5):
            pool, q = base.clone(), torch.zeros(B, n_q, 128, device=_dev())
            qkv.zero_()
            _native.check(lib.leankv_rmsnorm_rows_f16(src.data_ptr(), None, ones.data_ptr(), qkv.data_ptr(), B, n, 1e-5, _st()), "norm")
            rest = (Pk.data_ptr(), Pv.data_ptr(), rp.bounds.data_ptr(), pool.data_ptr(), rp.n_pages, pages_of.data_ptr(), n_q, n_kv,
                    q.data_ptr(), flags, _st())
            if B == 1:
                rc = lib.leankv_decode_qkv_post_flags(qkv.data_ptr(), inv.data_ptr(), state.data_ptr(), *rest)
            else:
                rc = lib.leankv_batch_qkv_post_flags(qkv.data_ptr(), B, inv.data_ptr(), pos.data_ptr(), indptr.data_ptr(), *rest)
            _native.check(rc, "post")
            got.append((pool, q))
    torch.cuda.synchronize()
    assert not torch.equal(got[0][0], base) and got[0][1].abs().sum() > 0
    assert all(torch.equal(p, got[0][0]) and torch.equal(q, got[0][1]) for p, q in got[1:])


def test_batched_step_matches_single_sequence_engines():
    """Dense projections either way (no thresholds): library GEMM rows vs the GEMV kernel differ in
    summation order only, so logits agree to fp16 rounding while tokens are teacher-forced."""
    B, T, n_new = 3, 40, 6
    g = torch.Generator().manual_seed(5)
    prompts = torch.randint(0, CFG.vocab_size, (B, T), generator=g)
    forced = torch.randint(0, CFG.vocab_size, (n_new, B), generator=g)

    eng = BatchDecodeEngine.random_init(CFG, _dev(), B, seed=9, max_seq_len=96)
    eng.prefill(prompts)
    got = [eng.prefill_logits.float().cpu()]
    for i in range(n_new):
        eng.tokens.copy_(forced[i].to(_dev()))
        eng.step()
        torch.cuda.synchronize()
        got.append(eng.logits.float().cpu())
    assert eng.pos.tolist() == [T + n_new] * B
    # 1 begin + 1 norm + per block (post, attention, norm, silu_mul, norm) + argmax; 4 GEMMs per block + lm_head
    assert eng.launches_per_step == 2 + 5 * CFG.num_layers + 1
    assert eng.gemms_per_step == 4 * CFG.num_layers + 1

    for b in range(B):
        one = DecodeEngine.random_init(CFG, _dev(), seed=9, max_seq_len=96)
        one.prefill(prompts[b].tolist())
        assert rel_l2(got[0][b], one.prefill_logits.float().cpu()) < 5e-3
        for i in range(n_new):
            one.token.fill_(int(forced[i, b]))
            one.step()
            torch.cuda.synchronize()
            err = rel_l2(got[i + 1][b], one.logits.float().cpu())
            assert err < 2e-2, (b, i, err)


def test_generate_returns_history_and_graph_equals_eager():
    B, T = 4, 33
    g = torch.Generator().manual_seed(6)
    prompts = torch.randint(0, CFG.vocab_size, (B, T), generator=g)
    a = BatchDecodeEngine.random_init(CFG, _dev(), B, seed=2, max_seq_len=64)
    toks = a.generate(prompts, 8)
    assert toks.shape == (B, 8)
    b = BatchDecodeEngine.random_init(CFG, _dev(), B, seed=2, max_seq_len=64)
    b.prefill(prompts)
    for _ in range(7):
        b.step(use_graph=False)
    torch.cuda.synchronize()
    assert torch.equal(toks, b.history[:, :8])
    assert a.kv_bytes_per_sequence(4096) == 256 * 2 * CFG.num_layers * CFG.num_kv_heads * 800


_OVERLAP_SNIPPET = r"""
import hashlib, sys, torch
sys.path[:0] = [%(root)r, %(tests)r]
from leankv_b200.batch_engine import BatchDecodeEngine
from leankv_b200.engine import DecodeEngine, DecoderConfig
from leankv_b200.mixer_engine import MixerDecodeEngine, MixerModelConfig
from leankv_b200.turboquant.quantizer import TurboQuantMSE
import pefitar_util, rorosun_util
dev, out = torch.device("cuda:0"), []
cfg = DecoderConfig(vocab_size=512, hidden_size=1024, intermediate_size=2048, num_layers=2, num_q_heads=8, num_kv_heads=2)
one = DecodeEngine.random_init(cfg, dev, seed=1, max_seq_len=700)
one.prefill([t %% 512 for t in range(600)], chunk=256)
for _ in range(4):
    one.step()
out += [one.logits, one.prefill_logits]
many = BatchDecodeEngine.random_init(cfg, dev, 5, seed=2, max_seq_len=128)
out.append(many.generate(torch.arange(5 * 100).reshape(5, 100) %% 512, 6))
for util in (rorosun_util, pefitar_util):
    layers = ([util.layer(heads=8, kv_heads=2, dim=64, vdim=64, size=48, pool=8, r_heads=4, r_dim=64, ff=320)] * 2 if util is rorosun_util else
              [util.attention(heads=8, kv_heads=2, dim=64, vdim=64, dims=64, ff=320), util.latent(heads=8, dim=64, rot_dim=64, vdim=64, q_rank=128, kv_rank=128, size=100)])
    cfg = util.config(layers=layers, vocab=512, width=256, **({} if util is rorosun_util else {"loop": (0, 1, 2)}))
    eng = MixerDecodeEngine(MixerModelConfig.from_dict(cfg), util.weights(cfg), dev, max_seq_len=600, dtype=torch.bfloat16, max_chunk=200)
    out += [eng.extend([t %% 512 for t in range(450)], range(0, 450, 7)), torch.cat([eng.extend([t], [0]) for t in range(5)])]
q = TurboQuantMSE(128, 3, dev)
x = torch.randn(5000, 128, generator=torch.Generator().manual_seed(1)).half().to(dev)
for _ in range(3):
    out.append(q.dequantize(q.quantize(x)))
torch.cuda.synchronize()
print("OUT", hashlib.sha256(b"".join(t.float().cpu().numpy().tobytes() for t in out)).hexdigest())
"""


def test_no_form_of_overlap_changes_a_result():
    """LEANKV_PDL: no launch before the one ahead has ended, every launch that may, those that gain by it. Kernels that hold tensor memory
    follow one another in all of them."""
    import os
    import subprocess
    import sys

    from conftest import ROOT

    code = _OVERLAP_SNIPPET % {"root": str(ROOT), "tests": os.path.join(str(ROOT), "tests")}
    outs = []
    for mode in "012":
        run = subprocess.run([sys.executable, "-c", code], env={**os.environ, "LEANKV_PDL": mode}, capture_output=True, text=True, timeout=300)
        assert run.returncode == 0, run.stderr[-2000:]
        outs.append(next(l for l in run.stdout.splitlines() if l.startswith("OUT")))
    assert len(set(outs)) == 1
