"""Kernels that a rule on sizes picks, at the sizes where each can go wrong, against the oracle.

Tolerances are those of the operators' own tests: the variants differ from one another in the order of fp32 sums only."""
import numpy as np
import pytest
import torch

from oracle import token_loop_oracle as O
from tests import test_engine_gpu as engine_tests
from tests.parity_cases import assert_close_bf16, decode_attention_case, prefill_attention_case, randn_bf16
from tests.test_engine_gpu import test_decode_with_norms_folded_into_the_gemms as folded_decode
from tests.test_moe_gpu import test_moe_forward_matches_oracle as moe_forward
from tests.test_ops_gpu import test_fused_add_rmsnorm as fused_add
from tests.test_saluzen_ops_gpu import DELTA, SSD, Recurrence, call, close  # noqa: F401  (call is a fixture)
from tests.test_saluzen_ops_gpu import BF16

pytestmark = pytest.mark.gpu
RTOL = 2 ** -7
NARROW, STREAM, TILE, PAIR = 1, 2, 3, 4   # what b200_gemm_kernel calls the kernels
BIG = (2e-3, 1e-3)   # absolute: sqrt(K / 1024) of the first, plus the second (as in test_linear_gpu.py)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(8, 64), (24, 64), (1000, 192), (520, 2048), (1024, 3072), (4096, 1024), (128, 5632), (3072, 2048), (2400, 1088)])
def test_linear_of_few_rows(L, pkg, M, N, K):
    """One and two tiles of tokens, features behind the last whole tile of 16, K within a register buffer and beyond two; two
    buffers with as many CTAs as SMs and with more."""
    assert pkg.load_library().b200_gemm_kernel(M, N, K, pkg.EPILOGUE_NONE, 0, 0, 0) == NARROW
    gen = torch.Generator().manual_seed(M + N + K)
    buf, w, b = randn_bf16(gen, M, K + 64), randn_bf16(gen, N, K, std=0.05), randn_bf16(gen, N)
    atol = BIG[0] * (K / 1024) ** 0.5 + BIG[1]
    x = buf[:, 64:]
    assert_close_bf16(L.linear(buf.cuda()[:, 64:], w.cuda(), b.cuda()), O.linear(x, w, b), 2 * atol, RTOL, "bias, strided rows")
    if N % 16 == 0:
        y = L.linear(x.contiguous().cuda(), w.cuda(), epilogue=pkg.EPILOGUE_SWIGLU)
        assert_close_bf16(y, O.silu_and_mul(O.linear(x, w)), 2 * atol, 3 * RTOL, "SwiGLU")
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("kind,nreq", [("qwen3", 12), ("llama", 9), ("qwen2", 16)])
def test_decode_of_two_token_tiles(pkg, monkeypatch, kind, nreq):
    folded_decode(pkg, monkeypatch, kind, nreq, "1")


def on_narrow(pkg, cfg, nreq):
    """Whether a decode step's projections that carry the norm run on the narrow kernel."""
    qkv = (cfg.num_qo_heads + 2 * cfg.num_kv_heads) * cfg.head_dim
    return pkg.load_library().b200_gemm_kernel(nreq, qkv, cfg.hidden_size, pkg.EPILOGUE_NONE, 0, 0, 1) == NARROW


@pytest.mark.parametrize("fold_heads", ["1", "0"])
@pytest.mark.parametrize("kind,nreq", [("qwen3", 20), ("llama", 24), ("qwen2", 17), ("llama", 33)])
def test_decode_on_split_projections_with_folded_norms(pkg, monkeypatch, kind, nreq, fold_heads):
    """More requests than the narrow kernel takes: the split-K kernel's accumulator of 32 tokens and the one of 64."""
    assert not on_narrow(pkg, engine_tests.small_cfg(kind), nreq)
    folded_decode(pkg, monkeypatch, kind, nreq, fold_heads)


@pytest.mark.parametrize("fold_heads", ["1", "0"])
@pytest.mark.parametrize("hidden,nreq,narrow", [(2304, 1, False), (2304, 5, False), (2304, 16, False), (2048, 1, True), (1984, 2, True), (2048, 9, False)])
@pytest.mark.parametrize("qwen", [True, False])
def test_decode_of_a_wide_layer(pkg, monkeypatch, qwen, hidden, nreq, narrow, fold_heads):
    """A handful of requests of a model too wide for the narrow kernel's norm (split-K, accumulator of 32 tokens), and of the
    widest that it takes (two register buffers).  The bars are for logits below 2, where a bf16 step is at most 2^-7: weights are
    scaled by 1 / sqrt(hidden), and the output head is its own (against the table of the embedding, one layer further on, a
    token's own logit is about 5, and one step 2^-5)."""
    cfg = O.ModelConfig(1, hidden, 4, 2, 128, 512, 1024, 1e-6, 1e6, 512, False, qwen, qwen)
    assert on_narrow(pkg, cfg, nreq) == narrow
    init = O.init_weights
    monkeypatch.setattr(engine_tests, "small_cfg", lambda kind: cfg)
    monkeypatch.setattr(engine_tests.O, "init_weights", lambda c, seed, std: init(c, seed=seed, std=std * (256 / hidden) ** 0.5))
    folded_decode(pkg, monkeypatch, "wide", nreq, fold_heads)


@pytest.mark.parametrize("nreq", [1, 8, 9, 16])
@pytest.mark.parametrize("inter", [576, 2048, 2112, 4032, 4096, 4160])   # steps of 32 that do not fall evenly to the warps; one and
def test_decode_with_staged_weights(pkg, monkeypatch, inter, nreq):      # two buffers; the most that is requested ahead, and more
    """The down projection of a decode step, K = `inter`, keeps its weights in shared memory."""
    cfg = O.ModelConfig(1, 256, 4, 2, 128, inter, 1024, 1e-6, 1e6, 512, True, True, True)
    assert on_narrow(pkg, cfg, nreq)
    monkeypatch.setattr(engine_tests, "small_cfg", lambda kind: cfg)
    folded_decode(pkg, monkeypatch, "long", nreq, "1")


@pytest.mark.parametrize("nreq", [1, 9])
def test_values_that_are_not_finite_stay_where_they_are(pkg, nreq):
    """Values are not rotated: an infinite one must not reach the feature that a rotation would pair it with."""
    cfg = engine_tests.small_cfg("qwen2")
    pr = engine_tests.Pair(pkg, cfg, 16, max_running_req=max(nreq, 8))
    reqs = [pr.hb.add_request(np.arange(1, 6 + i, dtype=np.int32), 4) for i in range(nreq)]
    pr.hb.prefill(reqs).synchronize()
    at = (cfg.num_qo_heads + cfg.num_kv_heads + 2) * 128
    bias = pr.w["layers"][0]["qkv_bias"].clone()
    bias[at + 3], bias[at + 70] = float("inf"), float("-inf")
    pr.engine.load("qkv_bias", 0, bias)
    pr.hb.allocate(reqs)
    slots = [int(pr.hb.slots_of(r)[r.device_len - 1]) for r in reqs]
    pr.hb.decode(reqs).synchronize()
    pool = pr.engine.device_view("kv_cache").view(torch.bfloat16).view(2, cfg.num_layers, -1, cfg.num_kv_heads, 128).cpu()
    for slot in slots:
        v = pool[1, 0, slot].float()
        assert v[2, 3] == float("inf") and v[2, 70] == float("-inf") and int(torch.isfinite(v).logical_not().sum()) == 2
    pr.engine.close()


@pytest.mark.parametrize("nreq", [1, 8, 9, 16])
def test_experts_layer_of_two_register_buffers(pkg, nreq):
    """Decode steps of a Qwen3-MoE layer of hidden 2048: qkv with its head operations on the narrow kernel, without a norm.
    Every token takes all experts (of two almost equal ones either could be chosen otherwise); weights as above."""
    cfg = O.ModelConfig(1, 2048, 4, 2, 128, 512, 1024, 1e-6, 1e6, 512, False, True, True, "silu", 8, 8, 128, True)
    rng = np.random.default_rng(nreq)
    with pytest.MonkeyPatch.context() as mp:
        init = O.init_weights
        mp.setattr(engine_tests.O, "init_weights", lambda c, seed, std: init(c, seed=seed, std=std * (256 / 2048) ** 0.5))
        pr = engine_tests.Pair(pkg, cfg, 16, num_pages=nreq * 4 + 8, max_running_req=max(nreq, 8))
    reqs = [pr.hb.add_request(rng.integers(0, cfg.vocab_size, size=int(n)).astype(np.int32), 6) for n in rng.integers(3, 40, size=nreq)]
    pr.host_tokens = {r.table_idx: list(r.input_ids[:r.device_len]) + [0] * 16 for r in reqs}
    for step in range(3):
        pr.hb.allocate(reqs)
        ob, pt = pr.oracle_batch(reqs, step == 0)
        want = pr.oracle.forward(ob, pr.kv, pt)
        (pr.hb.decode if step else pr.hb.prefill)(reqs).synchronize()
        engine_tests.check_logits(pr.engine.logits(nreq), want, f"step {step}")
        tok = want.argmax(-1).tolist()
        for r, t in zip(reqs, tok):
            pr.host_tokens[r.table_idx][r.cached_len] = t
        pr.engine.write_token_pool([r.table_idx for r in reqs], [r.cached_len for r in reqs], tok)
    assert pr.engine_status_clean()
    pr.engine.close()


@pytest.mark.parametrize("seq_lens,page_size,hq,hkv", [([700], 16, 16, 8), ([33], 16, 16, 8), ([5000, 2], 16, 16, 8), ([3000], 1, 8, 1),
                                                       ([900] * 5, 64, 32, 4), ([256, 257], 16, 16, 8), ([257], 16, 16, 8), ([256, 1, 300], 16, 6, 2), ([64] * 14, 16, 14, 2)])
def test_decode_of_few_requests_with_many_partials(L, seq_lens, page_size, hq, hkv):
    got, want, _ = decode_attention_case(L, seq_lens, page_size, hq, hkv, seed=len(seq_lens))
    assert_close_bf16(got, want, 2e-2, 2e-2, "decode attention")
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("tile", [0, 64, 128, 192, 256])
@pytest.mark.parametrize("M,N,K", [(257, 72, 64), (300, 1000, 192), (129, 520, 640), (1025, 384, 1024), (2600, 2064, 128)])
def test_tiles_of_every_width(L, pkg, monkeypatch, tile, M, N, K):
    """Rows behind a tile's first and second half, features behind its last, K from one block to more than the ring holds, and
    (2600 x 2064 with tiles of 64) more tiles than pairs of CTAs."""
    monkeypatch.setenv("B200_TILE_TN", str(tile))
    gen = torch.Generator().manual_seed(M + N)
    x, w, b = randn_bf16(gen, M, K), randn_bf16(gen, N, K, std=0.05), randn_bf16(gen, N)
    atol = BIG[0] * (K / 1024) ** 0.5 + BIG[1]
    assert_close_bf16(L.linear(x.cuda(), w.cuda(), b.cuda()), O.linear(x, w, b), 2 * atol, RTOL, "bias")
    if N % 16 == 0:
        y = L.linear(x.cuda(), w.cuda(), epilogue=pkg.EPILOGUE_SWIGLU)
        assert_close_bf16(y, O.silu_and_mul(O.linear(x, w)), 2 * atol, 3 * RTOL, "SwiGLU")
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("tile", [64, 128, 192, 256])
@pytest.mark.parametrize("K", [64, 384, 832])
def test_pairs_of_ctas_one_after_another(L, monkeypatch, tile, K):
    """Launches that follow each other at once, with fewer k-blocks than the ring has stages, and more: a CTA of the next launch
    takes the shared memory of one that has ended, which nothing may still be writing to."""
    monkeypatch.setenv("B200_TILE_TN", str(tile))
    gen = torch.Generator().manual_seed(K)
    x, w = randn_bf16(gen, 700, K), randn_bf16(gen, 3, 1032, K, std=0.05)
    xs, ws = x.cuda(), w.cuda()
    ys = [L.linear(xs, ws[i % 3]) for i in range(60)]
    for i in range(3):
        assert_close_bf16(ys[i], O.linear(x, w[i]), BIG[0] * (K / 1024) ** 0.5 + BIG[1], RTOL, "first")
        assert all(torch.equal(ys[i], y) for y in ys[i::3])
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("M,N,K,gated", [(65, 6144, 1024, True), (100, 12288, 1024, False), (181, 6144, 1024, True), (256, 4096, 1024, False)])
def test_batches_that_either_kernel_takes(L, pkg, monkeypatch, M, N, K, gated):
    """On tiles by the rule, and on slabs when the environment says so: each against the oracle, and against one another."""
    lib = pkg.load_library()
    gen = torch.Generator().manual_seed(M)
    x, w = randn_bf16(gen, M, K), randn_bf16(gen, N, K, std=0.05)
    xs, ws = x.cuda(), w.cuda()
    epilogue = pkg.EPILOGUE_SWIGLU if gated else pkg.EPILOGUE_NONE
    want = O.silu_and_mul(O.linear(x, w)) if gated else O.linear(x, w)
    atol, rtol = (2 * sum(BIG), 3 * RTOL) if gated else (sum(BIG), RTOL)   # (K is 1024)
    assert lib.b200_gemm_kernel(M, N, K, epilogue, 0, 0, 0) in (TILE, PAIR)
    y = L.linear(xs, ws, epilogue=epilogue)
    assert_close_bf16(y, want, atol, rtol, "tiles")
    monkeypatch.setenv("B200_GEMM_TILE_MIN_M", "1000000")
    assert lib.b200_gemm_kernel(M, N, K, epilogue, 0, 0, 0) == STREAM
    slabs = L.linear(xs, ws, epilogue=epilogue)
    assert_close_bf16(slabs, want, atol, rtol, "slabs")
    assert_close_bf16(y, slabs, 4e-3, 3 * RTOL, "tiles against slabs")


def expert_kernel(pkg, T, E, k, H, I):
    return pkg.load_library().b200_gemm_kernel(T * k, 2 * I, H, pkg.EPILOGUE_SWIGLU, E, T, 0)


@pytest.mark.parametrize("T,E,k,H,I,kernel", [(380, 4, 2, 128, 192, PAIR), (570, 3, 1, 1088, 1024, PAIR), (1520, 32, 4, 1024, 1024, PAIR),
                                              (2048, 6, 2, 640, 384, PAIR), (450, 3, 1, 128, 192, TILE), (1030, 8, 1, 128, 192, TILE)])
def test_experts_of_one_pair_tile(L, pkg, T, E, k, H, I, kernel):
    """151 to 222 rows per expert on average, or 640 and more, run on pairs of CTAs: K of two blocks and of more than the ring's
    six stages, tiles for two turns of every pair and more, one and several blocks of tokens per expert; other averages on
    single CTAs."""
    assert expert_kernel(pkg, T, E, k, H, I) == kernel
    moe_forward(L, T, E, k, H, I, True, "silu")


def test_experts_on_pair_tiles_that_tokens_do_not_choose_alike(L, pkg):
    """Experts with no row, a few, less than a block of 256, and several blocks, beside one another."""
    T, E, k, H, I = 1500, 24, 3, 576, 320
    assert expert_kernel(pkg, T, E, k, H, I) == PAIR
    gen = torch.Generator().manual_seed(24)
    liking = torch.linspace(-3, 3, E)[torch.randperm(E, generator=gen)]
    liking[::5] = -1e9
    gumbel = -torch.log(-torch.log(torch.rand(T, E, generator=gen).clamp(1e-6, 1 - 1e-6)))
    rank = (liking + gumbel).argsort(-1).argsort(-1)
    logits = ((rank.float() - E / 2) / 4).to(torch.bfloat16)      # (distinct in a row: no ties)
    rows = torch.bincount(rank.topk(k, -1).indices.flatten(), minlength=E)
    assert (rows == 0).any() and (rows > 512).any() and ((rows > 0) & (rows < 128)).any() and ((rows > 128) & (rows < 256)).any()
    hidden, gu, dn = randn_bf16(gen, T, H), randn_bf16(gen, E, 2 * I, H, std=H ** -0.5), randn_bf16(gen, E, H, I, std=I ** -0.5)
    moe = L.MoELayer(E, k, H, I, True, "silu")
    moe.gate_up_proj.copy_(gu.cuda())
    moe.down_proj.copy_(dn.cuda())
    want = O.moe_forward(hidden, logits, gu, dn, k, True, "silu", O.store_bf16)
    assert_close_bf16(moe.forward(hidden.cuda(), logits.cuda()), want, 2e-2, 4 * 2 ** -7, "skewed")
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("T,E,k,H,I,act", [(32, 16, 4, 2048, 1024, "silu"), (1, 64, 4, 1088, 64, "silu"), (9, 3, 1, 64, 192, "gelu"),
                                           (24, 16, 4, 1024, 2048, "silu")])
def test_experts_of_a_handful_of_rows(L, T, E, k, H, I, act):
    """At most 8 rows per expert on average, some with more and some with none; K of one and of two register buffers."""
    moe_forward(L, T, E, k, H, I, True, act)


@pytest.mark.parametrize("rows", [1023, 1024, 1027])
@pytest.mark.parametrize("hidden", [512, 768, 1024, 1536, 2048, 2560])
def test_norms_of_many_rows(L, rows, hidden):
    fused_add(L, rows, hidden)
    gen = torch.Generator().manual_seed(hidden)
    norm, x = L.RMSNorm(hidden, 1e-6), randn_bf16(gen, rows, hidden)
    norm.weight = randn_bf16(gen, hidden).cuda()
    assert_close_bf16(norm.forward(x.cuda()), O.rmsnorm(x, norm.weight.cpu(), 1e-6), 1e-6, RTOL, "norm")


@pytest.mark.parametrize("tokens,hq,hkv,qk_norm", [(4700, 5, 1, True), (1025, 16, 8, False), (2341, 6, 4, True), (900, 64, 8, True),
                                                     (500, 40, 40, False)])
def test_head_pass_of_many_tokens(L, tokens, hq, hkv, qk_norm):
    """Rows per token that are not a multiple of the four a warp takes at a time, keys beginning inside such a group: the same
    bits as in pieces that are few enough rows for the other kernel (which has its own test against the oracle)."""
    gen = torch.Generator().manual_seed(tokens)
    width = (hq + 2 * hkv) * 128
    qkv = randn_bf16(gen, tokens, width)
    pos = torch.randint(0, 2048, (tokens,), generator=gen, dtype=torch.int32).cuda()
    rot, qn, kn = L.RotaryEmbedding(128, 128, 2048, 1e6), None, None
    if qk_norm:
        qn, kn = L.RMSNorm(128, 1e-6), L.RMSNorm(128, 1e-6)
        qn.weight, kn.weight = randn_bf16(gen, 128).cuda(), randn_bf16(gen, 128).cuda()
    results = []
    for piece in (tokens, 499 if tokens * (hq + 2 * hkv) < 65536 else 300):
        cache = L.MHAKVCache(hkv, 1, 128, tokens // 16 + 2, 16)
        loc = torch.randperm(cache.total_slots, generator=torch.Generator().manual_seed(3))[:tokens].to(torch.int32).cuda()
        x = qkv.cuda()
        for t in range(0, tokens, piece):
            part = slice(t, min(t + piece, tokens))
            L.qknorm_rope_store(x[part], qn, kn, rot, pos[part], loc[part], cache, 0, hq, hkv, write_k_back=piece == tokens)
        results.append((x[:, :hq * 128].clone(), cache.k_cache(0).clone(), cache.v_cache(0).clone()))
        if piece == tokens:
            assert torch.equal(x[:, hq * 128:(hq + hkv) * 128].view(tokens, hkv, 128), cache.k_cache(0)[loc.long()])
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("rule", [SSD, DELTA])
@pytest.mark.parametrize("heads", [4, 12, 20])
@pytest.mark.parametrize("dv", [64, 128])
@pytest.mark.parametrize("lens", [[192, 65], [128, 65], [129, 3]])
def test_recurrence_in_slices_of_every_width(call, rule, heads, dv, lens):  # noqa: F811
    """Two requests, whole chunks and parts; 4 to 20 heads are dealt in 16, 32 and 64 value columns per CTA, up to two chunks in 64."""
    r = Recurrence(rule, lens, heads, heads // 2, 128, dv, 4, BF16, 1)
    states = r.states(3)
    got = r.run(call, states, [0, 0], [2, 0])
    outs, last = r.want()
    close(got, torch.cat(outs), BF16)
    for i, row in enumerate([2, 0]):
        close(states[0][row, :, :128, :dv], last[i], BF16)


@pytest.mark.parametrize("seq_lens,extend_lens,page_size,hq,hkv", [([128], [128], 16, 16, 8), ([129, 257], [129, 257], 16, 16, 8),
                                                                   ([640], [130], 1, 16, 8), ([385, 900], [200, 900], 64, 32, 4)])
def test_prefill_at_the_edges_of_tiles(L, seq_lens, extend_lens, page_size, hq, hkv):
    """Last tiles that are whole, of one key, in a slot of the ring that was in use and in one that was not."""
    got, want = prefill_attention_case(L, seq_lens, extend_lens, page_size, hq, hkv, seed=sum(seq_lens))
    assert_close_bf16(got, want, 2e-2, 2e-2, "prefill attention")
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("M", [1, 5, 8, 9, 13, 16])
@pytest.mark.parametrize("N,K", [(6664, 2112), (3336, 4160), (1000, 14336), (28672, 512)])
def test_linear_of_few_rows_of_a_large_w(L, pkg, M, N, K):
    """The ring kernel (the last shape: its neighbours): a last tile of 8 features, K that ends inside a stage of 512, fewer tiles than
    SMs, one and two blocks of tokens."""
    lib = pkg.load_library()
    assert lib.b200_gemm_kernel(M, N, K, pkg.EPILOGUE_NONE, 0, 0, 0) == (STREAM if K > 2048 or M > 8 else NARROW)
    gen = torch.Generator().manual_seed(M + N + K)
    buf, w, b = randn_bf16(gen, M, K + 64), randn_bf16(gen, N, K, std=0.05), randn_bf16(gen, N)
    atol = BIG[0] * (K / 1024) ** 0.5 + BIG[1]
    x = buf[:, 64:]
    assert_close_bf16(L.linear(buf.cuda()[:, 64:], w.cuda(), b.cuda()), O.linear(x, w, b), 2 * atol, RTOL, "bias, strided rows")
    if N % 16 == 0:
        y = L.linear(x.contiguous().cuda(), w.cuda(), epilogue=pkg.EPILOGUE_SWIGLU)
        assert_close_bf16(y, O.silu_and_mul(O.linear(x, w)), 2 * atol, 3 * RTOL, "SwiGLU")
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("T", [1, 8, 9, 17, 40])
@pytest.mark.parametrize("E,k,H,I", [(33, 4, 192, 576), (64, 3, 576, 64), (256, 1, 64, 128)])
@pytest.mark.parametrize("alike", [False, True])
def test_many_experts_of_few_rows(L, pkg, T, E, k, H, I, alike):
    """The ring kernel's experts: rows of an expert below, at and above the 8 and 16 of one pass, K within a stage and beyond."""
    lib = pkg.load_library()
    assert lib.b200_gemm_kernel(T * k, 2 * I, H, pkg.EPILOGUE_SWIGLU, E, T, 0) == NARROW
    gen = torch.Generator().manual_seed(T + E + H)
    hidden = randn_bf16(gen, T, H)
    logits = torch.randn(T, E, generator=gen).argsort(1).to(torch.bfloat16) / 32   # distinct in every row
    if alike:
        logits[:] = logits[0]
    moe = L.MoELayer(E, k, H, I, True, "silu")
    gu, dn = randn_bf16(gen, E, 2 * I, H, std=H ** -0.5), randn_bf16(gen, E, H, I, std=I ** -0.5)
    moe.gate_up_proj.copy_(gu.cuda())
    moe.down_proj.copy_(dn.cuda())
    assert_close_bf16(moe.forward(hidden.cuda(), logits.cuda()), O.moe_forward(hidden, logits, gu, dn, k, True, "silu", O.store_bf16),
                      2e-2, 4 * 2 ** -7, "experts")
    assert L.read_device_status() == (0, 0)


@pytest.mark.parametrize("M", [1, 5, 8, 9, 13, 16])
@pytest.mark.parametrize("N,K", [(6664, 2112), (3336, 4160), (1000, 14336), (28672, 512)])
def test_few_rows_of_a_large_w_are_the_ring_kernels(pkg, M, N, K):
    """What test_linear_of_few_rows_of_a_large_w runs on (the last shape: on its neighbours)."""
    assert pkg.load_library().b200_gemm_by_ring(M, N, K, pkg.EPILOGUE_NONE, 0, 0) == (K >= 2048)


@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("E,k,H,I,up,down", [(33, 3, 1600, 64, 99, 0), (32, 2, 64, 1600, 0, 96), (128, 2, 64, 512, 32, 0), (128, 2, 1024, 64, 0, 32)])
@pytest.mark.parametrize("alike", [False, True])
def test_experts_of_the_ring_kernel(L, pkg, T, E, k, H, I, up, down, alike):
    """Rows of an expert below, at and above the 8 and 16 of one pass, K of a part of a stage, of whole ones and of three and a part; up to
    `up` and `down` rows that projection is the ring kernel's."""
    lib = pkg.load_library()
    assert lib.b200_gemm_by_ring(T * k, 2 * I, H, pkg.EPILOGUE_SWIGLU, E, T) == (T * k <= up)
    assert lib.b200_gemm_by_ring(T * k, H, I, pkg.EPILOGUE_NONE, E, T) == (T * k <= down)
    test_many_experts_of_few_rows(L, pkg, T, E, k, H, I, alike)


def test_many_experts_on_the_narrow_kernel(L, pkg):
    """A K that is too short for the ring kernel, at most 8 rows per expert on average."""
    T, E, k, H, I = 64, 32, 2, 1088, 64
    lib = pkg.load_library()
    assert lib.b200_gemm_kernel(T * k, 2 * I, H, pkg.EPILOGUE_SWIGLU, E, T, 0) == NARROW
    assert not lib.b200_gemm_by_ring(T * k, 2 * I, H, pkg.EPILOGUE_SWIGLU, E, T)
    moe_forward(L, T, E, k, H, I, True, "silu")
