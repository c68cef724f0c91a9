"""Which kernel a projection runs on: shapes on either side of each rule's line, where both kernels were timed."""
import pytest

NARROW, STREAM, TILE, PAIR = 1, 2, 3, 4
PLAIN, SWIGLU = 0, 1


def experts(lib, tokens, experts, per_token, hidden, inter):
    """The kernels of an expert layer's two projections."""
    return (lib.b200_gemm_kernel(tokens * per_token, 2 * inter, hidden, SWIGLU, experts, tokens, 0),
            lib.b200_gemm_kernel(tokens * per_token, hidden, inter, PLAIN, experts, tokens, 0))


@pytest.mark.parametrize("shape,hidden,inter,narrow,not_narrow", [
    ((64, 4), 2048, 1024, (1, 8, 16, 32, 48), (64, 96, 128)),
    ((128, 8), 2048, 768, (1, 8), (24, 32, 64, 128)),
    ((32, 2), 2048, 1024, (8, 32, 64), (128,)),
    ((16, 4), 1024, 2048, (1, 8, 16, 32), (33, 64)),
    ((8, 2), 1024, 1024, (4, 16, 32), (33,)),
])
def test_experts_whose_tokens_may_all_choose_alike(pkg, shape, hidden, inter, narrow, not_narrow):
    """A CTA of the narrow kernel takes an expert's rows 8 at a time: it is left as soon as a batch in which every token chooses
    the same experts would be slower on it."""
    lib = pkg.load_library()
    for tokens in narrow:
        assert experts(lib, tokens, *shape, hidden, inter) == (NARROW, NARROW), tokens
    for tokens in not_narrow:
        assert NARROW not in experts(lib, tokens, *shape, hidden, inter), tokens


@pytest.mark.parametrize("hidden,narrow,not_narrow", [(768, (1, 8, 9, 16), (17,)), (1024, (1, 8, 9, 16), (17,)),
                                                      (1280, (1, 2), (3, 8, 9, 16)), (2048, (1, 2), (4, 8, 9, 16)), (2304, (), (1, 2, 16))])
def test_projections_that_carry_the_norm(pkg, hidden, narrow, not_narrow):
    lib = pkg.load_library()
    for rows, kernel in [(r, NARROW) for r in narrow] + [(r, STREAM) for r in not_narrow]:
        for N, epilogue in ((2 * hidden, PLAIN), (4 * hidden, SWIGLU)):
            assert lib.b200_gemm_kernel(rows, N, hidden, epilogue, 0, 0, 1) == kernel, (rows, N)
    assert [lib.b200_gemm_kernel(rows, 16384, 1024, SWIGLU, 0, 0, 1) for rows in (4, 5, 8)] == [NARROW, STREAM, STREAM]


@pytest.mark.parametrize("N,K,epilogue,narrow,not_narrow", [
    (4096, 1024, PLAIN, (1, 8, 9, 16), (17,)), (151936, 1024, PLAIN, (1, 8), (9,)), (12288, 1024, SWIGLU, (1, 8, 16), (17,)),
    (2048, 64, PLAIN, (1, 8, 16), ()), (151936, 64, PLAIN, (), (1, 8, 16)), (151936, 256, PLAIN, (), (1, 8)), (151936, 512, PLAIN, (1, 8), ()),
    (16384, 1088, SWIGLU, (1, 8), (9,)), (32768, 1088, PLAIN, (), (1, 8)), (32768, 1536, PLAIN, (), (1, 8)), (32768, 2048, PLAIN, (1, 4), (6, 8)),
    (6144, 1536, SWIGLU, (9, 16), ()), (8192, 1536, PLAIN, (8,), (9, 16)), (8192, 1536, SWIGLU, (8,), (9, 16)), (12288, 1088, SWIGLU, (8,), (9,)),
    (2048, 6144, PLAIN, (1, 16), ()), (4096, 3072, PLAIN, (8, 9, 16), ()), (3584, 3584, SWIGLU, (8,), (9, 16)), (4096, 4096, PLAIN, (), (1, 8, 16)),
])
def test_projections_of_a_handful_of_rows(pkg, N, K, epilogue, narrow, not_narrow):
    lib = pkg.load_library()
    for rows in narrow:
        assert lib.b200_gemm_kernel(rows, N, K, epilogue, 0, 0, 0) == NARROW, rows
    for rows in not_narrow:
        assert lib.b200_gemm_kernel(rows, N, K, epilogue, 0, 0, 0) == STREAM, rows


@pytest.mark.parametrize("N,K,epilogue,ring,not_ring", [
    (4096, 1024, PLAIN, (), (1, 8, 16)), (151936, 1024, PLAIN, (), (1, 8, 16)), (4096, 2048, PLAIN, (), (1, 8)), (6144, 2048, PLAIN, (1, 8, 16), (17,)),
    (2048, 6144, PLAIN, (1, 8, 9, 16), (17,)), (32768, 2048, PLAIN, (1, 4, 8, 16), ()), (4096, 4096, PLAIN, (1, 8, 16), (17,)),
    (28672, 4096, SWIGLU, (1, 16), (17,)), (1024, 16384, PLAIN, (1, 16), ()), (512, 32768, PLAIN, (1, 16), ()), (512, 4096, PLAIN, (), (1, 8)),
])
def test_projections_by_the_ring_kernel(pkg, N, K, epilogue, ring, not_ring):
    """What runs there is told apart from the kernel whose place it takes."""
    lib = pkg.load_library()
    assert [lib.b200_gemm_by_ring(r, N, K, epilogue, 0, 0) for r in ring + not_ring] == [1] * len(ring) + [0] * len(not_ring)
    assert all(lib.b200_gemm_kernel(r, N, K, epilogue, 0, 0, 0) in (NARROW, STREAM) for r in ring)


@pytest.mark.parametrize("N,K", [(3072, 4096), (3328, 3840), (3584, 3584), (3840, 3328), (4096, 3264), (4608, 2752)])
def test_tiles_that_go_round_the_ring_kernels_ctas_unevenly(pkg, N, K):
    """Up to 8 rows the kernel from memory to registers is the faster one (with 9 rows it is not)."""
    lib = pkg.load_library()
    assert [lib.b200_gemm_by_ring(r, N, K, PLAIN, 0, 0) for r in (1, 8, 9, 16)] == [0, 0, 1, 1]


def test_shapes_that_the_ring_kernel_does_not_take(pkg):
    lib = pkg.load_library()
    assert [lib.b200_gemm_by_ring(*a) for a in [(0, 4096, 4096, 0, 0, 0), (4, 4096, 4000, 0, 0, 0), (4, 4096, 4096, 99, 0, 0), (4, 4096, 4096, 0, 2, 0)]] == [0] * 4


@pytest.mark.parametrize("experts,per_token,N,K,epilogue,ring,not_ring", [
    (64, 4, 2048, 2048, SWIGLU, (1, 8, 32, 48), (49, 64)), (32, 4, 2048, 2048, SWIGLU, (1, 8, 32), (33, 48)), (32, 4, 1024, 1536, SWIGLU, (1, 24), (25, 32)),
    (64, 4, 1024, 2048, PLAIN, (1, 32, 48), (49,)), (31, 2, 2048, 2048, SWIGLU, (), (1, 32)), (128, 8, 1536, 2048, SWIGLU, (1, 8, 16), (64,)),
    # short K: many tiles of two stages; else only a launch of CTAs for groups without rows is behind
    (32, 4, 2048, 256, PLAIN, (), (1, 8, 32)), (64, 4, 2048, 1024, PLAIN, (1, 8, 32, 48), (49,)), (32, 4, 2048, 1024, PLAIN, (), (1, 8, 32)), (64, 4, 2032, 1024, PLAIN, (1, 4), (5, 32)),
    (64, 6, 1024, 512, SWIGLU, (1, 2), (3, 8, 32)),
    (64, 8, 1024, 1024, SWIGLU, (1, 2), (3, 24, 48)), (128, 4, 2048, 256, PLAIN, (1, 8), (9, 16)), (128, 4, 512, 1024, PLAIN, (), (1, 4, 32)), (256, 8, 256, 128, SWIGLU, (), (1, 8)),
])
def test_experts_by_the_ring_kernel(pkg, experts, per_token, N, K, epilogue, ring, not_ring):
    lib = pkg.load_library()
    for tokens, want in [(t, 1) for t in ring] + [(t, 0) for t in not_ring]:
        assert lib.b200_gemm_by_ring(tokens * per_token, N, K, epilogue, experts, tokens) == want, tokens


@pytest.mark.parametrize("M,N,K,epilogue,kernel", [
    (64, 6144, 1024, SWIGLU, STREAM), (65, 6144, 1024, SWIGLU, PAIR), (65, 3072, 640, PLAIN, STREAM), (128, 2048, 1024, PLAIN, STREAM),
    (65, 12288, 1024, PLAIN, PAIR), (129, 2048, 1024, PLAIN, PAIR), (129, 1024, 1024, PLAIN, STREAM), (256, 1024, 1024, PLAIN, PAIR),
    (256, 4096, 1024, PLAIN, PAIR), (256, 1024, 2048, PLAIN, STREAM), (257, 1024, 2048, PLAIN, PAIR), (600, 6144, 4096, PLAIN, TILE),
])
def test_batches_between_decoding_and_prompts(pkg, monkeypatch, M, N, K, epilogue, kernel):
    lib = pkg.load_library()
    assert lib.b200_gemm_kernel(M, N, K, epilogue, 0, 0, 0) == kernel
    monkeypatch.setenv("B200_GEMM_TILE_MIN_M", "257")   # one line, and nothing below it
    assert lib.b200_gemm_kernel(M, N, K, epilogue, 0, 0, 0) == (STREAM if M < 257 else kernel)


@pytest.mark.parametrize("M,N,K,kernel", [(300, 128, 512, TILE), (8000, 128, 640, TILE), (8000, 4096, 512, TILE), (8000, 4096, 640, TILE), (3000, 520, 640, TILE),
                                          (300, 1024, 640, PAIR), (1000, 1024, 768, PAIR), (8192, 4096, 1024, PAIR), (257, 64, 4096, PAIR)])
def test_tiles_of_a_short_k(pkg, M, N, K, kernel):
    assert pkg.load_library().b200_gemm_kernel(M, N, K, PLAIN, 0, 0, 0) == kernel


@pytest.mark.parametrize("rows,kernel", [(127, STREAM), (130, TILE), (150, TILE), (151, PAIR), (222, PAIR), (223, TILE), (300, TILE), (560, TILE), (630, TILE), (680, PAIR), (1000, PAIR), (1100, TILE), (1200, PAIR)])
def test_expert_tiles(pkg, rows, kernel):
    assert pkg.load_library().b200_gemm_kernel(rows * 16, 2048, 2048, SWIGLU, 16, rows * 16, 0) == kernel


def test_shapes_that_no_kernel_takes(pkg):
    lib = pkg.load_library()
    assert [lib.b200_gemm_kernel(*a) for a in [(0, 64, 64, 0, 0, 0, 0), (4, 64, 96, 0, 0, 0, 0), (4, 64, 64, 99, 0, 0, 0), (4, 64, 64, 0, 2, 0, 0)]] == [0] * 4


@pytest.mark.parametrize("q_heads,kv_heads,norms,by_tokens,by_rows", [
    (128, 8, 1, (900, 3000), (228, 342, 650, 740)), (40, 40, 1, (900,), (274, 411)), (64, 8, 1, (900, 1100), (410, 592)), (32, 8, 1, (900, 1024), (683, 740)),
    (16, 8, 1, (1024, 8192), (1023,)), (64, 8, 0, (500, 1500), (410, 450)), (40, 40, 0, (500,), (274,)), (128, 8, 0, (500,), (228, 342)), (32, 8, 0, (683,), (682,)),
])
def test_head_pass_of_few_tokens_with_many_heads(pkg, q_heads, kv_heads, norms, by_tokens, by_rows):
    """A warp per token only where that was the faster way to deal the rows."""
    lib = pkg.load_library()
    assert [lib.b200_head_pass_by_tokens(t, q_heads, kv_heads, 128, norms) for t in by_tokens + by_rows] == [1] * len(by_tokens) + [0] * len(by_rows)
    assert lib.b200_head_pass_by_tokens(8192, q_heads, kv_heads, 64, norms) == 0
