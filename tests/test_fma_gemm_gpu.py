"""General products on the FMA pipe (csrc/gemm_any.cu): row counts around the 16, 32 and 64 row tiles, widths around the 64
column tile, k around the block of 32 and off the four-element loads, both operand mixes, expert segments and epilogues,
against 64-bit torch."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from vllm_tgis_adapter_b200.engine._lib import load_library

    return load_library()


def p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def bound(x, w, K):
    # a sum of K products, each added with one rounding of a partial sum that the sum of magnitudes bounds (two halves of K / 2)
    return (x.double().abs() @ w.double().abs().T) * (K / 2 + 2) * 2.0 ** -24


@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,N,K,ld", [(1, 64, 32, 32), (16, 63, 33, 33), (21, 65, 36, 40), (37, 128, 31, 32), (64, 192, 64, 64), (65, 1, 4, 4),
                                      (700, 3000, 96, 96), (300, 70, 1, 1)])
def test_dense(lib, T, N, K, ld, wdt):
    gen = torch.Generator(device="cuda").manual_seed(T + N + K)
    x = torch.randn(T, ld, generator=gen, device="cuda")
    w = torch.randn(N, ld, generator=gen, device="cuda").to(wdt)
    y = torch.full((T + 1, N), 7.0, device="cuda")
    assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 0, int(wdt == torch.bfloat16), 0, T, N, K, ld, ld, N, 1, 0, 0, 0, None, 0, 0, None, 1, 0, None, 0) == 0
    ref = x[:, :K].double() @ w[:, :K].double().T
    assert float(((y[:T].double() - ref).abs() - bound(x[:, :K], w[:, :K], K)).max()) <= 0
    assert bool((y[T] == 7.0).all())


@pytest.mark.parametrize("counts", [[1], [0, 17, 64, 0, 33], [3] * 40, [200, 0, 1]])
@pytest.mark.parametrize("mode,K", [(0, 48), (1, 50), (3, 64), (5, 37), (6, 128)])
def test_segments_and_epilogues(lib, counts, mode, K):
    gen = torch.Generator(device="cuda").manual_seed(K + len(counts))
    E, rows, N = len(counts), sum(counts), 130
    seg = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    x = torch.randn((rows + 1) // 2, K, generator=gen, device="cuda")
    w = torch.randn(E, N, K, generator=gen, device="cuda") * K ** -0.5
    order = torch.randperm(rows, generator=gen, device="cuda").int()
    scale = torch.rand(rows, generator=gen, device="cuda") + 0.5
    expert = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(counts, device="cuda"))
    src = order.long() // 2
    acc, eps = (torch.empty(rows, N, dtype=torch.float64, device="cuda") for _ in range(2))
    for e in range(E):
        r = expert == e
        acc[r], eps[r] = x[src[r]].double() @ w[e].double().T, bound(x[src[r]], w[e], K)
    if mode in (1, 3):
        g, u = acc[:, 0::2], acc[:, 1::2]
        ref = (torch.nn.functional.silu(g) if mode == 1 else torch.nn.functional.gelu(g, approximate="tanh")) * u
        tol = 1.13 * eps[:, 0::2] * u.abs() + g.abs() * eps[:, 1::2] + 2e-6 * g.abs() * u.abs()
    elif mode == 5:
        s = scale[order.long()].double()[:, None]
        ref = (acc * s).clamp(min=0) ** 2
        tol = (2 * (acc * s).abs() + eps * s) * eps * s + 3e-7 * ref
    else:
        ref = torch.nn.functional.gelu(acc) if mode == 6 else acc
        tol = 1.13 * eps + 2e-6 * acc.abs()
    y = torch.full((rows + 1, ref.shape[1]), 7.0, device="cuda")
    assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 0, 0, 0, rows, N, K, K, K, y.shape[1], 1, 0, 0, 0, p(seg), E, N * K, p(order), 2, mode,
                               p(scale) if mode == 5 else None, 0) == 0
    assert float(((y[:rows].double() - ref).abs() - tol).max()) <= 0
    assert bool((y[rows] == 7.0).all())


@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,N,K,ld", [(1537, 1089, 289, 289), (1600, 1152, 300, 300), (1601, 1100, 260, 264)])
def test_dense_tiles_of_64_rows(lib, T, N, K, ld, wdt):
    """Launches of three and more 64 x 64 tiles for every SM and more than 256 products per sum."""
    test_dense(lib, T, N, K, ld, wdt)


@pytest.mark.parametrize("mode,K", [(0, 257), (1, 288), (3, 300), (5, 260), (6, 292)])
def test_segments_and_epilogues_in_tiles_of_64_rows(lib, mode, K):
    test_segments_and_epilogues(lib, [1000, 0, 63, 64, 65, 1, 2107] * 5, mode, K)   # 3 column tiles, 35 segments of 470 rows on average


@pytest.mark.parametrize("K", [64, 100, 300, 301])   # one chain a sum; 16 and 32 rows only; all three heights, wide and single loads
def test_a_row_is_the_same_in_every_tile_height(lib, K):
    gen = torch.Generator(device="cuda").manual_seed(3)
    x, w = torch.randn(1600, K, generator=gen, device="cuda"), torch.randn(1100, K, generator=gen, device="cuda")

    def run(a):
        y = torch.empty(a.shape[0], 1100, device="cuda")
        assert lib.tgis_k_gemm_any(p(a), p(w), p(y), 0, 0, 0, a.shape[0], 1100, K, K, K, 1100, 1, 0, 0, 0, None, 0, 0, None, 1, 0, None, 0) == 0
        return y

    whole = run(x)   # 450 tiles of 64 rows where K > 256
    assert torch.equal(run(x[40:100].contiguous()), whole[40:100])   # 32
    assert torch.equal(run(x[90:99].contiguous()), whole[90:99])     # 16


def test_rows_beyond_the_tiles_of_32_that_one_launch_holds(lib):
    T, N, K = 65535 * 32 + 33, 3, 5
    gen = torch.Generator(device="cuda").manual_seed(4)
    x, w = torch.randn(T, K, generator=gen, device="cuda"), torch.randn(N, K, generator=gen, device="cuda")
    y = torch.full((T + 1, N), 7.0, device="cuda")
    assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 0, 0, 0, T, N, K, K, K, N, 1, 0, 0, 0, None, 0, 0, None, 1, 0, None, 0) == 0
    assert float(((y[:T].double() - x.double() @ w.double().T).abs() - bound(x, w, K)).max()) <= 0
    assert bool((y[T] == 7.0).all())
