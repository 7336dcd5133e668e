"""Products of 17 to 256 tokens in equal shares of weight rows, and on CTA pairs from 129 (csrc/gemm_pair.cu): rows that no share
divides, one wave and two, one and two k-blocks to a barrier, token counts around the 32-token unit and the limits of the rules, every
epilogue, and nothing written outside Y."""
import ctypes as C

import pytest
import torch

from tests.test_pair_gemm_gpu import GEGLU, PLAIN, PLAIN_F32, RELU2, SWIGLU, test_pair_products as check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from vllm_tgis_adapter_b200.engine._lib import load_library

    return load_library()


@pytest.mark.parametrize("mode", [PLAIN, PLAIN_F32, SWIGLU, GEGLU, RELU2])
@pytest.mark.parametrize("T,N,K", [(17, 5920, 64), (32, 6144, 128), (33, 10256, 192), (48, 8192, 320), (49, 6002, 2112), (64, 18944, 256), (65, 592, 64),
                                   (96, 1184, 320), (100, 19000, 128), (128, 4096, 4096), (129, 18946, 192), (130, 520, 512), (200, 40000, 64),
                                   (255, 8190, 320), (256, 37890, 128), (256, 2048, 1088)])
def test_products(lib, T, N, K, mode):
    check(lib, T, N, K, mode)


def p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("T,n_q,n_kv,K", [(17, 48, 8, 576), (32, 48, 8, 768), (100, 32, 8, 512), (160, 32, 8, 512), (256, 32, 8, 512)])
def test_no_rotary_embedding_inside_these_products(lib, T, n_q, n_kv, K):
    """They have no fused form, and where they are taken the entry with one says so instead of taking another kernel: a row has the same
    bits with and without.  (The two launches are tested one by one.)"""
    N = (n_q + 2 * n_kv) * 128
    assert lib.tgis_k_gemm_route(T, N, K, 148, 0) in (1, 2)
    x, w, y = torch.zeros(256, K, device="cuda").bfloat16(), torch.zeros(N, K, device="cuda").bfloat16(), torch.full((256, N), 3.0, device="cuda").bfloat16()
    cs, cache = torch.zeros(64, 128, device="cuda").bfloat16(), torch.full((T + 32, n_kv * 128), 3.0, device="cuda").bfloat16()
    pos, slots = (C.c_int32 * T)(), (C.c_int32 * T)(*range(T))
    assert lib.tgis_k_gemm_rope(p(x), p(w), p(y), T, n_q, n_kv, K, 256, pos, slots, p(cs), p(cache), p(cache)) == 1
    assert bool((y == 3.0).all()) and bool((cache == 3.0).all())


@pytest.mark.parametrize("T", [257, 300, 1030])
@pytest.mark.parametrize("batch,N,K,mode,y_dt", [(16, 512, 128, 0, 0), (5, 128, 512, 2, 1), (3, 40, 64, 0, 1), (1, 65, 2048, 0, 0), (1, 64, 320, 4, 1), (2, 300, 192, 2, 1)])
def test_prompts_side_by_side_and_with_few_weight_rows(lib, T, batch, N, K, mode, y_dt):
    """Products of more than 256 tokens that only the general entry takes: one per head in neighbouring columns, a router's few rows,
    a tanh, a scale per row and head; columns between the problems and rows behind the last token stay as they are."""
    gen = torch.Generator(device="cuda").manual_seed(T + N + K)
    xs, ys = K + 8, N + 3
    x = torch.randn(T, batch, xs, device="cuda", generator=gen).bfloat16()
    w = (torch.randn(batch, N, K, device="cuda", generator=gen) * K ** -0.5).bfloat16()
    s = torch.rand(T, batch, device="cuda", generator=gen)
    y = torch.full((T + 1, batch, ys), 7.0, device="cuda", dtype=torch.bfloat16 if y_dt else torch.float32)
    rc = lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, y_dt, T, N, K, batch * xs, K, batch * ys, batch, xs, N * K, ys, None, 0, 0, None, 1, mode, p(s), batch)
    assert rc == 0
    a, b = x[:, :, :K].double(), w.double()
    want = torch.einsum("thk,hnk->thn", a, b)
    slack = torch.einsum("thk,hnk->thn", a.abs(), b.abs()) * (K / 16 + 8) * 2.0 ** -23   # as in the products above
    if mode == 2:
        want, slack = want * s.double()[:, :, None], slack * s.double()[:, :, None]
    if mode == 4:
        want, slack = torch.tanh(want), slack + 1e-6
    got = y[:T, :, :N].double()
    assert ((got - want).abs() <= slack + (2.0 ** -8 * want.abs() if y_dt else 1e-6 * want.abs())).all()
    assert bool((y[:T, :, N:] == 7.0).all()) and bool((y[T] == 7.0).all())


@pytest.mark.parametrize("N,K", [(40, 64), (300, 192)])
def test_expert_rows_with_a_scale_ahead_of_the_squared_relu(lib, N, K):
    """Segments around the 32 tokens that a warp of the epilogue takes at once, each gathered row with the scale of its origin."""
    gen = torch.Generator(device="cuda").manual_seed(N)
    lens = [0, 1, 31, 32, 33, 65, 257, 301]
    R, E = sum(lens), len(lens)
    x = torch.randn(R, K, device="cuda", generator=gen).bfloat16()
    w = (torch.randn(E, N, K, device="cuda", generator=gen) * K ** -0.5).bfloat16()
    s = torch.randn(R, device="cuda", generator=gen)
    order = torch.randperm(R, device="cuda", generator=gen).int()
    seg = torch.tensor([0] + lens, device="cuda").cumsum(0).int()
    y = torch.full((R + 1, N), 7.0, device="cuda", dtype=torch.bfloat16)
    assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, 1, R, N, K, K, K, N, 1, 0, 0, 0, p(seg), E, N * K, p(order), 1, 5, p(s), 0) == 0
    e = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(lens, device="cuda"))
    o = order.long()
    a = torch.einsum("rk,rnk->rn", x[o].double(), w[e].double()) * s[o].double()[:, None]
    slack = torch.einsum("rk,rnk->rn", x[o].double().abs(), w[e].double().abs()) * s[o].double().abs()[:, None] * (K / 16 + 8) * 2.0 ** -23
    want = a.clamp(min=0) ** 2
    assert ((y[:R].double() - want).abs() <= 2.0 ** -8 * want + 2 * a.abs() * slack + slack ** 2 + 1e-6 * want).all()
    assert bool((y[R] == 7.0).all())


@pytest.mark.parametrize("N,K", [(6144, 4096), (28672, 2304), (768, 768), (2048, 2048), (9728, 512)])
@pytest.mark.parametrize("tokens", [(33, 40, 48, 49, 64), (65, 66, 96, 128), (129, 200, 256)])
def test_a_row_changes_its_bits_only_where_the_token_tiles_change(lib, N, K, tokens):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    x = torch.randn(256, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    rows = []
    for T in tokens:
        y, ms = torch.empty(T, N, device="cuda", dtype=torch.float32), C.c_float()
        assert lib.tgis_k_gemm(p(x), p(w), p(y), T, N, K, 256, 0, 1, C.byref(ms), PLAIN_F32) == 0
        rows.append(y)
    assert all(torch.equal(r[: tokens[0]], rows[0]) for r in rows)


@pytest.mark.parametrize("N,K,dt,tokens", [(64, 2048, 1, (1, 32, 33, 64, 65, 128, 129, 256)), (127, 512, 1, (64, 65, 256)), (96, 1024, 0, (1, 8, 64)), (96, 1024, 0, (65, 86, 128))])
def test_a_row_of_a_tanh_map_has_the_same_bits_beside_many_others(lib, N, K, dt, tokens):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    to = torch.bfloat16 if dt else torch.float32
    x, w = torch.randn(256, K, generator=gen, device="cuda").to(to), (torch.randn(N, K, generator=gen, device="cuda") * K ** -0.5).to(to)
    rows = []
    for T in tokens:
        y = torch.empty(T, N, device="cuda")
        assert lib.tgis_k_gemm_any(p(x), p(w), p(y), dt, dt, 0, T, N, K, K, K, N, 1, 0, 0, 0, None, 0, 0, None, 1, 4, None, 0) == 0
        rows.append(y)
    assert all(torch.equal(r[: tokens[0]], rows[0]) for r in rows)
    want = torch.tanh(x[: len(y)].double() @ w.double().T)
    assert float((y.double() - want).abs().max()) <= K / 8 * 2.0 ** -24 * float((x.double().abs() @ w.double().abs().T).max()) + 1e-6
