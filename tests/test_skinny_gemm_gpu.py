"""Products of up to 32 tokens (csrc/gemm_skinny.cu) against 64-bit torch: token counts around the eight-token tiles, weight
rows around the CTA sizes and the lines between the variants, k from one chunk to more chunks than warps, every epilogue."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

PLAIN, PLAIN_F32, SWIGLU, GEGLU, RELU2 = 0, 1, 2, 3, 4   # tgis_k_gemm out modes


@pytest.fixture(scope="module")
def lib():
    from vllm_tgis_adapter_b200.engine._lib import load_library

    return load_library()


def p(t):
    return C.c_void_p(t.data_ptr())


def run(lib, x, w, T, mode):
    N, K = w.shape
    y = torch.full((T + 1, N), 7.0, device="cuda", dtype=torch.float32 if mode == PLAIN_F32 else torch.bfloat16)
    ms = C.c_float()
    assert lib.tgis_k_gemm(p(x), p(w), p(y), T, N, K, x.shape[0], 0, 1, C.byref(ms), mode) == 0, lib.tgis_k_last_error()
    return y


@pytest.mark.parametrize("mode", [PLAIN, PLAIN_F32, SWIGLU, GEGLU, RELU2])
@pytest.mark.parametrize("T", [1, 7, 8, 9, 17, 32])
@pytest.mark.parametrize("N,K", [(2, 64), (130, 192), (2368, 1024), (2370, 1088), (4738, 2112)])
def test_skinny_products(lib, T, N, K, mode):
    gen = torch.Generator(device="cuda").manual_seed(T + N + K)
    x = torch.randn(32, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    y = run(lib, x, w, T, mode)
    acc = x[:T].double() @ w.double().T
    # fp32 sums of K products in steps of 16: every step may lose an ulp of the running sum, which the sum of magnitudes bounds
    slack = (x[:T].double().abs() @ w.double().abs().T) * (K / 16 + 24) * 2.0 ** -23
    if mode in (SWIGLU, GEGLU):
        g, u, sg, su = acc[:, 0::2], acc[:, 1::2], slack[:, 0::2], slack[:, 1::2]
        if mode == SWIGLU:   # gate, up and silu(gate) are rounded to bf16
            ref = g * torch.sigmoid(g) * u
            tol = 5 * 2.0 ** -8 * ref.abs() + 1.1 * ((sg + 2.0 ** -8 * g.abs()) * u.abs() + g.abs() * su)   # |silu'| <= 1.1
            got, rest = y.reshape(-1)[: T * (N // 2)].view(T, N // 2), y.reshape(-1)[T * (N // 2):]
        else:
            ref = torch.nn.functional.gelu(g, approximate="tanh") * u
            tol = 2.0 ** -8 * ref.abs() + 1.13 * sg * u.abs() + g.abs() * su + 1e-6 * g.abs() * u.abs()
            got, rest = y[:T, : N // 2], torch.cat([y[:T, N // 2:].reshape(-1), y[T]])   # (this hook: rows of N elements)
    else:
        got, rest = y[:T], y[T]
        ref, tol = (acc.clamp(min=0) ** 2, (2 * acc.abs() + slack) * slack) if mode == RELU2 else (acc, slack)
        tol = tol + (0 if mode == PLAIN_F32 else 2.0 ** -8) * ref.abs()
    over = (got.double() - ref).abs() - tol
    assert float(over.max()) <= 0, float(over.max())
    assert bool((rest == 7.0).all())


@pytest.mark.parametrize("T", [1, 8, 9, 32])
@pytest.mark.parametrize("n_q,n_kv", [(6, 2), (8, 8), (32, 8)])
def test_skinny_qkv_with_rope_equals_the_two_launches(lib, T, n_q, n_kv):
    """The fused rotary embedding and cache scatter, bit for bit what the product and the rope kernel do one after the other;
    a token without a slot leaves the cache alone."""
    K, N, blocks = 768, (n_q + 2 * n_kv) * 128, 4
    gen = torch.Generator(device="cuda").manual_seed(T + n_q)
    x = torch.randn(32, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=gen, device="cuda") * 0.05).bfloat16()
    cs = torch.randn(64, 128, generator=gen, device="cuda").bfloat16()
    pos = (C.c_int32 * T)(*[(7 * i) % 64 for i in range(T)])
    slots = (C.c_int32 * T)(*[-1 if i == T - 1 and T > 1 else (5 * i + 3) % (blocks * 32) for i in range(T)])
    caches = [[torch.full((blocks, n_kv, 32 * 128), 3.0, device="cuda").bfloat16() for _ in range(2)] for _ in range(2)]
    y = [torch.empty(32, N, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    rc = lib.tgis_k_gemm_rope(p(x), p(w), p(y[0]), T, n_q, n_kv, K, 32, pos, slots, p(cs), p(caches[0][0]), p(caches[0][1]))
    if rc == 1:
        pytest.skip("this shape does not fuse")
    assert rc == 0
    y[1][:T] = run(lib, x, w, T, PLAIN)[:T]
    assert lib.tgis_k_rope_kv(p(y[1]), pos, slots, p(cs), p(caches[1][0]), p(caches[1][1]), T, n_q, n_kv) == 0
    assert torch.equal(y[0][:T], y[1][:T])
    for a, b in zip(*caches):
        assert torch.equal(a, b)


@pytest.mark.parametrize("N,K", [(2368, 1024), (2384, 1024), (4480, 960), (4736, 896), (4864, 896), (768, 3072)])
@pytest.mark.parametrize("mode", [PLAIN_F32, SWIGLU])
def test_a_row_is_the_same_beside_7_8_or_31_others(lib, N, K, mode):
    gen = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(32, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    n = N // 2 if mode == SWIGLU else N
    rows = {T: run(lib, x, w, T, mode).reshape(-1)[: T * n].view(T, n) for T in (1, 8, 9, 32)}
    assert torch.equal(rows[1], rows[32][:1]) and torch.equal(rows[8], rows[32][:8]) and torch.equal(rows[9], rows[32][:9])
