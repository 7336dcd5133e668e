"""A norm between two products of a few tokens, inside them (csrc/gemm_skinny.cu) and as a launch of its own: the same bits, in the residual
stream and behind the second product, for every variant of either and at the edges of the column groups whose squares are summed; behind a qkv
product also with rotary embedding and the scatter into the caches inside it."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 2])   # plain, SwiGLU
@pytest.mark.parametrize("T", [1, 2, 5, 7, 8])
@pytest.mark.parametrize("K1,H,N2", [(64, 64, 128), (768, 768, 2304), (2048, 768, 2370), (192, 1024, 4738), (704, 1984, 4736), (2048, 2048, 6144), (128, 320, 16)])
def test_norm_inside_the_products_has_the_bits_of_its_own_launch(K1, H, N2, T, mode):
    from vllm_tgis_adapter_b200.engine._lib import load_library

    lib = load_library()
    p = lambda t: C.c_void_p(t.data_ptr())
    gen = torch.Generator(device="cuda").manual_seed(K1 + H + N2 + T)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=gen, device="cuda") * scale).bfloat16()
    a, w1, w2, wn, resid = rnd(T, K1), rnd(H, K1, scale=K1 ** -0.5), rnd(N2, H, scale=H ** -0.5), rnd(H), rnd(T, H, scale=3.0)
    res = []
    for fused in (0, 1):
        r = torch.cat([resid, resid[:1] * 0 + 7])
        y = torch.full((T * N2 // (2 if mode == 2 else 1) + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
        assert lib.tgis_k_skinny_norm_chain(p(a), p(w1), p(r), p(wn), p(w2), p(y), T, K1, H, N2, C.c_float(1e-5), mode, fused) == 0
        assert bool((r[T] == 7).all()) and bool((y[-8:] == 7).all())
        res.append((r[:T], y[:-8]))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    # ... which are those of the arithmetic: products rounded, stream rounded, norm rounded twice
    z = ((a.double() @ w1.double().T).bfloat16().double() + resid.double()).bfloat16().double()
    assert ((res[1][0].double() - z).abs() <= 2.0 ** -7 * z.abs() + 2e-2).all()
    assert res[1][1].isfinite().all() and res[1][1].abs().max() > 0


@pytest.mark.parametrize("T", [1, 2, 5, 8])
@pytest.mark.parametrize("K1,H,n_q,n_kv", [(768, 768, 12, 12), (1024, 2048, 24, 8), (64, 320, 1, 1), (2048, 2048, 35, 1), (2048, 2048, 36, 1)])   # (4736 columns: two waves)
def test_norm_and_rotary_embedding_inside_the_product(K1, H, n_q, n_kv, T):
    from vllm_tgis_adapter_b200.engine._lib import load_library

    lib, N, blocks = load_library(), (n_q + 2 * n_kv) * 128, 4
    p = lambda t: C.c_void_p(t.data_ptr())
    gen = torch.Generator(device="cuda").manual_seed(K1 + H + N + T)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=gen, device="cuda") * scale).bfloat16()
    a, w1, w2, wn, resid, table = rnd(T, K1), rnd(H, K1, scale=K1 ** -0.5), rnd(N, H, scale=H ** -0.5), rnd(H), rnd(T, H, scale=3.0), rnd(64, 128)
    ints = lambda v: (C.c_int32 * T)(*v)
    positions, slots = ints([(7 * t + 3) % 64 for t in range(T)]), ints([(37 * t + 5) % (32 * blocks) for t in range(T)])
    res = []
    for fused in (0, 1):
        r = torch.cat([resid, resid[:1] * 0 + 7])
        y = torch.full((T * N + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
        k, v = (torch.full((blocks * 32 * n_kv * 128 + 8,), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        assert lib.tgis_k_skinny_norm_rope(p(a), p(w1), p(r), p(wn), p(w2), p(y), T, K1, H, n_q, n_kv, C.c_float(1e-5), positions, slots, p(table), p(k), p(v), fused) == 0
        assert all(bool((t[-8:] == 7).all()) for t in (r[T], y, k, v))
        res.append((r, y, k, v))
    assert all(torch.equal(s, t) for s, t in zip(*res))
    assert all(int((t != 7).sum()) > 0.9 * T * n_kv * 128 for t in res[1][2:])   # (all of the tokens' keys and values)
