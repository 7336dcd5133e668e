"""Products of more than 256 tokens (64 where there are many weight rows) and of expert segments on CTA pairs (csrc/gemm_pair.cu) against 64-bit torch: token counts around the 32-token
unit and the 256-token tile, weight rows around the 256-row pair tile, every epilogue, and nothing written outside Y."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

PLAIN, PLAIN_F32, SWIGLU, GEGLU, RELU2 = 0, 1, 2, 3, 4   # tgis_k_gemm out modes


@pytest.fixture(scope="module")
def lib():
    from vllm_tgis_adapter_b200.engine._lib import load_library

    return load_library()


def run(lib, x, w, T, mode, rows):
    N, K = w.shape
    y = torch.full((T + 1, N), 7.0, device="cuda", dtype=torch.float32 if mode == PLAIN_F32 else torch.bfloat16)
    ms = C.c_float()
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.tgis_k_gemm(p(x), p(w), p(y), T, N, K, rows, 0, 1, C.byref(ms), mode) == 0, lib.tgis_k_last_error()
    return y


@pytest.mark.parametrize("mode", [PLAIN, PLAIN_F32, SWIGLU, GEGLU, RELU2])
@pytest.mark.parametrize("T,N,K", [(257, 256, 256), (288, 258, 320), (289, 130, 64), (511, 520, 512), (512, 8, 768), (513, 2128, 256), (2050, 3000, 1088), (65, 9474, 192), (256, 9600, 320)])
def test_pair_products(lib, T, N, K, mode):
    gen = torch.Generator(device="cuda").manual_seed(T + N + K)
    rows = max(T, 256) + 3   # fewer rows than the last token tile covers: the rest is read as zeros
    x = torch.randn(rows, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    y = run(lib, x, w, T, mode, rows)
    acc = x[:T].double() @ w.double().T
    # fp32 sums of K products in steps of 16: every step may lose an ulp of the running sum, which the sum of magnitudes bounds
    slack = (x[:T].double().abs() @ w.double().abs().T) * (K / 16 + 8) * 2.0 ** -23
    if mode == SWIGLU:   # gate, up and silu(gate) are rounded to bf16: 2^-8 each, and the result's own rounding
        g, u = acc[:, 0::2], acc[:, 1::2]
        sg, su = slack[:, 0::2], slack[:, 1::2]
        ref = g * torch.sigmoid(g) * u
        tol = 5 * 2.0 ** -8 * ref.abs() + 1.1 * ((sg + 2.0 ** -8 * g.abs()) * u.abs() + g.abs() * su)   # |silu'| <= 1.1
    elif mode == GEGLU:
        g, u = acc[:, 0::2], acc[:, 1::2]
        ref = torch.nn.functional.gelu(g, approximate="tanh") * u
        tol = 2.0 ** -8 * ref.abs() + 1.13 * slack[:, 0::2] * u.abs() + g.abs() * slack[:, 1::2] + 1e-6 * g.abs() * u.abs()
    elif mode == RELU2:
        ref = acc.clamp(min=0) ** 2
        tol = 2.0 ** -8 * ref + (2 * acc.abs() + slack) * slack
    else:
        ref, tol = acc, slack + (0 if mode == PLAIN_F32 else 2.0 ** -8) * acc.abs()
    flat = y.reshape(-1)
    if mode == GEGLU:   # (this hook gives the GeGLU product rows of N elements, half of each written)
        got, rest = y[:T, : N // 2], torch.cat([y[:T, N // 2:].reshape(-1), y[T]])
    elif mode == SWIGLU:
        got, rest = flat[: T * (N // 2)].view(T, N // 2), flat[T * (N // 2):]
    else:
        got, rest = y[:T], y[T]
    over = (got.double() - ref).abs() - tol
    assert float(over.max()) <= 0, (float(over.max()), float((over > 0).double().mean()))
    assert bool((rest == 7.0).all())
    assert torch.equal(run(lib, x, w, T, mode, rows), y)   # an output is one sum in ascending k: the same bits every time


def test_pair_product_does_not_depend_on_the_other_tokens(lib):
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(1200, 512, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(640, 512, generator=gen, device="cuda") * 512 ** -0.5).bfloat16()
    whole = run(lib, x, w, 1200, PLAIN_F32, 1200)
    part = run(lib, x[700:].contiguous(), w, 300, PLAIN_F32, 500)   # other tiles, other neighbours
    assert torch.equal(part[:300], whole[700:1000])


ANY = dict(plain=0, swiglu=1, geglu=3, relu2=5, gelu=6)   # include/tgis_kernels.h tgis_k_gemm_any modes


@pytest.mark.parametrize("mode", list(ANY))
@pytest.mark.parametrize("counts,N,K,gathered", [
    ([1], 256, 64, True), ([0, 33, 0, 31, 32], 130, 72, True), ([256, 257, 0, 1], 300, 192, False), ([700, 0, 5], 512, 264, True),
    ([2, 3] * 40 + [0] * 20, 96, 128, True), ([0, 0, 3], 64, 64, False)])
def test_pair_expert_segments(lib, counts, N, K, gathered, mode):
    """One weight matrix per row segment: empty, single-row and ragged segments, rows gathered through an index list (two
    places per row) or in place; bf16 results, and the plain sums in fp32 too."""
    gen = torch.Generator(device="cuda").manual_seed(N + K + len(counts))
    E, rows = len(counts), sum(counts)
    seg = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    expert = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(counts, device="cuda"))
    x = torch.randn((rows + 1) // 2 if gathered else rows, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(E, N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    order = torch.randperm(rows, generator=gen, device="cuda").int()
    scale = torch.rand(rows, generator=gen, device="cuda") + 0.5
    src = (order.long() // 2) if gathered else torch.arange(rows, device="cuda")
    acc, mag = (torch.empty(rows, N, dtype=torch.float64, device="cuda") for _ in range(2))
    for e in range(E):
        r = expert == e
        acc[r] = x[src[r]].double() @ w[e].double().T
        mag[r] = x[src[r]].double().abs() @ w[e].double().abs().T
    slack = mag * (K / 16 + 8) * 2.0 ** -23
    if mode in ("swiglu", "geglu"):
        act = torch.nn.functional.silu if mode == "swiglu" else (lambda v: torch.nn.functional.gelu(v, approximate="tanh"))
        g, u = acc[:, 0::2], acc[:, 1::2]
        ref = act(g) * u
        tol = 1.13 * slack[:, 0::2] * u.abs() + g.abs() * slack[:, 1::2] + 1e-6 * g.abs() * u.abs()   # |act'| <= 1.13
    elif mode == "relu2":
        s = (scale[order.long()] if gathered else scale).double()[:, None]
        ref, tol = (acc * s).clamp(min=0) ** 2, (2 * (acc * s).abs() + slack * s) * slack * s
    else:
        ref = torch.nn.functional.gelu(acc) if mode == "gelu" else acc
        tol = 1.13 * slack + (1e-6 * acc.abs() if mode == "gelu" else 0)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    for y_dt in ([1, 0] if mode == "plain" else [1]):
        y = torch.full((rows + 1, ref.shape[1]), 7.0, device="cuda", dtype=torch.bfloat16 if y_dt else torch.float32)
        assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, y_dt, rows, N, K, K, K, y.shape[1], 1, 0, 0, 0, p(seg), E, N * K,
                                   p(order) if gathered else None, 2, ANY[mode], p(scale) if mode == "relu2" else None, 0) == 0, lib.tgis_k_last_error()
        over = (y[:rows].double() - ref).abs() - tol - (2.0 ** -8 * ref.abs() if y_dt else 0)
        assert float(over.max()) <= 0, float(over.max())
        assert bool((y[rows] == 7.0).all())


def test_expert_swiglu_divides_as_the_other_kernels_do(lib):
    """Every bf16 gate (with bits below it, infinities and NaN among them) and ups of every size: the bits of the one-CTA product
    over the same rows, whose epilogue divides with IEEE rounding."""
    gen = torch.Generator(device="cuda").manual_seed(11)
    gate = torch.arange(-32768, 32768, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)
    low = (gate.double() * (torch.rand(65536, generator=gen, device="cuda").double() - 0.5) * 2.0 ** -8).bfloat16()   # gate + low is one fp32 number
    low = torch.where(gate.float().abs().isfinite() & (gate.float().abs() > 2.0 ** -100), low, torch.zeros_like(low))
    T, N, K = 301, 131072, 64
    w = torch.zeros(N, K, device="cuda", dtype=torch.bfloat16)
    w[0::2, 0], w[0::2, 1], w[1::2, 2] = gate, low, 1.0
    x = torch.zeros(T, K, device="cuda", dtype=torch.bfloat16)
    x[:, 0] = 1.0
    x[1::2, 1] = 1.0
    x[:, 2] = (torch.randn(T, generator=gen, device="cuda") * torch.exp2(torch.randint(-30, 30, (T,), generator=gen, device="cuda").float())).bfloat16()
    x[:6, 2] = torch.tensor([1.0, 1.0, -1.0, 0.0, 3e38, 1e-38], device="cuda").bfloat16()
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731

    def product(seg):
        y = torch.empty(T, N // 2, device="cuda", dtype=torch.bfloat16)
        assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, 1, T, N, K, K, K, N // 2, 1, 0, 0, 0, p(seg), 1 if seg is not None else 0, N * K, None, 1, ANY["swiglu"],
                                   None, 0) == 0, lib.tgis_k_last_error()
        return y

    pairs, one_cta = product(torch.tensor([0, T], device="cuda", dtype=torch.int32)), product(None)
    assert torch.equal(pairs.isnan(), one_cta.isnan())
    differ = (pairs.view(torch.int16) != one_cta.view(torch.int16)) & ~pairs.isnan()
    assert int(differ.sum()) == 0, (int(differ.sum()), gate[differ.any(0)][:8].tolist())


def test_dense_swiglu_divides_as_the_register_kernel_does(lib):
    """Every bf16 gate through the epilogue that skips the IEEE division where it cannot matter, against the kernel of up to 8
    tokens, which always divides."""
    gen = torch.Generator(device="cuda").manual_seed(12)
    gate = torch.arange(-32768, 32768, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)
    K = 64
    w = torch.zeros(131072, K, device="cuda", dtype=torch.bfloat16)
    w[0::2, 0], w[1::2, 1] = gate, 1.0
    x = torch.zeros(300, K, device="cuda", dtype=torch.bfloat16)
    x[:, 0] = 1.0
    x[:, 1] = torch.randn(300, generator=gen, device="cuda").bfloat16()
    x[:4, 1] = torch.tensor([1.0, -1.0, 0.0, 3e38], device="cuda").bfloat16()
    many = run(lib, x, w, 300, SWIGLU, 300).reshape(-1)[: 300 * 65536].view(300, 65536)[:8]
    few = torch.cat([run(lib, x[:256].contiguous(), w[at: at + 16384].contiguous(), 8, SWIGLU, 256).reshape(-1)[: 8 * 8192].view(8, 8192) for at in range(0, 131072, 16384)], 1)
    assert torch.equal(many.isnan(), few.isnan())
    assert bool(((many.view(torch.int16) == few.view(torch.int16)) | many.isnan()).all())


@pytest.mark.parametrize("groups", [2047, 2048, 2049])
def test_many_segments_of_few_rows(lib, groups):
    """More segments than rows, up to the number that the launch takes and one more (which goes to the one-CTA kernel)."""
    gen = torch.Generator(device="cuda").manual_seed(groups)
    rows, N, K = 45, 72, 64
    owner = torch.sort(torch.randint(0, groups, (rows,), generator=gen, device="cuda")).values
    owner[-1] = groups - 1
    seg = torch.zeros(groups + 1, device="cuda", dtype=torch.int64)
    seg[1:] = torch.bincount(owner, minlength=groups).cumsum(0)
    seg = seg.int()
    x = torch.randn(rows, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(groups, N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    y = torch.full((rows + 1, N), 7.0, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    lib.tgis_k_pair_fault(0)
    assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, 0, rows, N, K, K, K, N, 1, 0, 0, 0, p(seg), groups, N * K, None, 1, 0, None, 0) == 0, lib.tgis_k_last_error()
    assert lib.tgis_k_pair_fault(0) == (1 if groups <= 2048 else 0)
    wd = w[owner].double()
    want, slack = torch.einsum("rk,rnk->rn", x.double(), wd), torch.einsum("rk,rnk->rn", x.double().abs(), wd.abs()) * 12 * 2.0 ** -23
    assert float(((y[:rows].double() - want).abs() - slack).max()) <= 0
    assert bool((y[rows] == 7.0).all())


def test_gathered_rows_without_room_go_to_the_one_cta_kernel(lib):
    gen = torch.Generator(device="cuda").manual_seed(3)
    counts, N, K = [100, 0, 33, 7], 136, 128
    rows, E = sum(counts), len(counts)
    seg = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    expert = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(counts, device="cuda"))
    x = torch.randn(rows // 2, K, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(E, N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    order = torch.randperm(rows, generator=gen, device="cuda").int()
    src = x[order.long() // 2].double()
    want = torch.einsum("rk,rnk->rn", src, w[expert].double())
    slack = torch.einsum("rk,rnk->rn", src.abs(), w[expert].double().abs()) * (K / 16 + 8) * 2.0 ** -23
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    try:
        for room, pairs in ((-1, 1), (rows * K * 2, 1), (rows * K * 2 - 2, 0), (0, 0)):
            lib.tgis_k_gemm_any_room(room)
            y = torch.full((rows + 1, N), 7.0, device="cuda")
            lib.tgis_k_pair_fault(0)
            assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, 0, rows, N, K, K, K, N, 1, 0, 0, 0, p(seg), E, N * K, p(order), 2, 0, None, 0) == 0, lib.tgis_k_last_error()
            assert lib.tgis_k_pair_fault(0) == pairs
            assert float(((y[:rows].double() - want).abs() - slack).max()) <= 0
            assert bool((y[rows] == 7.0).all())
    finally:
        lib.tgis_k_gemm_any_room(-1)
