"""Kernels of steps with one token per sequence: the memories' and the selective scan's against the kernels that also take longer
portions (the same bits, whatever the mode), the row tail and the products of few rows against 64 bits."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.fixture(scope="module")
def lib():
    from vllm_tgis_adapter_b200.engine._lib import load_library

    return load_library()


MODES = ["decay", "gated", "hgrn", "ssd", "lightning", "retention", "gla"]


def _scan(lib, mode, d, dv, H, fresh, extra):
    """One token for each of 5 sequences; `extra`: one more sequence of two tokens, so that the launch takes the general kernel."""
    n, gen = 5, torch.Generator(device="cuda").manual_seed(d * 1000 + dv + len(mode))
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    T, f = n + 2, C.c_float
    x = rnd(T, 3 * H * d + H * dv + 2 * H + 16)
    ld, q, k, dec, v, gate = x.shape[1], x, x[:, H * d:], x[:, 2 * H * d:], x[:, 3 * H * d:], x[:, 3 * H * d + H * dv:]
    S, nrm, mx = rnd(n + 1, H, d, dv), rnd(n + 1, H, d).abs(), rnd(n + 1, H)
    w0, u, b1, b2, last = rnd(H * d), rnd(H * d).sigmoid(), rnd(H), rnd(H), torch.zeros(n + 1, 24, device="cuda")
    out = torch.zeros(T, H * dv, device="cuda")
    kv = 1 if fresh else 9
    meta = [e for s in range(n) for e in (s, 1, kv + (s == 2), 0)] + ([n, 2, 6, 0] if extra else [])
    slots = torch.tensor([3, 1, 4, 0, 2, 5, 5], dtype=torch.int32, device="cuda")
    seqs, ns, pos = (C.c_int32 * len(meta))(*meta), n + (1 if extra else 0), torch.zeros(T, dtype=torch.int32, device="cuda")
    sl, heads = slots, rnd(H).sigmoid()
    if mode in ("decay", "gated", "hgrn"):
        rc = lib.tgis_k_outer_scan({"decay": 0, "gated": 1, "hgrn": 3}[mode], p(q), p(k), p(v), ld, ld, ld, f(d ** -0.5), p(dec), ld, p(w0), p(u), p(gate),
                                   p(gate[:, H:]), ld, p(b1), p(b2), f(6.0), p(S), p(nrm), p(mx), p(out), H * dv, H, d, dv, p(x), p(last), 24, seqs, ns, p(sl))
    elif mode == "ssd":
        rc = lib.tgis_k_ssd_scan(p(q), p(k), p(v), ld, ld, ld, p(gate), ld, p(b1), p(b2), p(heads), p(S), p(out), H * dv, H, 1, d, dv, seqs, ns, p(sl))
    elif mode == "lightning":
        rc = lib.tgis_k_lightning_scan(p(q), p(k), p(v), ld, ld, ld, p(heads), p(S), p(out), H * dv, H, d, dv, seqs, ns, p(sl), 0)
    elif mode == "retention":
        table = torch.tensor([[1.0, 0.0]], device="cuda")
        rc = lib.tgis_k_retention_scan(p(x), ld, 0, H * d, 3 * H * d, p(table), p(pos), 2, f(0.5), p(heads), p(S), p(out), H * dv, H, d, dv, seqs, ns, p(sl), T, 0)
    else:
        a2 = rnd(H * d, 16).bfloat16()
        rc = lib.tgis_k_gla_scan(p(x), ld, 0, H * d, 3 * H * d, ld - 16, f(0.5), p(a2), 16, p(w0), f(0.25), p(S), p(out), H * dv, H, d, dv, seqs, ns, p(sl), T, 0)
    assert rc == 0
    return [t.clone() for t in (out[:n], S[:n], nrm[:n], mx[:n], last[:n])]


@pytest.mark.parametrize("fresh", [True, False])
@pytest.mark.parametrize("d,dv,H", [(64, 64, 4), (128, 256, 2), (128, 64, 1), (64, 384, 3)])
@pytest.mark.parametrize("mode", MODES)
def test_memory_step_has_the_bits_of_the_general_kernel(lib, mode, d, dv, H, fresh):
    step, general = _scan(lib, mode, d, dv, H, fresh, False), _scan(lib, mode, d, dv, H, fresh, True)
    assert step[0].abs().max() > 0
    for a, b in zip(step, general):
        assert torch.equal(a, b)


@pytest.mark.parametrize("taps", [1, 4, 7])
@pytest.mark.parametrize("inner", [64, 100])
def test_selective_step_has_the_bits_of_the_general_kernel(lib, inner, taps):
    res = []
    for extra in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(inner + taps)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
        n, N, R = 4, 16, 8
        T = n + 2
        x, xz, proj, dt = rnd(T, inner), rnd(T, 2 * inner), rnd(T, R + 2 * N), rnd(T, inner)
        b, A, D = rnd(inner), rnd(inner, N), rnd(inner)
        S, conv, out = rnd(n + 1, inner, N), rnd(n + 1, max(taps - 1, 1), inner), torch.zeros(T, inner, device="cuda")
        meta = [e for s, kv in enumerate((1, 2, 5, 40)) for e in (s, 1, kv, 0)] + ([n, 2, 9, 0] if extra else [])
        slots = torch.tensor([2, 0, 3, 1, 4, 4], dtype=torch.int32, device="cuda")
        rc = lib.tgis_k_selective_scan(p(x), p(xz), 2 * inner, p(proj), R + 2 * N, R, p(dt), p(b), p(A), p(D), p(S), p(conv), p(out), 0, inner, N, taps,
                                       (C.c_int32 * len(meta))(*meta), n + (1 if extra else 0), p(slots))
        assert rc == 0
        res.append([out[:n].clone(), S[:n].clone(), conv[:n].clone()])
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("hidden", [4, 1020, 1024, 1028, 2048, 2052])
@pytest.mark.parametrize("top,side", [(0, False), (6, True), (8, False), (11, True)])
def test_row_tail_with_and_without_experts(lib, hidden, top, side):
    few, T, eps, gen = 3, 150, 1e-5, torch.Generator(device="cuda").manual_seed(hidden + top)   # more rows than SMs: the other kernel
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    main, rows, inv = rnd(T, hidden), rnd(T * max(top, 1), hidden), torch.randperm(T * max(top, 1), device="cuda", generator=gen).int()
    mix, sy, sg, wp, wq, resid = rnd(T, max(top, 1)), rnd(T, hidden), rnd(T), rnd(hidden), rnd(hidden), rnd(T, hidden)
    want, out = resid.to(F64), torch.zeros(T, hidden, device="cuda")
    y = main.to(F64) if top == 0 else torch.einsum("tk,tkh->th", mix.to(F64), rows.to(F64)[inv.long()].view(T, top, hidden))
    if side:
        y = y + sg.to(F64)[:, None] * sy.to(F64)
    rms = lambda z: z / torch.sqrt((z * z).mean(1, keepdim=True) + eps)
    want = want + 0.5 * rms(y) * (1 + wp.to(F64))
    res = []
    for n in (few, T):
        res.append((resid.clone(), out.clone()))
        rc = lib.tgis_k_resid_tail(p(main) if top == 0 else None, p(rows) if top else None, p(inv), p(mix), top, p(sy) if side else None,
                                   p(sg) if side else None, p(wp), p(wq), p(res[-1][0]), p(res[-1][1]), 0, C.c_float(0.5), C.c_float(1.0), C.c_float(eps), n, hidden)
        assert rc == 0
    for a, b in zip(*res):
        assert torch.equal(a[:few], b[:few])
    resid, out = res[1]
    # fp32: twelve terms a value, sums of up to 2052 squares over 256 threads, three roundings of a product each
    assert ((resid - want).abs() <= 3e-6 * (1 + want.abs())).all()
    assert ((out - rms(want) * (1 + wq.to(F64))).abs() <= 2e-5 * (1 + want.abs())).all()


@pytest.mark.parametrize("hidden", [4, 1020, 1024, 1028, 2048])
@pytest.mark.parametrize("out_dt", [0, 1])
@pytest.mark.parametrize("form", ["pair", "pair, cast", "pair, no norm", "extra", "extra, no norm", "two norms and a gate", "mixture and a gate"])
def test_row_tail_has_the_bits_of_the_general_kernel(lib, hidden, out_dt, form):
    few, T, top, eps, gen = 5, 150, 3, C.c_float(1e-5), torch.Generator(device="cuda").manual_seed(hidden)   # more rows than SMs: the general one
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    y, z, resid, ws, rows = rnd(T, hidden), rnd(T, hidden), rnd(T, hidden), [rnd(hidden) for _ in range(5)], rnd(T * top, hidden)
    inv, gate = torch.randperm(T * top, device="cuda", generator=gen).int(), rnd(T)
    res = []
    for n in (few, T):
        r, dot = resid.clone(), torch.zeros(T, device="cuda")
        o, o2 = (torch.zeros(T, hidden, device="cuda", dtype=torch.bfloat16 if out_dt else torch.float32) for _ in range(2))
        post, pre = None if "no norm" in form else p(ws[0]), p(ws[1])
        if form.startswith("pair"):
            cast = form == "pair, cast"
            rc = lib.tgis_k_resid_tail_pair(p(y), p(z), p(ws[2]), p(ws[3]), post, None if cast else pre, p(r), p(o), out_dt, int(cast), eps, n, hidden)
        elif form == "mixture and a gate":
            rc = lib.tgis_k_resid_tail_plain(None, p(rows), p(inv), C.c_float(0.3), top, p(z), p(gate), pre, p(r), p(o), out_dt, p(ws[4]), p(dot), eps, n, hidden)
        else:
            two = form.startswith("two")
            rc = lib.tgis_k_resid_tail_two(p(y), p(z), post, pre, p(ws[2]) if two else None, p(ws[4]) if two else None, p(r), p(o), p(o2) if two else None,
                                           out_dt, p(dot) if two else None, C.c_float(0.7), C.c_float(1.0), eps, n, hidden)
        assert rc == 0
        res.append([t[:few] for t in (r, o, o2, dot)])
    assert all(torch.equal(a, b) for a, b in zip(*res))
    assert not torch.equal(res[0][0], resid[:few]) and bool(res[0][1].any())
    assert bool(res[0][2].any()) == form.startswith("two") and bool(res[0][3].any()) == ("gate" in form)


@pytest.mark.parametrize("T", [1, 8, 9, 32])
@pytest.mark.parametrize("heads,N,K,scaled,y_dt", [(16, 512, 128, False, 0), (16, 128, 512, True, 1), (3, 40, 64, False, 1), (5, 24, 320, True, 0)])
def test_products_per_head(lib, T, heads, N, K, scaled, y_dt):
    gen = torch.Generator(device="cuda").manual_seed(T * N + K)
    x = torch.randn(T, heads, K + 8, device="cuda", generator=gen).bfloat16()
    w = (torch.randn(heads, N, K, device="cuda", generator=gen) * K ** -0.5).bfloat16()
    s, y = torch.rand(T, heads, device="cuda", generator=gen), torch.zeros(T, heads, N + 4, device="cuda", dtype=torch.bfloat16 if y_dt else torch.float32)
    rc = lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, y_dt, T, N, K, heads * (K + 8), K, heads * (N + 4), heads, K + 8, N * K, N + 4, None, 0, 0, None, 1,
                             2 if scaled else 0, p(s), heads)
    assert rc == 0
    want = torch.einsum("thk,hnk->thn", x[:, :, :K].to(F64), w.to(F64)) * (s.to(F64)[:, :, None] if scaled else 1)
    bound = 1e-5 + (2 ** -8 * want.abs() if y_dt else 0)   # fp32 sums of products of about K^-0.5; the result's rounding
    assert ((y[:, :, :N].to(F64) - want).abs() <= bound).all()
    assert (y[:, :, N:] == 0).all()


@pytest.mark.parametrize("T,N,K", [(1, 64, 2048), (32, 64, 2048), (5, 7, 300), (64, 127, 256)])
@pytest.mark.parametrize("y_dt", [0, 1])
def test_tanh_of_few_outputs(lib, T, N, K, y_dt):
    gen = torch.Generator(device="cuda").manual_seed(T * N + K)
    x, w = torch.randn(T, K, device="cuda", generator=gen).bfloat16(), (torch.randn(N, K, device="cuda", generator=gen) * K ** -0.5).bfloat16()
    y = torch.zeros(T, N, device="cuda", dtype=torch.bfloat16 if y_dt else torch.float32)
    assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, y_dt, T, N, K, K, K, N, 1, 0, 0, 0, None, 0, 0, None, 1, 4, None, 0) == 0
    want = torch.tanh(x.to(F64) @ w.to(F64).T)
    assert ((y.to(F64) - want).abs() <= 1e-5 + (2 ** -8 * want.abs() if y_dt else 0)).all()


@pytest.mark.parametrize("inner", [128, 516])
def test_short_convolution_of_prompts_has_the_bits_of_single_tokens(lib, inner):
    """300 tokens in portions of every length around the run of eight, fresh and carried on, against the same tokens in launches of
    fewer than 256 (the kernel with a token per thread)."""
    gen = torch.Generator(device="cuda").manual_seed(inner)
    lens, before = [1, 2, 3, 4, 7, 8, 9, 16, 17, 40, 93, 100], [0, 5, 1, 0, 2, 3, 0, 1, 9, 2, 0, 30]
    T, n = sum(lens), len(lens)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    xz, w, b, state = rnd(T, 2 * inner), rnd(inner, 4), rnd(inner), rnd(n, 3, inner)
    slot = torch.tensor([s for s, k in enumerate(lens) for _ in range(k)], dtype=torch.int32, device="cuda")
    pos = torch.tensor([q + i for k, q in zip(lens, before) for i in range(k)], dtype=torch.int32, device="cuda")
    res, cut = [], sum(lens[:-1])
    for parts in ([(0, T)], [(0, cut), (cut, T)]):
        f32, op = torch.zeros(T, inner, device="cuda"), torch.zeros(T, inner, device="cuda", dtype=torch.bfloat16)
        for a, e in parts:
            assert lib.tgis_k_short_conv(p(xz[a:]), 2 * inner, inner, p(w), p(b), 4, p(pos[a:].clone()), p(slot[a:].clone()), p(state), p(f32[a:]), p(op[a:]), 1, e - a) == 0
        res.append((f32, op))
    assert T == 300 and cut < 256
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
