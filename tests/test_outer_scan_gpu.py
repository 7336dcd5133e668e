"""The outer-product memories against the recurrence written out in 64 bits: more column blocks than the chip holds at once, and keys
that fill the kernel's row groups exactly, by less than four rows, or not at all."""
from __future__ import annotations

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _gated(q, k, v, ig, fg, S, n, m, cap):
    """q, k [H, T, d], v [H, T, dv], gates [H, T]; the state is updated in place.  Out [H, T, dv] and what its rounding errors
    scale with: the sums of the absolute terms, the denominator's share carried through the quotient."""
    out, size, Sa, na = [], [], S.abs(), n.abs()
    for t in range(q.shape[1]):
        i, f = cap * torch.tanh(ig[:, t] / cap), torch.nn.functional.logsigmoid(cap * torch.tanh(fg[:, t] / cap))
        mn = torch.maximum(f + m, i)
        da, db = torch.exp(f + m - mn), torch.exp(i - mn)
        S.mul_(da[:, None, None]).add_(db[:, None, None] * k[:, t, :, None] * v[:, t, None, :])
        n.mul_(da[:, None]).add_(db[:, None] * k[:, t])
        Sa = da[:, None, None] * Sa + (db[:, None, None] * k[:, t, :, None] * v[:, t, None, :]).abs()
        na = da[:, None] * na + (db[:, None] * k[:, t]).abs()
        m.copy_(mn)
        den = (torch.maximum((n * q[:, t]).sum(1).abs(), torch.exp(-m)) + 1e-6)[:, None]
        out.append(torch.einsum("hd,hdv->hv", q[:, t], S) / den)
        size.append((torch.einsum("hd,hdv->hv", q[:, t].abs(), Sa) + out[-1].abs() * (na * q[:, t].abs()).sum(1)[:, None]) / den)
    return torch.stack(out, 1), torch.stack(size, 1), Sa, na


@pytest.mark.parametrize("d,dv,H,slots,T", [(128, 256, 8, 40, 2), (64, 64, 2, 3, 37), (256, 33, 1, 2, 17), (67, 40, 2, 2, 16), (2, 3, 1, 2, 33)])
def test_gated_memory_carried_on(d, dv, H, slots, T):
    """The portion before left a state in every slot: each column block of a head starts from the same normaliser and maximum."""
    from vllm_tgis_adapter_b200.engine._lib import load_library

    lib = load_library()
    g = torch.Generator().manual_seed(d)
    width = H * (2 * d + dv + 2)
    x = torch.randn(slots * T, width, generator=g)
    S, n, m = torch.randn(slots, H, d, dv, generator=g), torch.rand(slots, H, d, generator=g) + 0.5, torch.randn(slots, H, generator=g)
    ib, fb = torch.randn(H, generator=g), torch.randn(H, generator=g)
    y, Sg, ng, mg = x.cuda(), S.cuda(), n.cuda(), m.cuda()
    out = torch.full((slots * T, H * dv), float("nan"), device="cuda")
    meta = [e for s in range(slots) for e in (s * T, T, 5 + T, 0)]
    tok_slot = torch.arange(slots, dtype=torch.int32).repeat_interleave(T).cuda()
    ibg, fbg = ib.cuda(), fb.cuda()
    rc = lib.tgis_k_outer_scan(1, _p(y), _p(y[:, H * d:]), _p(y[:, 2 * H * d:]), width, width, width, ctypes.c_float(d ** -0.5), None, 0, None,
                               None, _p(y[:, width - 2 * H:]), _p(y[:, width - H:]), width, _p(ibg), _p(fbg), ctypes.c_float(6.0), _p(Sg), _p(ng),
                               _p(mg), _p(out), H * dv, H, d, dv, None, None, 0, (ctypes.c_int32 * len(meta))(*meta), slots, _p(tok_slot))
    assert rc == 0
    for s in range(slots):
        r = x[s * T:(s + 1) * T].to(F64)
        heads = lambda a, w: r[:, a:a + H * w].reshape(T, H, w).transpose(0, 1)
        S1, n1, m1 = S[s].to(F64), n[s].to(F64), m[s].to(F64)
        q = heads(0, d) * d ** -0.5
        ref, size, Sa, na = _gated(q, heads(H * d, d), heads(2 * H * d, dv), r[:, width - 2 * H:width - H].t() + ib[:, None],
                                   r[:, width - H:].t() + fb[:, None], S1, n1, m1, 6.0)
        # a step rounds a state entry three times; its two exponentials take arguments of up to ~12 whose own rounding counts in full
        # (a gate is three functions of 4 ulp), ~27 units of roundoff together; an output then sums d terms
        c = (27 * T + 64) * 2.0 ** -24
        assert ((Sg[s].cpu().to(F64) - S1).abs() <= c * Sa + 1e-30).all() and ((ng[s].cpu().to(F64) - n1).abs() <= c * na + 1e-30).all()
        assert (mg[s].cpu().to(F64) - m1).abs().max() <= c * 12
        o = out[s * T:(s + 1) * T].cpu().to(F64).reshape(T, H, dv).transpose(0, 1)
        assert ((o - ref).abs() <= (c + d * 2.0 ** -24) * size).all()


@pytest.mark.parametrize("d,H,T", [(64, 3, 37), (128, 1, 16), (256, 1, 17), (62, 2, 5), (3, 1, 20)])
def test_decayed_memory_carried_on(d, H, T):
    """A decay per row, keys that fill the row groups and keys that do not: out = q (S + u k v), then S = w S + k v."""
    from vllm_tgis_adapter_b200.engine._lib import load_library

    lib = load_library()
    g = torch.Generator().manual_seed(d + T)
    A = H * d
    r, k, v, raw = (torch.randn(T, A, generator=g) for _ in range(4))
    w0, u, S = torch.randn(A, generator=g) - 1.0, torch.randn(A, generator=g), torch.randn(1, H, d, d, generator=g)
    dev = [t.cuda() for t in (r, k, v, raw, w0, u)]
    Sg, out = S.cuda(), torch.full((T, A), float("nan"), device="cuda")
    tok_slot = torch.zeros(T, dtype=torch.int32, device="cuda")
    rc = lib.tgis_k_outer_scan(0, _p(dev[0]), _p(dev[1]), _p(dev[2]), A, A, A, ctypes.c_float(0.5), _p(dev[3]), A, _p(dev[4]), _p(dev[5]), None, None, 0,
                               None, None, ctypes.c_float(0.0), _p(Sg), None, None, _p(out), A, H, d, d, None, None, 0,
                               (ctypes.c_int32 * 4)(0, T, 9 + T, 0), 1, _p(tok_slot))
    assert rc == 0
    per_head = lambda t: t.to(F64).reshape(T, H, d)
    q, kk, vv = per_head(r) * 0.5, per_head(k), per_head(v)
    w = torch.exp(-torch.exp(per_head(raw) + w0.to(F64).reshape(H, d)))
    S1, Sa, uu = S[0].to(F64), S[0].to(F64).abs(), u.to(F64).reshape(H, d)
    # three roundings a step; a decay's inner exponential (up to ~e^3) passes its error of ~4 units on multiplied by its value
    c = (3 + 4 * 20) * T * 2.0 ** -24
    for t in range(T):
        kv = kk[t, :, :, None] * vv[t, :, None, :]
        o = torch.einsum("hd,hdv->hv", q[t], S1 + uu[:, :, None] * kv)
        size = torch.einsum("hd,hdv->hv", q[t].abs(), Sa + uu[:, :, None].abs() * kv.abs())
        assert ((out[t].cpu().to(F64).reshape(H, d) - o).abs() <= (c + (d + 4) * 2.0 ** -24) * size).all()
        S1, Sa = w[t, :, :, None] * S1 + kv, w[t, :, :, None] * Sa + kv.abs()
    assert ((Sg[0].cpu().to(F64) - S1).abs() <= c * Sa + 1e-30).all()


def test_gated_memory_in_a_slot_of_any_number():
    """The hook's own counters reach as far as the slots it is given."""
    from vllm_tgis_adapter_b200.engine._lib import load_library

    lib, d, dv, slot, T = load_library(), 8, 40, 5000, 19
    g = torch.Generator().manual_seed(5)
    width = 2 * d + dv + 2
    y, bias = torch.randn(T, width, generator=g).cuda(), torch.zeros(1, device="cuda")
    outs = []
    for at in (0, slot):
        S, n, m = (torch.zeros(slot + 1, *shape, device="cuda") for shape in ((d, dv), (d,), ()))
        out, tok_slot = torch.full((T, dv), float("nan"), device="cuda"), torch.full((T,), at, dtype=torch.int32, device="cuda")
        assert lib.tgis_k_outer_scan(1, _p(y), _p(y[:, d:]), _p(y[:, 2 * d:]), width, width, width, ctypes.c_float(1.0), None, 0, None, None,
                                     _p(y[:, width - 2:]), _p(y[:, width - 1:]), width, _p(bias), _p(bias), ctypes.c_float(6.0), _p(S), _p(n), _p(m), _p(out), dv, 1, d, dv,
                                     None, None, 0, (ctypes.c_int32 * 4)(0, T, T, 0), 1, _p(tok_slot)) == 0
        outs += [out, S[at].clone(), n[at].clone(), m[at].clone()]
        assert int(S[at].count_nonzero()) == int(S.count_nonzero()) > 0
    assert all(torch.equal(a, b) for a, b in zip(outs[:4], outs[4:])) and bool(outs[0].isfinite().all())
