"""Scans over portions of several tokens: what a portion leaves and answers has the bits of its tokens one launch each (the kernels of
single tokens), for lengths around the staged chunks, sequences of unequal length, columns that fill no whole piece, and rows that 16-byte
loads reach and do not reach."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
F = C.c_float


def p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.fixture(scope="module")
def lib():
    from vllm_tgis_adapter_b200.engine._lib import load_library

    return load_library()


def _runs(lengths, one_by_one):
    """Launches of (first row, tokens, context with them, table row) for sequences that begin at position 0, 3, 6, ..."""
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    if not one_by_one:
        return [[(starts[i], n, 3 * i + n, 0) for i, n in enumerate(lengths)]]
    return [[(starts[i] + t, 1, 3 * i + t + 1, 0) for i, n in enumerate(lengths) if t < n] for t in range(max(lengths))]


@pytest.mark.parametrize("lengths", [[1, 2, 15], [16, 17, 3, 33], [47, 64], [5] * 9])
@pytest.mark.parametrize("d,dv,H", [(64, 64, 3), (128, 256, 2), (128, 40, 1), (256, 33, 1)])
@pytest.mark.parametrize("mode", ["decay", "gated", "hgrn", "ssd", "lightning"])
@pytest.mark.parametrize("odd", [0, 1, 2])
def test_memories(lib, mode, d, dv, H, lengths, odd):
    n, T, res = len(lengths), sum(lengths), []
    for one_by_one in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(d + dv + T)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
        x = rnd(T, -(-(3 * H * d + H * dv + 2 * H) // 4) * 4 + odd)
        ld, q, k, dec, v, gate = x.shape[1], x, x[:, H * d:], x[:, 2 * H * d:], x[:, 3 * H * d:], x[:, 3 * H * d + H * dv:]
        S, nrm, mx = rnd(n, H, d, dv), rnd(n, H, d).abs(), rnd(n, H)
        w0, u, b1, b2, last, heads = rnd(H * d), rnd(H * d).sigmoid(), rnd(H), rnd(H), torch.zeros(n, 24, device="cuda"), rnd(H).sigmoid()
        out = torch.full((T, H * dv), float("nan"), device="cuda")
        slots = torch.cat([torch.full((m,), n - 1 - i, dtype=torch.int32, device="cuda") for i, m in enumerate(lengths)])
        for run in _runs(lengths, one_by_one):
            meta = [e for s in run for e in s]
            seqs = (C.c_int32 * len(meta))(*meta)
            if mode in ("decay", "gated", "hgrn"):
                rc = lib.tgis_k_outer_scan({"decay": 0, "gated": 1, "hgrn": 3}[mode], p(q), p(k), p(v), ld, ld, ld, F(d ** -0.5), p(dec), ld, p(w0), p(u), p(gate),
                                           p(gate[:, H:]), ld, p(b1), p(b2), F(6.0), p(S), p(nrm), p(mx), p(out), H * dv, H, d, dv, p(x), p(last), 24, seqs, len(run), p(slots))
            elif mode == "ssd":
                rc = lib.tgis_k_ssd_scan(p(q), p(k), p(v), ld, ld, ld, p(gate), ld, p(b1), p(b2), p(heads), p(S), p(out), H * dv, H, 1, d, dv, seqs, len(run), p(slots))
            else:
                rc = lib.tgis_k_lightning_scan(p(q), p(k), p(v), ld, ld, ld, p(heads), p(S), p(out), H * dv, H, d, dv, seqs, len(run), p(slots), 0)
            assert rc == 0
        res.append([out, S, nrm, mx, last])
    assert not res[0][0].isnan().any() and res[0][0].abs().max() > 0
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lengths", [[1, 2, 7], [8, 9, 3, 25], [40, 64], [5] * 70])
@pytest.mark.parametrize("inner,N", [(64, 16), (100, 16), (40, 7)])
def test_selective_scan(lib, inner, N, lengths):
    n, T, taps, R, res = len(lengths), sum(lengths), 4, 8, []
    for one_by_one in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(inner + N + T)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
        xz, proj, dt, xc = rnd(T, 2 * inner), rnd(T, R + 2 * N), rnd(T, inner), rnd(T, inner)
        dtb, A, Dv, S, conv = rnd(inner) - 2, rnd(inner, N) * 0.5, rnd(inner), rnd(n, inner, N), rnd(n, taps - 1, inner)
        out = torch.full((T, inner), float("nan"), device="cuda")
        slots = torch.cat([torch.full((m,), n - 1 - i, dtype=torch.int32, device="cuda") for i, m in enumerate(lengths)])
        for run in _runs(lengths, one_by_one):
            meta = [e for s in run for e in s]
            assert lib.tgis_k_selective_scan(p(xc), p(xz), 2 * inner, p(proj), R + 2 * N, R, p(dt), p(dtb), p(A), p(Dv), p(S), p(conv), p(out), 0, inner, N, taps,
                                             (C.c_int32 * len(meta))(*meta), len(run), p(slots)) == 0
        res.append([out, S, conv])
    assert not res[0][0].isnan().any()
    for a, b in zip(*res):
        assert torch.equal(a, b)
