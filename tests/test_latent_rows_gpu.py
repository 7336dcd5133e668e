"""Latent attention of fp32 prompts, two or four tiles of a sequence per CTA (csrc/attention_latent.cu latent_attn_rows_kernel): against a
dense softmax in 64 bits, and the same bits as tile by tile, wherever a portion begins in a group."""
import ctypes as C

import pytest
import torch

from vllm_tgis_adapter_b200.engine._lib import TgisKLatentGeom, load_library

pytestmark = pytest.mark.gpu
GEOMS = [(16, 512, 64), (8, 256, 64), (20, 128, 16), (6, 136, 12), (3, 72, 8), (33, 64, 0)]


def p(t):
    return C.c_void_p(t.data_ptr())


def _attend(q, cache, seqs, table, geom, o_dt=0):
    out = torch.full((q.shape[0] + 1, geom.heads, geom.kv_rank), 7.0, device="cuda", dtype=torch.bfloat16 if o_dt else torch.float32)
    stride = max(len(r) for r in table)
    flat = [v for r in table for v in r + [0] * (stride - len(r))]
    assert load_library().tgis_k_latent_attn(p(q), p(cache), 0, (C.c_int32 * (4 * len(seqs)))(*[v for s in seqs for v in s]), len(seqs),
                                             (C.c_int32 * len(flat))(*flat), len(table), stride, p(out), o_dt, C.byref(geom)) == 0
    assert bool((out[-1] == 7.0).all())
    return out[:-1]


def _geom(heads, kv_rank, rot_dim, window):
    return TgisKLatentGeom(heads=heads, dim=8, rot_dim=rot_dim, vdim=8, kv_rank=kv_rank, q_rank=8, window=window, rot_dims=0, scale=(kv_rank + rot_dim) ** -0.5)


@pytest.mark.parametrize("window", [0, 50])
@pytest.mark.parametrize("heads,kv_rank,rot_dim", GEOMS)
@pytest.mark.parametrize("o_dt", [0, 1])
def test_prompts_match_dense_softmax(heads, kv_rank, rot_dim, window, o_dt):
    gen = torch.Generator(device="cuda").manual_seed(heads * 1000 + kv_rank)
    D, shapes = kv_rank + rot_dim, [(0, 211), (37, 150), (64, 97), (31, 130), (0, 33)]
    T, geom = sum(n for _, n in shapes), _geom(heads, kv_rank, rot_dim, window)
    nb = [-(-(c + n) // 32) for c, n in shapes]
    cache, q = torch.randn(sum(nb), 32, D, generator=gen, device="cuda") * 1.5, torch.randn(T, heads, D, generator=gen, device="cuda") * 2
    order, at, row, table, seqs = torch.randperm(sum(nb), generator=torch.Generator().manual_seed(1)).tolist(), 0, 0, [], []
    want = torch.empty(T, heads, kv_rank, dtype=torch.float64, device="cuda")
    size = torch.empty_like(want)
    for i, (c, n) in enumerate(shapes):
        table.append(order[at: at + nb[i]])
        seqs.append((row, n, c + n, i))
        k = cache[table[-1]].reshape(-1, D)[: c + n].double()
        s = torch.einsum("qhd,kd->qhk", q[row: row + n].double() * geom.scale, k)
        dist = torch.arange(c, c + n, device="cuda")[:, None] - torch.arange(c + n, device="cuda")[None, :]
        w = torch.softmax(s.masked_fill(((dist < 0) | ((dist >= window) if window else (dist < 0)))[:, None], -float("inf")), -1)
        want[row: row + n], size[row: row + n] = torch.einsum("qhk,kd->qhd", w, k[:, :kv_rank]), torch.einsum("qhk,kd->qhd", w, k[:, :kv_rank].abs())
        at, row = at + nb[i], row + n
    out = _attend(q, cache, seqs, table, geom, o_dt)
    # scores of up to ~60 from chains of D fp32 multiply-adds: D 2^-24 of their absolute terms (below 30 in the mean), into the exponent
    tol = (2.0 ** -24 * (D * 30 + 400)) * size + (2.0 ** -8 * want.abs() if o_dt else 0) + 1e-7
    assert float(((out.double() - want).abs() - tol).max()) <= 0


@pytest.mark.parametrize("window", [0, 50])
@pytest.mark.parametrize("heads,kv_rank,rot_dim", GEOMS)
@pytest.mark.parametrize("n", [171, 1250])   # (1250: four tiles a CTA, two behind some heads' tiles)
def test_a_prompt_has_the_same_bits_tile_by_tile(heads, kv_rank, rot_dim, window, n):
    """Alone a portion goes to the rows kernel; beside many single tokens the same portion goes tile by tile.  Also from the middle of a group."""
    gen = torch.Generator(device="cuda").manual_seed(kv_rank + window)
    D, cached, extra = kv_rank + rot_dim, 45, n + 10
    nb = -(-(cached + n) // 32)
    cache, q = torch.randn(nb + 8, 32, D, generator=gen, device="cuda") * 1.5, torch.randn(n + extra, heads, D, generator=gen, device="cuda") * 2
    geom, blocks = _geom(heads, kv_rank, rot_dim, window), list(range(nb))
    alone = _attend(q[:n].contiguous(), cache, [(0, n, cached + n, 0)], [blocks], geom)
    company = _attend(q, cache, [(0, n, cached + n, 0)] + [(n + i, 1, 3 + i % 20, 1 + i % 8) for i in range(extra)], [blocks] + [[nb + i] for i in range(8)], geom)
    assert torch.equal(alone, company[:n])
    assert torch.equal(alone[6:], _attend(q[6:n].contiguous(), cache, [(0, n - 6, cached + n, 0)], [blocks], geom))


def test_hidden_rows_of_any_value_are_left_out():
    """What lies behind a token in the cache, in its own block too, does not reach it."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    heads, kv_rank, n = 8, 128, 198
    geom, D = _geom(heads, kv_rank, 8, 0), kv_rank + 8
    cache, q = torch.randn(7, 32, D, generator=gen, device="cuda"), torch.randn(n, heads, D, generator=gen, device="cuda")
    run = lambda: _attend(q, cache, [(0, n, 26 + n, 0)], [list(range(7))], geom)   # tokens at positions 26 .. 223
    clean = run()
    cache[2, 7:] = float("nan")   # positions 71 on
    dirty = run()
    assert torch.equal(dirty[:45], clean[:45]) and bool(dirty[45:].isnan().all())


@pytest.mark.parametrize("n", [171, 1250])
def test_a_key_of_no_weight_leaves_no_trace(n):
    """A key whose scores are all minus infinity has a weight of zero and is left out, whatever its values are: alone and tile by tile."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    heads, kv_rank, cached, extra = 8, 128, 45, n + 10
    geom, D, nb = _geom(heads, kv_rank, 8, 0), kv_rank + 8, -(-(45 + n) // 32)
    cache, q = torch.randn(nb + 8, 32, D, generator=gen, device="cuda"), torch.randn(n + extra, heads, D, generator=gen, device="cuda")
    q[..., 0] = -q[..., 0].abs() - 0.1
    k = cache[:nb].reshape(-1, D).double()
    cache[0, 17, 0] = cache[1, 3, 0] = float("inf")   # positions 17 and 35, every token's past
    s = torch.einsum("qhd,kd->qhk", q[:n].double() * geom.scale, k)
    hidden = torch.arange(nb * 32, device="cuda")[None, :] > torch.arange(cached, cached + n, device="cuda")[:, None]
    hidden[:, [17, 35]] = True
    want = torch.einsum("qhk,kd->qhd", torch.softmax(s.masked_fill(hidden[:, None], -float("inf")), -1), k[:, :kv_rank])
    alone = _attend(q[:n].contiguous(), cache, [(0, n, cached + n, 0)], [list(range(nb))], geom)
    assert ((alone.double() - want).abs() <= 2.0 ** -24 * (D * 30 + 400) * (want.abs() + 1)).all()
    company = _attend(q, cache, [(0, n, cached + n, 0)] + [(n + i, 1, 3 + i % 10, 1 + i % 8) for i in range(extra)], [list(range(nb))] + [[nb + i] for i in range(8)], geom)
    assert torch.equal(alone, company[:n])
