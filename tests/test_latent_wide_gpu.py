"""Latent attention of prompts, several tiles of a sequence per CTA (csrc/attention_latent.cu latent_attn_wide_kernel): token
counts off the four-tile groups, contexts off the cache blocks, head counts that fill a tile, divide it or need two groups, row
lengths with k padding, windows -- against a dense softmax in 64 bits over the same bf16 operands."""
import ctypes as C

import pytest
import torch

from vllm_tgis_adapter_b200.engine._lib import TgisKLatentGeom, load_library

pytestmark = pytest.mark.gpu


def p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("window", [0, 50])
@pytest.mark.parametrize("heads,kv_rank,rot_dim", [(16, 512, 64), (8, 256, 64), (20, 128, 16), (6, 136, 8), (3, 72, 8), (33, 64, 0)])
@pytest.mark.parametrize("o_dt", [0, 1])
def test_prompts_match_dense_softmax(heads, kv_rank, rot_dim, window, o_dt):
    gen = torch.Generator(device="cuda").manual_seed(heads * 1000 + kv_rank)
    D = kv_rank + rot_dim
    shapes = [(0, 211), (37, 150), (64, 97), (31, 130), (0, 33)]   # (tokens already in the cache, tokens of this step)
    T, scale = sum(n for _, n in shapes), D ** -0.5
    n_blocks = sum(-(-(c + n) // 32) for c, n in shapes)
    cache = (torch.randn(n_blocks, 32, D, generator=gen, device="cuda") * 1.5).bfloat16()
    q = torch.randn(T, heads, D, generator=gen, device="cuda") * 2
    order, at, row = torch.randperm(n_blocks, generator=torch.Generator().manual_seed(1)).tolist(), 0, 0
    stride = max(-(-(c + n) // 32) for c, n in shapes)
    table, seqs, want, slack = [], [], torch.empty(T, heads, kv_rank, dtype=torch.float64, device="cuda"), torch.empty(T, heads, kv_rank, dtype=torch.float64, device="cuda")
    for i, (c, n) in enumerate(shapes):
        nb = -(-(c + n) // 32)
        blocks = order[at: at + nb]
        at += nb
        table += blocks + [0] * (stride - nb)
        seqs += [row, n, c + n, i]
        k = cache[blocks].reshape(-1, D)[: c + n].double()
        s = torch.einsum("qhd,kd->qhk", (q[row: row + n] * scale).bfloat16().double(), k)
        dist = torch.arange(c, c + n, device="cuda")[:, None] - torch.arange(c + n, device="cuda")[None, :]
        hidden = (dist < 0) | ((dist >= window) if window else (dist < 0))
        w = torch.softmax(s.masked_fill(hidden[:, None], -float("inf")), -1)
        want[row: row + n] = torch.einsum("qhk,kd->qhd", w, k[:, :kv_rank])
        # softmax weights are rounded to bf16 (2^-8 each); scores are fp32 sums of D products (D / 16 roundings of at most 60)
        slack[row: row + n] = (2.0 ** -8 + 5e-4) * torch.einsum("qhk,kd->qhd", w, k[:, :kv_rank].abs())
        row += n
    out = torch.full((T + 1, heads, kv_rank), 7.0, device="cuda", dtype=torch.bfloat16 if o_dt else torch.float32)
    geom = TgisKLatentGeom(heads=heads, dim=8, rot_dim=rot_dim, vdim=8, kv_rank=kv_rank, q_rank=8, window=window, rot_dims=0, scale=scale)
    assert load_library().tgis_k_latent_attn(p(q), p(cache), 1, (C.c_int32 * len(seqs))(*seqs), len(shapes), (C.c_int32 * len(table))(*table), len(shapes),
                                             stride, p(out), o_dt, C.byref(geom)) == 0
    tol = slack + 1e-5 + (2.0 ** -8 * want.abs() if o_dt else 0)
    over = (out[:T].double() - want).abs() - tol
    assert float(over.max()) <= 0, (float(over.max()), float((over > 0).double().mean()))
    assert bool((out[T] == 7.0).all())


@pytest.mark.parametrize("window", [0, 50])
@pytest.mark.parametrize("heads,kv_rank,rot_dim", [(16, 512, 64), (16, 256, 64), (20, 120, 8), (16, 64, 24)])
def test_a_prompt_has_the_same_bits_beside_decoding_requests(heads, kv_rank, rot_dim, window):
    """Alone, a portion's tiles are four and more per sequence and go to the wide kernel; beside many single tokens the step's
    are not, and the same portion goes tile by tile.  Also from the middle of a group of four tiles on."""
    gen = torch.Generator(device="cuda").manual_seed(kv_rank + window)
    D, cached, n, extra = kv_rank + rot_dim, 45, 171, 70
    nb = -(-(cached + n) // 32)
    cache = (torch.randn(nb + extra, 32, D, generator=gen, device="cuda") * 1.5).bfloat16()
    q = torch.randn(n + extra, heads, D, generator=gen, device="cuda") * 2
    geom = TgisKLatentGeom(heads=heads, dim=8, rot_dim=rot_dim, vdim=8, kv_rank=kv_rank, q_rank=8, window=window, rot_dims=0, scale=D ** -0.5)

    def run(q, seqs, table):
        out = torch.full((q.shape[0], heads, kv_rank), 7.0, device="cuda")
        rows, flat = len(seqs), [v for row in table for v in row + [0] * (nb - len(row))]
        assert load_library().tgis_k_latent_attn(p(q), p(cache), 1, (C.c_int32 * (4 * rows))(*[v for s in seqs for v in s]), rows, (C.c_int32 * len(flat))(*flat), rows,
                                                 nb, p(out), 0, C.byref(geom)) == 0
        return out

    blocks = list(range(nb))
    alone = run(q[:n].contiguous(), [(0, n, cached + n, 0)], [blocks])
    company = run(q, [(0, n, cached + n, 0)] + [(n + i, 1, 3 + i % 20, 1 + i) for i in range(extra)], [blocks] + [[nb + i] for i in range(extra)])
    assert torch.equal(alone, company[:n])
    later = run(q[6:n].contiguous(), [(0, n - 6, cached + n, 0)], [blocks])
    assert torch.equal(alone[6:], later)


def test_a_later_block_cannot_reach_a_token():
    """Rows of the next block hold NaN: the tokens before it keep their values, wherever in a group of four the portion begins."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    heads, kv_rank, D, n = 16, 128, 136, 198
    cache = (torch.randn(7, 32, D, generator=gen, device="cuda")).bfloat16()
    q = torch.randn(n, heads, D, generator=gen, device="cuda")
    geom = TgisKLatentGeom(heads=heads, dim=8, rot_dim=8, vdim=8, kv_rank=kv_rank, q_rank=8, window=0, rot_dims=0, scale=D ** -0.5)

    def run():
        out = torch.full((n, heads, kv_rank), 7.0, device="cuda")   # tokens 30 .. 227: groups of four cross the block borders
        assert load_library().tgis_k_latent_attn(p(q), p(cache), 1, (C.c_int32 * 4)(0, n - 6, 30 + n - 6, 0), 1, (C.c_int32 * 7)(*range(7)), 1, 7, p(out), 0, C.byref(geom)) == 0
        return out

    clean = run()
    cache[2] = float("nan")
    dirty = run()
    assert torch.equal(dirty[:34], clean[:34]) and bool(dirty[34: n - 6].isnan().all())   # token 34 is position 64, the first of block 2
