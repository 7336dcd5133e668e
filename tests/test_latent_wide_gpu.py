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
