"""Latent attention of prompts in head space (csrc/attention_heads.cu): against a dense softmax in 64 bits over the keys and values that
the up-projections give, at token counts and contexts off the tiles, with windows, gates and sinks; numbers that are not finite stay with
the rows that see them; an engine whose step mixes such prompts with short portions and single tokens against the oracle."""
import ctypes as C
import dataclasses

import numpy as np
import pytest
import torch

from vllm_tgis_adapter_b200.engine._lib import TgisKLatentGeom, load_library

pytestmark = pytest.mark.gpu
F64 = torch.float64
SHAPES = [(0, 211), (37, 150), (64, 97), (31, 330), (0, 33), (300, 1)]   # (tokens already in the cache, tokens of this step)


def p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


class Case:
    def __init__(self, heads, kv_rank, window=0, scale=192 ** -0.5, rot_dims=64, shapes=SHAPES):
        gen = torch.Generator(device="cuda").manual_seed(heads * 1000 + kv_rank + window)
        rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")
        self.shapes, self.T, self.heads, self.window, self.scale = shapes, sum(n for _, n in shapes), heads, window, scale
        nb = [-(-(c + n) // 32) for c, n in shapes]
        self.cache = (rnd(sum(nb) + 1, 32, kv_rank + 64) * 1.5).bfloat16()
        self.w = (rnd(heads * 256, kv_rank) * kv_rank ** -0.5).bfloat16()
        self.q = (rnd(self.T, heads, 192) * 2).bfloat16()
        self.gate, self.sink = torch.sigmoid(rnd(self.T, heads)), rnd(heads) + 2
        self.pos = torch.cat([torch.arange(c, c + n) for c, n in shapes]).int().cuda()
        angle = torch.rand(4096, rot_dims // 2, generator=gen, device="cuda") * 6
        self.cs = torch.cat([angle.cos(), angle.sin()], 1).contiguous()
        order, at, row, self.blocks, self.seqs, self.stride = torch.randperm(sum(nb), generator=torch.Generator().manual_seed(1)).tolist(), 0, 0, [], [], max(nb)
        for i, (c, n) in enumerate(shapes):
            self.blocks.append(order[at: at + nb[i]])
            self.seqs += [row, n, c + n, i]
            at, row = at + nb[i], row + n
        self.geom = TgisKLatentGeom(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=kv_rank, q_rank=8, window=window, rot_dims=rot_dims, scale=scale)
        first = [max(0, c - window + 1) // 128 * 128 if window else 0 for c, _ in shapes]
        self.first, self.keys = first, [c + n - f for (c, n), f in zip(shapes, first)]

    def run(self, kv=None, gate=True, sink=True):
        q, out = self.q.clone(), torch.full((self.T + 1, self.heads, 128), 7.0, device="cuda", dtype=torch.bfloat16)
        given = kv is not None
        kv = kv if given else torch.empty(sum(self.keys), self.heads * 256, device="cuda", dtype=torch.bfloat16)
        flat = [v for b in self.blocks for v in b + [0] * (self.stride - len(b))]
        rc = load_library().tgis_k_latent_heads(p(q), p(self.cache), None if given else p(self.w), p(self.pos), p(self.cs), p(self.gate) if gate else None,
                                                p(self.sink) if sink else None, (C.c_int32 * len(self.seqs))(*self.seqs), len(self.shapes),
                                                (C.c_int32 * len(flat))(*flat), len(self.shapes), self.stride, p(kv), p(out), C.byref(self.geom))
        assert rc == 0 and bool((out[self.T] == 7.0).all())
        return out[: self.T], kv, q

    def dense(self, kv, q, gate=True, sink=True):
        """From the turned queries and the keys and values as they were made; and what a row's rounding errors scale with."""
        want, size, at, row = torch.empty(self.T, self.heads, 128, dtype=F64, device="cuda"), torch.empty(self.T, self.heads, 128, dtype=F64, device="cuda"), 0, 0
        for i, (c, n) in enumerate(self.shapes):
            k0, rows = self.first[i], self.cache[self.blocks[i]].reshape(-1, self.cache.shape[-1])
            part = kv[at: at + self.keys[i]].double()
            k = torch.cat([part[:, : self.heads * 128].view(-1, self.heads, 128), rows[k0: c + n, None, -64:].double().expand(-1, self.heads, -1)], -1)
            v = part[:, self.heads * 128:].view(-1, self.heads, 128)
            s = torch.einsum("qhd,khd->qhk", q[row: row + n].double(), k) * self.scale
            dist = torch.arange(c, c + n, device="cuda")[:, None] - torch.arange(k0, c + n, device="cuda")[None]
            s = s.masked_fill(((dist < 0) | ((dist >= self.window) if self.window else (dist < 0)))[:, None], -float("inf"))
            if sink:
                s = torch.cat([s, self.sink.double()[None, :, None].expand(n, -1, 1)], -1)
            w = torch.softmax(s, -1)[..., : k.shape[0]] * (self.gate[row: row + n].double()[..., None] if gate else 1)
            want[row: row + n] = torch.einsum("qhk,khd->qhd", w, v)
            size[row: row + n] = torch.einsum("qhk,khd->qhd", w, v.abs())
            at, row = at + self.keys[i], row + n
        return want, size


@pytest.mark.parametrize("window", [0, 50, 200])
@pytest.mark.parametrize("heads,kv_rank,rot_dims", [(16, 512, 64), (8, 256, 32), (3, 64, 64)])
@pytest.mark.parametrize("extras", [False, True])
def test_prompts_match_dense_softmax(heads, kv_rank, rot_dims, window, extras):
    case = Case(heads, kv_rank, window, rot_dims=rot_dims)
    out, kv, q = case.run(gate=extras, sink=extras)
    # keys and values: a product of bf16 operands, rounded once (2^-9) after sums in fp32
    at = 0
    for i, (c, n) in enumerate(case.shapes):
        rows = case.cache[case.blocks[i]].reshape(-1, kv_rank + 64)[case.first[i]: c + n, :kv_rank].double()
        ref = rows @ case.w.double().T
        assert ((kv[at: at + case.keys[i]].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * (rows.abs() @ case.w.double().abs().T)).all()
        at += case.keys[i]
    # the rotary part: fp32 arithmetic, rounded once
    half = rot_dims // 2
    cs, x = case.cs[case.pos.long()].double()[:, None], case.q[..., 128: 128 + rot_dims].double()
    a, b, cos, sin = x[..., :half], x[..., half:], cs[..., :half], cs[..., half:]
    turned = torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    assert ((q[..., 128: 128 + rot_dims].double() - turned).abs() <= 2.0 ** -8 * turned.abs() + 1e-5).all()
    assert torch.equal(q[..., :128], case.q[..., :128]) and torch.equal(q[..., 128 + rot_dims:], case.q[..., 128 + rot_dims:])
    want, size = case.dense(kv, q, extras, extras)
    # weights are rounded to bf16 (2^-9 each), scores are fp32 sums; the result is rounded once
    over = (out.double() - want).abs() - ((2.0 ** -8 + 5e-4) * size + 2.0 ** -8 * want.abs() + 1e-5)
    assert float(over.max()) <= 0, float(over.max())


@pytest.mark.parametrize("scale", [-(192 ** -0.5), 0.0, 3.0])
def test_scales(scale):
    case = Case(2, 64, scale=scale, shapes=[(0, 140), (5, 33)])
    out, kv, q = case.run(gate=False, sink=False)
    want, size = case.dense(kv, q, False, False)
    slack = (2.0 ** -8 + 5e-4 + 1e-6 * abs(scale) * 192 * 30) * size + 2.0 ** -8 * want.abs() + 1e-5
    assert bool(((out.double() - want).abs() <= slack).all())


def test_rows_do_not_depend_on_their_company():
    case = Case(4, 128)
    out = case.run()[0]
    row = 0
    for c, n in case.shapes:
        i = case.shapes.index((c, n))
        alone = Case(4, 128)
        for name in ("q", "gate", "pos"):
            setattr(alone, name, getattr(alone, name)[row: row + n].contiguous())
        alone.shapes, alone.T, alone.seqs, alone.blocks = [(c, n)], n, [0, n, c + n, 0], [case.blocks[i]]
        alone.first, alone.keys = [case.first[i]], [case.keys[i]]
        # (the same keys and values: the product's own order of sums depends on its number of rows)
        kv = case.run()[1][sum(case.keys[:i]): sum(case.keys[: i + 1])].contiguous()
        assert torch.equal(alone.run(kv=kv)[0], out[row: row + n])
        row += n


@pytest.mark.parametrize("window", [0, 60])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_numbers_that_are_not_finite_stay_with_the_rows_that_see_them(window, bad):
    shapes = [(0, 300), (0, 70)]
    case = Case(3, 64, window, shapes=shapes)
    clean, kv, _ = case.run()
    kv2 = kv.clone()
    key, head, dim = 150, 1, 5
    kv2[key, 3 * 128 + head * 128 + dim] = bad          # a value of the first sequence
    dirty = case.run(kv=kv2)[0]
    sees = torch.zeros(370, dtype=torch.bool, device="cuda")
    sees[key: min(300, key + window) if window else 300] = True
    assert not dirty[sees, head, dim].isfinite().any()
    rest = torch.ones_like(dirty, dtype=torch.bool)
    rest[sees, head] = False
    assert dirty[rest].isfinite().all()
    assert ((dirty[rest].double() - clean[rest].double()).abs() <= 2.0 ** -7 * clean[rest].double().abs() + 2e-2).all()   # (some are summed in another order)
    assert torch.equal(dirty[:, 0], clean[:, 0]) and torch.equal(dirty[300:], clean[300:])
    kv2 = kv.clone()
    kv2[300, head * 128 + dim] = bad                    # a key of the second sequence, right behind the first one's last tile
    assert torch.equal(case.run(kv=kv2)[0][:300], clean[:300])


def test_an_engine_mixes_both_forms():
    """Prompts in head space beside short portions and single tokens, in one step and in portions, against the oracle and alone."""
    from oracle import ponenex_oracle as O
    from vllm_tgis_adapter_b200.engine.core import NativeEngine, cache_block_bytes
    from vllm_tgis_adapter_b200.engine.ponenex import PRESETS, synthetic_weights

    base = PRESETS["ponenex-tiny"]
    layers = [dataclasses.replace(base.layers[0], heads=4, dim=128, rot_dim=64, vdim=128, kv_rank=64, rot_dims=64, scale=192 ** -0.5, window=w) for w in (0, 100)]
    layers.append(dataclasses.replace(base.layers[0], window=70))          # (a layer that keeps the folded form)
    mc = dataclasses.replace(base, n_layers=3, layers=layers, max_model_len=512)
    weights = synthetic_weights(mc, 7)
    eng = NativeEngine(mc, max_num_seqs=6, max_batched_tokens=1024, kv_cache_bytes=cache_block_bytes(mc) * 64)
    eng.load_weights(weights)
    gen = torch.Generator().manual_seed(3)
    reqs = {f"q{i}": torch.randint(0, mc.vocab, (n,), generator=gen).tolist() for i, n in enumerate((300, 140, 37, 5, 64))}
    ref = {k: O.forward(mc, weights, t) for k, t in reqs.items()}
    plans = [{k: [len(t)] for k, t in reqs.items()},
             {"q0": [160, 1, 100, 39], "q1": [33, 31, 32, 44], "q2": [1, 35, 1], "q3": [1, 1, 2, 1], "q4": [20, 44]}]
    for plan in plans:
        at, got = {k: 0 for k in reqs}, {k: [] for k in reqs}
        for step in range(max(len(v) for v in plan.values())):
            entries, ends = [], []
            for k, sizes in plan.items():
                if step < len(sizes):
                    n = sizes[step]
                    entries.append((k, reqs[k][at[k]: at[k] + n], list(range(n))))
                    at[k] += n
                    if at[k] == len(reqs[k]):
                        ends.append(k)
            out, o = eng.trace_step(entries, ends), 0
            for k, t, _ in entries:
                got[k].append(out[o: o + len(t)])
                o += len(t)
        for k in reqs:
            d = torch.as_tensor(np.concatenate(got[k])).double() - ref[k]
            d = d - d.mean(-1, keepdim=True)
            rel = d.pow(2).mean(-1).sqrt() / ref[k].std(-1)
            # bf16 weights and activations of three layers; a token whose expert choice falls the other way may be further off
            assert float(rel.median()) < 3e-2, (k, float(rel.median()))
    eng.close()
