"""Attention of prompts on tcgen05 (csrc/attention_prefill.cu) where its tiles end: query tokens around the rows of one and of two
accumulators (128 / G and twice that), contexts around the 32-token blocks and the 128-token tiles, every group size -- against a
softmax in 64 bits over the same bf16 operands; and the bits of a row, which depend on its own keys alone."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    from tests import tgis_gpu_utils

    return tgis_gpu_utils


class Case:
    def __init__(self, g, n_q, n_kv, kv_lens, seed, size=1.0):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        self.g, self.n_q, self.n_kv, self.kv_lens = g, n_q, n_kv, kv_lens
        blocks = [-(-n // 32) for n in kv_lens]
        order = np.random.RandomState(seed).permutation(sum(blocks)).astype(np.int32)   # scattered physical blocks
        self.bt = np.zeros((len(kv_lens), max(blocks)), dtype=np.int32)
        rows = sum(blocks) * 32
        self.k, self.v = ((torch.randn(rows, n_kv, 128, device="cuda", generator=gen)).bfloat16() for _ in range(2))
        self.q = [(torch.randn(n, n_q, 128, device="cuda", generator=gen) * size).bfloat16() for n in kv_lens]
        self.slots, at = [], 0
        for i, (n, b) in enumerate(zip(kv_lens, blocks)):
            self.bt[i, :b] = order[at: at + b]
            at += b
            self.slots.append(torch.tensor(np.concatenate([np.arange(32) + 32 * x for x in self.bt[i, :b]])[:n], device="cuda"))
        self.kc, self.vc = g.k_cache_from_dense(self.k, sum(blocks)), g.v_cache_from_dense(self.v, sum(blocks))

    def run(self, parts, scale=128 ** -0.5):
        """parts: (sequence, first query position, one past the last); the outputs of one launch, in order"""
        seqs, at, rows = [], 0, []
        for s, a, b in parts:
            seqs.append((at, b - a, b, s))
            rows.append(self.q[s][a:b])
            at += b - a
        qkv = torch.zeros(at, self.n_q + 2 * self.n_kv, 128, dtype=torch.bfloat16, device="cuda")
        qkv[:, : self.n_q] = torch.cat(rows)
        out = torch.full((at, self.n_q, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
        sq, bt, g = np.array(seqs, dtype=np.int32), self.bt, self.g
        rc = g.lib().tgis_k_attention(g.ptr(qkv), g.ptr(self.kc), g.ptr(self.vc), g.i32p(sq.reshape(-1)), len(parts), g.i32p(bt.reshape(-1)),
                                      bt.shape[0], bt.shape[1], g.ptr(out), self.n_q, self.n_kv, C.c_float(scale))
        assert rc == 0, g.kerr()
        return list(out.split([b - a for _, a, b in parts]))

    def exact(self, s, a, b, scale=128 ** -0.5):
        k, v = (t[self.slots[s][:b]].double().repeat_interleave(self.n_q // self.n_kv, 1) for t in (self.k, self.v))
        x = torch.einsum("qhd,khd->hqk", self.q[s][a:b].double(), k) * scale
        x = x.masked_fill(torch.arange(b, device="cuda")[None] > torch.arange(a, b, device="cuda")[:, None], -math.inf)
        return torch.einsum("hqk,khd->qhd", torch.softmax(x, -1), v)


@pytest.mark.parametrize("size,scale", [(1.0, 128 ** -0.5), (6.0, 128 ** -0.5), (1.0, -0.05)])
@pytest.mark.parametrize("n_q,n_kv", [(8, 2), (8, 1), (2, 2), (6, 2), (5, 1), (7, 1), (4, 2)])
def test_tile_edges_match_a_softmax_in_64_bits(g, n_q, n_kv, size, scale):
    tm = 128 * n_kv // n_q // 8 * 8   # query tokens of one accumulator
    parts = [(c, c + q) for c in (0, 31, 97, 128) for q in (2, tm - 1, tm, tm + 1, 2 * tm, 2 * tm + 3)]
    parts += [(0, 127), (0, 128), (0, 129), (0, 257), (300, 384), (511, 641)]
    case = Case(g, n_q, n_kv, [b for _, b in parts], seed=n_q * 10 + n_kv, size=size)
    out = case.run([(s, a, b) for s, (a, b) in enumerate(parts)], scale)
    for s, (a, b) in enumerate(parts):
        want = case.exact(s, a, b, scale)
        # the result's rounding to 8 bits (half a unit in the last place: at most 2^-8 of it); the probabilities' 16 bits (2^-16 of a
        # sum of |v| <= 5); scores of up to 100, summed in fp32 (128 terms: 2^-19 of them, which e^x hands on)
        bound = 1.001 * 2 ** -8 * want.abs() + 5 * (2 ** -16 + 100 * 2 ** -19)
        off = (out[s].double() - want).abs() - bound
        assert float(off.max()) <= 0.0, (s, a, b, float(off.max()))


@pytest.mark.parametrize("n_q,n_kv", [(8, 2), (6, 2), (2, 2)])
def test_a_row_has_the_same_bits_whole_in_portions_and_beside_others(g, n_q, n_kv):
    case = Case(g, n_q, n_kv, [700, 45, 333], seed=3, size=4.0)   # large scores: the running maximum moves often
    whole = case.run([(0, 0, 700)])[0]
    beside = case.run([(1, 0, 45), (0, 0, 700), (2, 100, 333)])[1]
    assert torch.equal(whole, beside)
    cuts = [0, 2, 33, 64, 200, 511, 513, 700]
    portions = torch.cat([case.run([(2, 0, 9), (0, a, b)])[1] for a, b in zip(cuts, cuts[1:])])
    assert torch.equal(whole, portions)


def test_keys_that_score_minus_infinity_weigh_nothing(g):
    """Keys 0 .. 131 score -inf under every query: a whole 128-token tile without a finite score, then part of one."""
    case = Case(g, 8, 2, [300], seed=11)
    case.q[0][..., 0] = case.q[0][..., 0].abs() + 0.125
    case.k[case.slots[0][:132], :, 0] = -math.inf
    case.kc = g.k_cache_from_dense(case.k, case.bt.shape[1])
    want = case.exact(0, 0, 300)
    assert bool(want[:132].isnan().all()) and bool(want[132:].isfinite().all())
    got = case.run([(0, 0, 300)])[0].double()
    assert bool(got[:132].isnan().all())
    bound = 1.001 * 2 ** -8 * want.abs() + 5 * (2 ** -16 + 100 * 2 ** -19)   # as above
    assert float(((got - want).abs() - bound)[132:].max()) <= 0.0


@pytest.mark.parametrize("n_q,n_kv,scale", [(8, 2, 128 ** -0.5), (2, 2, 128 ** -0.5), (8, 1, 128 ** -0.5), (6, 2, -0.05)])
def test_values_that_are_not_finite_reach_only_the_rows_that_see_them(g, n_q, n_kv, scale):
    """Infinities and a NaN in the values of later tokens, and in the cache behind the sequence: a row in front of them is what it is
    without them; a row that sees one has numbers that are not finite in that dim, and its own in the others."""
    case = Case(g, n_q, n_kv, [420], seed=5)
    blocks = case.bt.shape[1]
    k, v = case.slots[0], case.v.clone()
    clean = case.run([(0, 0, 420)], scale)[0]
    bad = ((70, 3, math.inf), (260, 127, -math.inf), (300, 64, math.nan))   # (position, dim, value) in the last kv head
    for t, d, x in bad:
        case.v[k[t], n_kv - 1, d] = x
    case.vc = g.v_cache_from_dense(case.v, blocks)
    behind = case.vc.view(blocks, n_kv, 32, 128)[int(case.bt[0, -1])]        # positions 416 .. 447: four are the sequence's
    behind[:, 4:] = math.inf
    got = case.run([(0, 0, 420)], scale)[0]
    case.v = v
    want = case.exact(0, 0, 420, scale)
    sees = torch.zeros(420, n_q, 128, dtype=torch.bool, device="cuda")
    for t, d, _ in bad:
        sees[t:, n_q - n_q // n_kv:, d] = True
    assert not bool(got[sees].isfinite().any())
    bound = 1.001 * 2 ** -8 * want.abs() + 5 * (2 ** -16 + 100 * 2 ** -19)   # as above
    assert float(((got.double() - want).abs() - bound)[~sees].max()) <= 0.0
    if n_kv > 1:   # the last block reaches the last unit of the other heads alone: the rows in front keep their bits
        first = 420 - 2 * (128 // (n_q // n_kv) // 8 * 8) - 1
        assert torch.equal(got[:first, : n_q // n_kv], clean[:first, : n_q // n_kv])


@pytest.mark.parametrize("n_q,n_kv,scale", [(8, 2, 128 ** -0.5), (8, 1, 128 ** -0.5), (2, 2, 128 ** -0.5), (6, 2, -0.05), (5, 1, 128 ** -0.5)])
def test_few_short_prompts_have_the_bits_of_many(g, n_q, n_kv, scale):
    """Up to 128 keys and no more units than SMs: one accumulator per CTA and rings as long as the longest sequence.  Every length around
    its blocks and rows, alone and two at a time, against 64 bits and against the launch that a longer prompt beside it asks for."""
    parts = [(a, b) for b in (2, 17, 32, 33, 63, 64, 65, 96, 97, 127, 128) for a in (0, 1, 30, 31, 32, 95) if b - a > 1]
    case = Case(g, n_q, n_kv, [b for _, b in parts] + [300], seed=n_q + n_kv, size=3.0)
    beside = case.run([(len(parts), 0, 300)] + [(s, a, b) for s, (a, b) in enumerate(parts)], scale)[1:]
    alone = [case.run([(s, a, b)], scale)[0] for s, (a, b) in enumerate(parts)]
    for s in range(len(parts) - 1):
        alone[s: s + 2] = case.run([(i, *parts[i]) for i in (s, s + 1)], scale) if s % 3 == 0 else alone[s: s + 2]
    for s, (a, b) in enumerate(parts):
        want = case.exact(s, a, b, scale)
        assert torch.equal(alone[s], beside[s]), (a, b)
        bound = 1.001 * 2 ** -8 * want.abs() + 5 * (2 ** -16 + 100 * 2 ** -19)   # as above
        assert float(((alone[s].double() - want).abs() - bound).max()) <= 0.0, (a, b)


def test_a_value_that_is_not_finite_in_a_short_prompt(g):
    case = Case(g, 8, 2, [60], seed=8)
    want = case.exact(0, 0, 60)
    case.v[case.slots[0][40], 0, 9] = math.inf
    case.vc = g.v_cache_from_dense(case.v, case.bt.shape[1])
    got = case.run([(0, 0, 60)])[0].double()
    sees = torch.zeros(60, 8, 128, dtype=torch.bool, device="cuda")
    sees[40:, :4, 9] = True
    bound = 1.001 * 2 ** -8 * want.abs() + 5 * (2 ** -16 + 100 * 2 ** -19)   # as above
    assert not bool(got[sees].isfinite().any()) and float(((got - want).abs() - bound)[~sees].max()) <= 0.0


def test_sums_that_overflow_before_they_are_divided(g):
    """Values near the largest of their type: a row's sum in front of the division may pass it, its result does not."""
    case = Case(g, 8, 2, [200], seed=4)
    case.v = (case.v.sign() * 3e38 * torch.rand(case.v.shape, device="cuda").clamp(min=0.5)).bfloat16()
    case.vc = g.v_cache_from_dense(case.v, case.bt.shape[1])
    want, got = case.exact(0, 0, 200), case.run([(0, 0, 200)])[0].double()
    assert bool(got.isfinite().all())
    assert float(((got - want).abs() - 1.001 * 2 ** -8 * want.abs()).max()) <= 3e38 * (2 ** -16 + 100 * 2 ** -19)
