"""Capped attention with 128-wide heads (csrc/attention_capped.cu): the forms whose sizes are known when they are compiled, for tiles of
queries and for single tokens with the heads of a group in the rows, against the oracle, and bit for bit against each other: a row's
bits do not depend on the portion it came in.  Groups of one, four and sixteen heads, block edges, with and without cap and gate scale."""
import pytest
import torch

from test_zz_falerax_gpu import BF16, _cap_weights, _close, _run_capattn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,softcap", [(16, 4, 30.0), (3, 3, 0.0), (16, 1, 8.0), (20, 1, 8.0)])   # (twenty heads a group: no single-token form)
@pytest.mark.parametrize("T", [1, 31, 32, 33, 97, 150])
def test_known_sizes_and_single_tokens(heads, kv_heads, softcap, T):
    from oracle import falerax_oracle as O

    m = dict(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, scale=0.09, softcap=softcap, q_temp=dict(coef=0.3, every=20))
    g = torch.Generator().manual_seed(T)
    wq, wk = 1.0 + 0.2 * torch.randn(128, generator=g), 1.0 + 0.2 * torch.randn(128, generator=g)
    width, w = _cap_weights(m, wq, wk)
    h = torch.randn(T, width, generator=g)
    whole = _run_capattn(h, m, wq, wk, BF16, [T])
    _close(whole, O.capped_attention(h.double(), w, m, 1e-5), 3e-2)   # (bf16 operands, weights and output: the bound of the other shapes)
    for sizes in ([1], [2, 33, 1, 17, 64]):
        assert torch.equal(_run_capattn(h, m, wq, wk, BF16, sizes), whole)
