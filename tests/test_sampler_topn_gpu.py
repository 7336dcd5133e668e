"""The sampler's top-n (csrc/sampler.cu) where its candidate list is at an edge: all logits equal or more ties than the list
holds, the largest entries all in one thread's or one slice's share, every cluster size, and n from one to twelve -- in order
of value, then of index, exactly as a sort gives them."""
import numpy as np
import pytest
import torch

import tgis_gpu_utils as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 40, 80, 150])
@pytest.mark.parametrize("V,dtype", [(8, torch.float32), (1024, torch.bfloat16), (128256, torch.bfloat16), (50272, torch.float32)])
def test_topn_is_a_sort(rows, V, dtype):
    gen = torch.Generator().manual_seed(V + rows)
    logits = torch.randn(rows, V, generator=gen)
    for i in range(rows):
        kind = i % 6
        if kind == 1:
            logits[i] = 0.5                                      # all equal
        elif kind == 2:
            logits[i] = (logits[i] > 0).float()                  # half of them tied at the top
        elif kind == 3:
            logits[i, V // 2: V // 2 + 8] += 9.0                 # one thread's group of eight holds the largest
        elif kind == 4:
            logits[i, : max(8, V // 9)] += 9.0                   # one slice does
        elif kind == 5:
            logits[i, 3:] = -float("inf")                        # three entries left
    logits = logits.to(dtype)
    r = np.zeros(rows, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"] = 1.0, 1.0, 1.0, -1, -1
    r["logits_row"] = np.arange(rows)
    r["flags"] = U.SAMPLE_GREEDY | U.SAMPLE_LOGPROBS
    r["n_topn"] = [1 + i % 12 if V > 8 else 1 + i % 8 for i in range(rows)]
    out = U.run_sampler(logits.cuda(), r)
    for i in range(rows):
        x = logits[i].double()
        order = sorted(range(V), key=lambda j: (-float(x[j]), j))[:12] if V <= 1024 else torch.sort(x, descending=True, stable=True).indices[:12].tolist()
        n = int(r["n_topn"][i])
        assert out["topn_ids"][i][:n].tolist() == order[:n], i
        assert out["token"][i] == order[0]
        lp = torch.log_softmax(x, -1)[order[:n]].numpy()
        got = out["topn_lps"][i][:n]
        same = np.isinf(lp)
        assert np.array_equal(np.isinf(got), same)
        np.testing.assert_allclose(got[~same], lp[~same], atol=2e-4)
        assert out["rank"][i] == int((x >= x[order[0]]).sum())
