"""The sampler's selections (csrc/sampler.cu) at the edges of what they list: typical-p, top-k and top-p over rows where the entries of
one step of the first sweep are none, a few, or more than the list holds (all equal, two values, a fine ramp), rows masked to a few
tokens, at cluster sizes one to eight.  With one seed the kept set is known in fp64 but for entries at the threshold itself, and the race
over it has one winner."""
import numpy as np
import pytest
import torch

import tgis_gpu_utils as U

pytestmark = pytest.mark.gpu


def kept_typical(x, p, slack):
    """Those surely kept and those surely not: with the mass reached `slack` sooner or later, and keys closer than `slack` alike."""
    lp = torch.log_softmax(x, -1)
    pr = lp.exp()
    ent = -(torch.where(pr > 0, pr * lp, torch.zeros_like(lp))).sum()
    key = (-lp - ent).abs()
    order = torch.argsort(key)
    cum = pr[order].cumsum(0)
    at = lambda t: key[order[min(int((cum < t).sum()), len(x) - 1)]]  # noqa: E731
    return key <= at(p - slack) - slack, key > at(p + slack) + slack


def rows_of_all_kinds(rows, V):
    gen = torch.Generator().manual_seed(V)
    logits = torch.randn(rows, V, generator=gen)
    for i in range(rows):
        kind = i % 6
        if kind == 1:
            logits[i] = 0.5                                      # one key for all
        elif kind == 2:
            logits[i] = (logits[i] > 0).float() * 2.0            # two
        elif kind == 3:
            logits[i] = torch.linspace(0.0, 1e-3, V)             # more entries to a step than the list holds
        elif kind == 4:
            logits[i, 7 * i] += 18.0                             # one entry is all there is
        elif kind == 5:
            logits[i, 3:] = -float("inf")
    return logits


@pytest.mark.parametrize("cluster", ["1", "2", "4", "8"])
@pytest.mark.parametrize("V,dtype", [(1024, torch.float32), (50272, torch.float32), (128256, torch.bfloat16)])
def test_typical_rows_keep_what_sorting_keeps(V, dtype, cluster, monkeypatch):
    monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
    rows = 12
    logits = rows_of_all_kinds(rows, V).to(dtype)
    r = np.zeros(rows, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"] = 1.0, 1.0, 1.0, -1, -1
    r["logits_row"], r["typical_p"], r["flags"] = np.arange(rows), 0.6, U.SAMPLE_TYPICAL | U.SAMPLE_LOGPROBS
    seen = []
    for seed in range(8):
        r["seed_lo"] = 100 + seed
        seen.append(U.run_sampler(logits.cuda(), r)["token"].copy())
    for i in range(rows):
        x = logits[i].double()
        # keys are differences of fp32 numbers up to 20: 4 ulp of that; masses are summed in steps of 2^-30
        sure, never = kept_typical(x, 0.6, 1e-5)
        for tokens in seen:
            assert not bool(never[tokens[i]]), (i, int(tokens[i]))
        if int((~never).sum()) == 1:
            assert all(t[i] == int(torch.nonzero(~never)) for t in seen)
        elif int(sure.sum()) > 100:
            assert len({int(t[i]) for t in seen}) > 1


@pytest.mark.parametrize("cluster", ["1", "2", "4", "8"])
@pytest.mark.parametrize("V,dtype", [(1024, torch.float32), (50272, torch.float32), (128256, torch.bfloat16)])
def test_top_k_and_top_p_keep_what_sorting_keeps(V, dtype, cluster, monkeypatch):
    """At temperature one the k-th largest logit is exact; the mass below top-p's threshold is known to 1e-5 (steps of 2^-30 an entry,
    expf to 2 ulp).  Rows with fewer than k entries left keep them all."""
    monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
    rows, k, p = 18, 50, 0.7
    logits = rows_of_all_kinds(rows, V).to(dtype)
    r = np.zeros(rows, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["rep_penalty"], r["eos_id"], r["seq_slot"] = 1.0, 1.0, -1, -1
    r["logits_row"] = np.arange(rows)
    r["top_k"] = [k if i // 6 != 1 else 0 for i in range(rows)]
    r["top_p"] = [p if i // 6 != 0 else 1.0 for i in range(rows)]
    seen = []
    for seed in range(8):
        r["seed_lo"] = 100 + seed
        seen.append(U.run_sampler(logits.cuda(), r)["token"].copy())
    for i in range(rows):
        x = logits[i].double()
        left = x > -float("inf")
        if r["top_k"][i]:
            left &= x >= torch.sort(x, descending=True).values[k - 1]
        never = ~left
        if r["top_p"][i] < 1:
            pr = torch.softmax(torch.where(left, x, torch.full_like(x, -float("inf"))), -1)
            order = torch.argsort(x)
            cum = pr[order].cumsum(0)
            thr = x[order[min(int((cum <= 1 - p - 1e-5).sum()), V - 1)]]     # entries below it are out whatever rounds how
            never |= x < thr
        assert not any(bool(never[t[i]]) for t in seen), i
        if int((~never).sum()) == 1:
            assert all(t[i] == int(torch.nonzero(~never)) for t in seen)
        elif float(torch.softmax(torch.where(never, torch.full_like(x, -float("inf")), x), -1).max()) < 0.1:   # (not eight times the same)
            assert len({int(t[i]) for t in seen}) > 1


@pytest.mark.parametrize("V,dtype", [(8, torch.float32), (50272, torch.float32), (128256, torch.bfloat16)])
def test_tokens_and_probabilities_at_every_cluster_size(V, dtype, monkeypatch):
    """Integer masses and a fixed order make a row's token the same however it is split; its log probability is the same sum in
    another order (2e-5: 2^-24 of a term, 32 partial sums a thread and five levels of combining)."""
    rows = 16
    gen = torch.Generator().manual_seed(V)
    logits = (torch.randn(rows, V, generator=gen) * 3).to(dtype)
    r = np.zeros(rows, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"] = 0.9, 1.0, 1.0, -1, -1
    r["logits_row"], r["seed_lo"] = np.arange(rows), 5 + np.arange(rows)
    r["flags"] = [(0, U.SAMPLE_GREEDY)[i % 2] | U.SAMPLE_LOGPROBS for i in range(rows)]
    r["top_k"] = [(0, 0, 5, 0)[i % 4] for i in range(rows)]
    outs = []
    for cluster in ("1", "2", "4", "8"):
        monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
        outs.append(U.run_sampler(logits.cuda(), r))
    for o in outs:
        assert np.array_equal(o["token"], outs[0]["token"]) and np.array_equal(o["rank"], outs[0]["rank"])
        want = torch.log_softmax(logits.double(), -1)[torch.arange(rows), torch.from_numpy(o["token"].astype(np.int64))].numpy()
        np.testing.assert_allclose(o["logprob"], want, atol=2e-5)
