"""The sampler's random draw at the end of its range, and rows with entries that are no numbers (csrc/sampler.cu, oracle/sampler_oracle.py).

u = (24 bits + 1/2) / 2^24 has to stay below one: 2^24 - 1/2 is no fp32 number, and an entry with u = 1 would win whatever its probability.
The places below are where the generator's 24 bits are all ones; the entry there is one that e^10 times likelier ones surround."""
import numpy as np
import pytest
import torch

import tgis_gpu_utils as U
from oracle import sampler_oracle as so

ALL_ONES = [(1024, 45, 174, 140), (1024, 148, 15, 222), (128256, 192, 0, 100010), (50272, 404, 0, 28925)]   # vocabulary, seed, step, index


def unlikely(V, index):
    logits = torch.zeros(V)
    logits[index] = -10.0
    return logits


@pytest.mark.parametrize("V,seed,step,index", ALL_ONES)
def test_the_oracles_u_is_below_one(V, seed, step, index):
    u = so.philox_uniform(V, seed, step)
    assert u.dtype == np.float32 and 0 < u.min() and u.max() < 1 and u[index] == np.float32(1) - np.float32(2.0 ** -24) == u.max()
    case = so.SamplingCase(greedy=False, seed=seed, n_out=step)
    assert so.sample_row(unlikely(V, index), case)["token"] != index


@pytest.mark.gpu
@pytest.mark.parametrize("cluster", ["1", "8"])
@pytest.mark.parametrize("how", ["plain", "top_k", "typical"])   # (the race over all entries, over kept ones, over a list of what is left)
@pytest.mark.parametrize("V,seed,step,index", ALL_ONES)
def test_an_unlikely_entry_is_not_drawn_for_its_place(V, seed, step, index, how, cluster, monkeypatch):
    monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
    logits = unlikely(V, index)
    r = np.zeros(1, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"], r["seed_lo"], r["step"] = 1.0, 1.0, 1.0, -1, -1, seed, step
    if how == "top_k":
        r["top_k"], logits[0] = V - 1, -20.0      # (all but entry 0, which is less likely still)
    if how == "typical":
        r["typical_p"], r["flags"] = 1.0, U.SAMPLE_TYPICAL   # (the whole mass: every entry that has some)
    out = U.run_sampler(logits.unsqueeze(0).cuda(), r)
    want = so.sample_row(logits, so.SamplingCase(greedy=False, seed=seed, n_out=step, top_k=int(r["top_k"][0])))["token"]
    assert want != index and int(out["token"][0]) == want


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["plain", "typical"])
@pytest.mark.parametrize("V", [8, 1024])
def test_an_entry_that_is_no_number_is_not_drawn(V, how):
    """It compares with nothing, so it is not among those at or above a threshold: by the sweep over all entries and by the list alike."""
    rows = 64
    logits, at = torch.zeros(rows, V), torch.arange(rows) % V
    logits[torch.arange(rows), at] = float("nan")
    r = np.zeros(rows, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"] = 1.0, 1.0, 1.0, -1, -1
    r["logits_row"], r["seed_lo"] = np.arange(rows), 7 + np.arange(rows)
    if how == "typical":
        r["typical_p"], r["flags"] = 0.9, U.SAMPLE_TYPICAL
    token = U.run_sampler(logits.cuda(), r)["token"]
    assert ((token >= 0) & (token < V) & (token != at.numpy())).all()


@pytest.mark.gpu
@pytest.mark.parametrize("top_p", [1.0, 0.9])
@pytest.mark.parametrize("V,dtype", [(1024, torch.float32), (50272, torch.bfloat16), (50272, torch.float32)])
def test_entries_that_are_no_numbers_are_not_among_the_k_largest(V, dtype, top_p):
    """Every other entry a NaN, of either sign: what is drawn is one of the six largest numbers."""
    gen = torch.Generator().manual_seed(V)
    logits = torch.randn(16, V, generator=gen)
    logits[:, ::2] = float("nan")
    logits[8:, ::2] = -logits[8:, ::2]
    logits = logits.to(dtype)
    r = np.zeros(16, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["top_k"], r["rep_penalty"], r["eos_id"], r["seq_slot"] = 1.0, top_p, 6, 1.0, -1, -1
    r["logits_row"], r["seed_lo"] = np.arange(16), 7 + np.arange(16)
    token = torch.from_numpy(U.run_sampler(logits.cuda(), r)["token"].astype(np.int64))
    numbers = torch.where(logits.isnan(), torch.full_like(logits, -100.0), logits).float()
    assert (numbers[torch.arange(16), token] >= torch.topk(numbers, 6).values[:, -1]).all()
