"""The sampler's selections (csrc/sampler.cu) where the keys of the selected step share digits: all alike, alike but in the first, the
second, the third or the last digit, or in bits of several -- over rows whose entries the selection's list holds and rows it does not."""
import numpy as np
import pytest
import torch

import tgis_gpu_utils as U
from oracle import sampler_oracle as so

pytestmark = pytest.mark.gpu
BITS = [0x00000000, 0x000000FF, 0x0000FF00, 0x007F0000, 0x3F000000, 0x00012001, 0x3F00FF00, 0x000F00F0]


def rows_of(V, many):
    """Row j: numbers near 1.5 that differ in BITS[j] alone, half of the row or a few hundred entries of it."""
    gen, rows = torch.Generator().manual_seed(V), []
    for bits in BITS:
        x = torch.full((V,), -30.0)
        at = torch.randperm(V, generator=gen)[: V // 2 if many else 300]
        x[at] = (0x3FC00000 ^ (torch.randint(0, 1 << 30, (len(at),), generator=gen, dtype=torch.int32) & bits)).view(torch.float32).clamp(max=4.0)
        rows.append(x)
    return torch.stack(rows)


@pytest.mark.parametrize("cluster", ["1", "8"])
@pytest.mark.parametrize("many", [True, False])
@pytest.mark.parametrize("k", [1, 40, 290])
def test_top_k_among_keys_that_share_digits(k, many, cluster, monkeypatch):
    monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
    V, n = 50272, len(BITS)
    logits = rows_of(V, many)
    r = np.zeros(n, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"], r["top_k"], r["logits_row"] = 1.0, 1.0, 1.0, -1, -1, k, np.arange(n)
    for seed in range(3):
        r["seed_lo"] = 50 * seed + np.arange(n)
        token = U.run_sampler(logits.cuda(), r)["token"]
        for i in range(n):
            assert int(token[i]) == so.sample_row(logits[i], so.SamplingCase(greedy=False, top_k=k, seed=50 * seed + i))["token"], (i, seed)


@pytest.mark.parametrize("cluster", ["1", "8"])
@pytest.mark.parametrize("many", [True, False])
@pytest.mark.parametrize("how", ["top_p", "typical"])
def test_masses_among_keys_that_share_digits(how, many, cluster, monkeypatch):
    """The mass in front of a threshold is known to 1e-5 (steps of 2^-30 an entry, expf to 2 ulp), typical-p's distances to 1e-5 (4 ulp of 11)."""
    monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
    V, n, mass, slack = 50272, len(BITS), 0.4, 1e-5
    logits = rows_of(V, many)
    r = np.zeros(n, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"], r["logits_row"] = 1.0, 1.0, 1.0, -1, -1, np.arange(n)
    if how == "top_p":
        r["top_p"] = mass
    else:
        r["typical_p"], r["flags"] = mass, U.SAMPLE_TYPICAL
    never = []
    for x in logits.double():
        lp = torch.log_softmax(x, -1)
        key = -lp if how == "top_p" else (-lp + (lp.exp() * lp).sum()).abs()
        order = torch.argsort(key)
        reached = int((lp.exp()[order].cumsum(0) < mass + slack).sum())
        never.append(key > key[order[min(reached, V - 1)]] + (0 if how == "top_p" else slack))
    for seed in range(6):
        r["seed_lo"] = 50 * seed + np.arange(n)
        token = U.run_sampler(logits.cuda(), r)["token"]
        assert not any(bool(never[i][token[i]]) for i in range(n)), (seed, token)


@pytest.mark.parametrize("cluster", ["1", "4", "8"])
@pytest.mark.parametrize("V,dtype", [(1024, torch.float32), (50272, torch.float32), (128256, torch.bfloat16)])
def test_topn_of_rows_in_order(V, dtype, cluster, monkeypatch):
    """Rows whose largest entries stand side by side, so that few warps have them all: rising, falling, in saw teeth, with ties at the end."""
    monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
    up, rows = torch.linspace(-3, 3, V), []
    for i in range(12):
        rows.append([up, up.flip(0), torch.arange(V) % 2048 / 512.0, torch.arange(V) % 256 / 64.0, up.clamp(max=2.97), (up * 400).round() / 400][i % 6])
    logits = torch.stack(rows).to(dtype)
    r = np.zeros(12, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"], r["logits_row"] = 1.0, 1.0, 1.0, -1, -1, np.arange(12)
    r["flags"], r["n_topn"] = U.SAMPLE_GREEDY | U.SAMPLE_LOGPROBS, 1 + np.arange(12)
    out = U.run_sampler(logits.cuda(), r)
    for i in range(12):
        want = torch.sort(logits[i].double(), descending=True, stable=True).indices
        assert out["topn_ids"][i][: i + 1].tolist() == want[: i + 1].tolist(), i
        assert int(out["token"][i]) == int(want[0])


@pytest.mark.parametrize("cluster", ["1", "4", "8"])
@pytest.mark.parametrize("V", [8, 16, 24, 40, 256, 264, 1024, 1032, 4096])
def test_topn_of_short_rows(V, cluster, monkeypatch):
    """Slices shorter than the list, which few warps sweep: numbers, ties, rows of which all but a few or none are minus infinity."""
    monkeypatch.setenv("TGIS_SAMPLER_CLUSTER", cluster)
    gen, rows, n = torch.Generator().manual_seed(V), 24, min(V, 12)
    logits = torch.randn(rows, V, generator=gen)
    for i in range(rows):
        if i % 4 == 1:
            logits[i] = (logits[i] > 0.5).float()
        elif i % 4 == 2:
            logits[i, torch.randperm(V, generator=gen)[: V - 3]] = -float("inf")
        elif i % 4 == 3:
            logits[i] = logits[i].sort().values
    r = np.zeros(rows, dtype=U.SAMPLE_ROW_DTYPE)
    r["temperature"], r["top_p"], r["rep_penalty"], r["eos_id"], r["seq_slot"], r["logits_row"] = 1.0, 1.0, 1.0, -1, -1, np.arange(rows)
    r["flags"], r["n_topn"] = U.SAMPLE_GREEDY | U.SAMPLE_LOGPROBS, 1 + np.arange(rows) % n
    out = U.run_sampler(logits.cuda(), r)
    for i in range(rows):
        k = int(r["n_topn"][i])
        want = torch.sort(logits[i].double(), descending=True, stable=True).indices[:k]
        assert out["topn_ids"][i][:k].tolist() == want.tolist(), i
        np.testing.assert_allclose(out["topn_lps"][i][:k], torch.log_softmax(logits[i].double(), -1)[want].numpy(), atol=2e-5)
