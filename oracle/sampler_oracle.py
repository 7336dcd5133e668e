"""CPU oracle for the sampling half of the hot path — TEST INFRASTRUCTURE ONLY (see llama_oracle.py header).

Restates, per request row and in fp32, what the reference stack does between the lm_head logits and the
(token, logprob, rank, top-n) record.  Each function cites what it follows:

  exp_decay_length_penalty  src/vllm_tgis_adapter/tgis_utils/logits_processors.py:33-47   (R7)
  typical_mask              src/vllm_tgis_adapter/tgis_utils/logits_processors.py:11-21   (R8)
                            -> transformers generation/logits_process.py:836-856 (TypicalLogitsWarper.__call__)
  min_tokens                vllm v1/sample/logits_processor/builtin.py:168-240                            (S2)
  repetition_penalty        vllm model_executor/layers/utils.py:51-89, _custom_ops.py:360-408             (S3)
  greedy / temperature      vllm v1/sample/sampler.py:223-236                                             (S4,S5)
  top-k / top-p             vllm v1/sample/ops/topk_topp_sampler.py:328-369                               (S6)
  exponential race          vllm v1/sample/ops/topk_topp_sampler.py:395-416                               (S7)
  logprobs / rank / top-n   vllm v1/sample/sampler.py:79-88,300-351 ; v1/sample/ops/logprobs.py:10-27     (S1,S8)

Processor order is the contract (V0 ordering the adapter was written for):
raw log-softmax -> typical-p -> ExpDecay(EOS, no-op on a non-finite logit) -> min_tokens -> repetition penalty ->
greedy argmax | temperature -> top-k -> top-p -> sample.

PARITY PINNING: the reference's tests never exercise these processors.  tests/golden/sampler_*.json
are generated by oracle/gen_golden.py by running the reference's OWN logits_processors.py (imported from
its source tree), transformers' TypicalLogitsWarper and vLLM 0.22's CPU sampler ops on seeded
logits; tests/test_oracle_cpu.py checks this file against them.

The random draw: torch's Philox stream cannot be reproduced by a custom kernel, so the engine defines
its own counter-based generator (Philox4x32-10 keyed by the request seed, counter = (vocab index, output position)).
`philox_uniform` restates it bit-exactly in numpy so that even sampled tokens can be compared.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch


@dataclasses.dataclass
class SamplingCase:
    greedy: bool = True
    temperature: float = 1.0
    top_k: int = 0            # <= 0 off
    top_p: float = 1.0        # >= 1 off
    typical_p: float = 0.0    # (0,1) on, sampling only
    repetition_penalty: float = 1.0
    length_penalty: tuple[int, float] | None = None   # (start_index, decay_factor)
    eos_token_id: int = 2
    min_tokens: int = 0
    n_out: int = 0            # tokens generated so far (== len(output ids))
    num_logprobs: int = 0     # vLLM `logprobs`
    seed: int = 0


# ---------------------------------------------------------------------------------------------- processors
def typical_keep_mask(logits: torch.Tensor, mass: float) -> torch.Tensor:
    """Boolean keep-mask equal to what TypicalLogitsWarper leaves finite (hf logits_process.py:836-856)."""
    normalized = torch.log_softmax(logits, dim=-1)
    p = torch.exp(normalized)
    ent = -(normalized * p).nansum(-1, keepdim=True)
    shifted = torch.abs((-normalized) - ent)
    sorted_scores, sorted_idx = torch.sort(shifted, descending=False)
    sorted_logits = logits.gather(-1, sorted_idx)
    cum = sorted_logits.softmax(dim=-1).cumsum(dim=-1)
    last_ind = (cum < mass).sum(dim=-1).clamp_(max=sorted_scores.shape[-1] - 1)
    thr = sorted_scores.gather(-1, last_ind.view(-1, 1) if logits.dim() == 2 else last_ind.view(1))
    return ~(shifted > thr)


def exp_decay_length_penalty(logits: torch.Tensor, n_out: int, start: int, decay: float, eos: int) -> None:
    """In place.  logits_processors.py:38-46, plus the no-op-on-non-finite rule."""
    tokens_past = max(0, n_out - start)
    p_factor = pow(decay, tokens_past)          # python float (double)
    if p_factor != 1 and bool(torch.isfinite(logits[eos])):
        eos_logit = logits[eos]
        logits[eos] = eos_logit + torch.abs(eos_logit) * (p_factor - 1)


def apply_repetition_penalty(logits: torch.Tensor, seen: torch.Tensor, penalty: float) -> None:
    """In place; seen = bool mask over vocab of prompt U output ids.  CUDA op semantics
    (vllm csrc sampler: logit > 0 ? logit / penalty : logit * penalty)."""
    pen = torch.tensor(penalty, dtype=torch.float32)
    pos = logits > 0
    upd = torch.where(pos, logits / pen, logits * pen)
    logits.copy_(torch.where(seen, upd, logits))


def process_logits(raw: torch.Tensor, case: SamplingCase, seen: torch.Tensor | None) -> torch.Tensor:
    """Steps 2-5 of the contract on one fp32 row; returns the processed (pre-temperature) logits."""
    y = raw.clone()
    if 0.0 < case.typical_p < 1.0:   # the caller zeroes typical_p for method == GREEDY (grpc_server.py:562-565)
        keep = typical_keep_mask(raw, case.typical_p)
        y = y.masked_fill(~keep, float("-inf"))
    if case.length_penalty is not None:
        exp_decay_length_penalty(y, case.n_out, case.length_penalty[0], case.length_penalty[1], case.eos_token_id)
    if case.n_out < case.min_tokens:
        y[case.eos_token_id] = float("-inf")
    if case.repetition_penalty != 1.0 and seen is not None:
        apply_repetition_penalty(y, seen, case.repetition_penalty)
    return y


def topk_topp_mask(y: torch.Tensor, k: int, p: float) -> torch.Tensor:
    """vllm topk_topp_sampler.py:328-369 `apply_top_k_top_p` (sort based reference path), one row."""
    out = y.clone()
    V = y.numel()
    if k is not None and 0 < k < V:
        kth = torch.topk(out, k).values[-1]
        out = out.masked_fill(out < kth, float("-inf"))
    if p is not None and p < 1.0:
        srt, idx = out.sort(descending=False)
        probs = srt.softmax(dim=-1)
        cum = probs.cumsum(dim=-1)
        mask = cum <= 1 - p
        mask[-1] = False
        srt = srt.masked_fill(mask, float("-inf"))
        out = torch.empty_like(out).scatter_(0, idx, srt)
    return out


# ---------------------------------------------------------------------------------------------- engine RNG
def _mulhilo(a: np.ndarray, b: int) -> tuple[np.ndarray, np.ndarray]:
    prod = a.astype(np.uint64) * np.uint64(b)
    return (prod >> np.uint64(32)).astype(np.uint32), (prod & np.uint64(0xFFFFFFFF)).astype(np.uint32)


def philox_uniform(n: int, seed: int, step: int) -> np.ndarray:
    """u[i] in (0,1) exactly as csrc/sampler.cu: Philox4x32-10, key=(seed_lo, seed_hi), ctr=(i, step, 0, 0), x word."""
    c0 = np.arange(n, dtype=np.uint32)
    c1 = np.full(n, step & 0xFFFFFFFF, dtype=np.uint32)
    c2 = np.zeros(n, dtype=np.uint32)
    c3 = np.zeros(n, dtype=np.uint32)
    k0 = np.uint32(seed & 0xFFFFFFFF)
    k1 = np.uint32((seed >> 32) & 0xFFFFFFFF)
    for _ in range(10):
        hi0, lo0 = _mulhilo(c0, 0xD2511F53)
        hi1, lo1 = _mulhilo(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = hi1 ^ c1 ^ k0, lo1, hi0 ^ c3 ^ k1, lo0
        k0 = np.uint32((int(k0) + 0x9E3779B9) & 0xFFFFFFFF)
        k1 = np.uint32((int(k1) + 0xBB67AE85) & 0xFFFFFFFF)
    u = ((c0 >> np.uint32(8)).astype(np.float32) + np.float32(0.5)) * np.float32(1.0 / 16777216.0)
    return np.minimum(u, np.float32(1) - np.float32(2.0 ** -24))   # (24 ones and a half round to 2^24)


# ---------------------------------------------------------------------------------------------- full row
def unpack_token_bitmask(words: np.ndarray, vocab: int) -> torch.Tensor:
    """xgrammar's token bitmask (int32 words, bit (i & 31) of word (i >> 5) set = token i allowed) -> bool [vocab]."""
    w = np.ascontiguousarray(words).view(np.uint32).reshape(-1)
    idx = np.arange(vocab)
    return torch.from_numpy(((w[idx >> 5] >> (idx & 31).astype(np.uint32)) & 1).astype(bool))


def apply_token_bitmask(raw: torch.Tensor, allow: torch.Tensor) -> torch.Tensor:
    """Guided decoding: vLLM masks the logits before its sampler sees them (v1/worker/gpu_model_runner.py ->
    v1/structured_output/utils.py `apply_grammar_bitmask` -> xgrammar `apply_token_bitmask_inplace`): every token whose
    bit is clear becomes -inf.  Pinned against xgrammar's own CPU kernel in tests/test_guided_cpu.py."""
    return raw.masked_fill(~allow, float("-inf"))


def sample_row(raw_logits: torch.Tensor, case: SamplingCase, seen: torch.Tensor | None = None,
               allow: torch.Tensor | None = None) -> dict:
    """One row through the whole contract.  raw_logits: 1-D fp32 (the fp32 view of the model-dtype logits);
    allow: bool [V] guided-decoding mask of this step (None: unconstrained)."""
    raw = raw_logits.float()
    if allow is not None:
        raw = apply_token_bitmask(raw, allow)
    V = raw.numel()
    y = process_logits(raw, case, seen)
    allowed = None
    if case.greedy:
        token = int(torch.argmax(y))           # first max index (torch semantics; sampler.py:235-236)
    else:
        z = y / torch.tensor(case.temperature, dtype=torch.float32)
        z = topk_topp_mask(z, case.top_k, case.top_p)
        allowed = torch.isfinite(z)
        u = torch.from_numpy(philox_uniform(V, case.seed, case.n_out))
        score = (z - z[allowed].max()) - torch.log(-torch.log(u))
        score = score.masked_fill(~allowed, float("-inf"))
        token = int(torch.argmax(score))
    res = {"token": token, "allowed": allowed, "processed": y}
    if case.num_logprobs > 0:
        lp = torch.log_softmax(raw, dim=-1)     # raw_logprobs mode (sampler.py:79-88)
        tok_lp = lp[token]
        res["logprob"] = float(tok_lp)
        res["rank"] = int((lp >= tok_lp).sum())  # ops/logprobs.py:27
        n = min(case.num_logprobs, V)
        top = torch.topk(lp, n)
        res["topn_ids"] = top.indices.tolist()
        res["topn_logprobs"] = top.values.tolist()
    return res


def check_stop(n_out: int, token: int, n_total: int, *, eos: int, min_tokens: int, max_tokens: int,
               max_model_len: int, stop_token_ids: tuple[int, ...] = ()) -> tuple[str | None, int | None]:
    """vllm v1/core/sched/utils.py:94-130 -> (finish_reason, stop_reason)."""
    if n_out < min_tokens:
        return None, None
    if token == eos:
        return "stop", None
    if token in stop_token_ids:
        return "stop", token
    if n_total >= max_model_len or n_out >= max_tokens:
        return "length", None
    return None, None


def len_penalty_factor_m1(n_out: int, start: int, decay: float) -> float:
    """What the host passes to the kernel: float32(pow(decay, max(0, n_out-start)) - 1) (python double then cast)."""
    return float(np.float32(math.pow(decay, max(0, n_out - start)) - 1.0))
