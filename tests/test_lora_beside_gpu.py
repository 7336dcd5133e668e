"""The adapters' shrink beside the projection it corrects (csrc/lora.cu): a step in which it starts under the running projection gives
the bits of one whose kernels run one after the other, on every kernel that a projection is sent to, with requests of several adapters and
of none in a step.  ROUTES says which kernels a step of so many requests has: register products (the shrink stays ahead of those), equal
shares, token tiles on pairs with maps of their own, weights cut along k with tiles of 16 (7 and 12 requests), 32 (24) and 64 tokens (40); the
prompts of 150 requests go through the token tiles on pairs with the engine's maps."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
REGISTERS, SHARES, SMALL_PAIRS, PAIRS, CUT = range(5)   # tgis_k_gemm_route
# hidden width, requests -> kernels of the four projections' decode steps (4224 wide: no product is small enough for the registers)
ROUTES = {(2048, 7): {REGISTERS}, (2048, 12): {REGISTERS, CUT}, (2048, 24): {REGISTERS, SHARES, CUT}, (2048, 40): {SHARES, CUT}, (2048, 150): {SMALL_PAIRS},
          (4224, 7): {CUT}, (4224, 24): {CUT}}


def config(hidden):
    from oracle.llama_oracle import LlamaConfig

    q = 16 if hidden == 2048 else 32
    return LlamaConfig(n_layers=3 if q == 16 else 2, hidden=hidden, n_q_heads=q, n_kv_heads=q // 4, ffn=4096, vocab=2048, max_model_len=256)


def child(root, hidden, n):
    import numpy as np

    from oracle.llama_oracle import rope_table, synthetic_weights
    from test_lora_cpu import make_peft_dir
    from vllm_tgis_adapter_b200.engine.core import ModelConfig, NativeEngine, make_sampling_params
    from vllm_tgis_adapter_b200.engine.lora import read_adapter

    cfg = config(hidden)
    eng = NativeEngine(ModelConfig(n_layers=cfg.n_layers, hidden=cfg.hidden, n_q_heads=cfg.n_q_heads, n_kv_heads=cfg.n_kv_heads, ffn=cfg.ffn,
                                   vocab=cfg.vocab, rope_theta=cfg.rope_theta, rms_eps=cfg.rms_eps, max_model_len=cfg.max_model_len),
                       max_loras=3, max_lora_rank=16, max_num_seqs=n, max_batched_tokens=2048, kv_cache_bytes=256 << 20)
    eng.load_weights({k: w.cpu() for k, w in synthetic_weights(cfg, seed=1, device="cuda").items()})
    eng.load_weight("tgis.rope_cos_sin", rope_table(cfg))
    for s in (1, 2, 3):
        d = make_peft_dir(root, f"a{s}", n_layers=cfg.n_layers, hidden=cfg.hidden, q_dim=cfg.q_dim, kv_dim=cfg.kv_dim, ffn=cfg.ffn,
                          r=8 * (1 + s % 2), alpha=16, seed=s)
        eng.load_adapter(s, read_adapter(str(d), n_layers=cfg.n_layers, max_rank=16)[1])
    rng = np.random.RandomState(n)
    prompts = [rng.randint(3, cfg.vocab, size=9 + i % 17).tolist() for i in range(n)]
    sps = [make_sampling_params(greedy=True, max_tokens=8, min_tokens=8, num_logprobs=1, eos_token_id=2, lora_slot=i % 4) for i in range(n)]
    for _ in range(2):   # the second time on captured graphs
        for recs in eng.generate_sync(prompts, sps):
            print("out", [(r.new_token, r.logprob.hex()) for r in recs if r.new_token is not None])
    eng.close()


def test_the_steps_take_the_kernels_they_are_there_for():
    import torch

    from vllm_tgis_adapter_b200.engine._lib import load_library

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for (hidden, n), routes in ROUTES.items():
        c = config(hidden)
        at = lambda T: {load_library().tgis_k_gemm_route(T, N, K, sms, 0) for N, K in (
            (c.q_dim + 2 * c.kv_dim, hidden), (hidden, c.q_dim), (2 * c.ffn, hidden), (hidden, c.ffn))}
        assert at(n) == routes, (hidden, n, at(n))
    assert at(2048) == {PAIRS}


@pytest.mark.parametrize("hidden,n", list(ROUTES))
def test_side_by_side_is_one_after_the_other(hidden, n, tmp_path):
    def run(pdl):
        os.makedirs(tmp_path / pdl)
        env = dict(os.environ, TGIS_PDL=pdl, PYTHONPATH=os.pathsep.join([HERE, os.path.dirname(HERE), os.environ.get("PYTHONPATH", "")]))
        p = subprocess.run([sys.executable, __file__, str(tmp_path / pdl), str(hidden), str(n)], env=env, capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-2000:]
        out = [line for line in p.stdout.splitlines() if line.startswith("out")]
        assert len(out) == 2 * n
        return out

    assert run("1") == run("0")


if __name__ == "__main__":
    from pathlib import Path

    child(Path(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3]))
