"""The adapters' shrink beside the projection it corrects (csrc/lora.cu): a step in which it starts under the running projection gives
the bits of one whose kernels run one after the other, on every kernel that a projection is sent to -- weights cut along k (7 requests),
equal shares (40), token tiles on pairs (150, and the prompts) -- with requests of several adapters and of none in a step."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def child(root, n):
    import numpy as np

    from oracle.llama_oracle import LlamaConfig, rope_table, synthetic_weights
    from test_lora_cpu import make_peft_dir
    from vllm_tgis_adapter_b200.engine.core import ModelConfig, NativeEngine, make_sampling_params
    from vllm_tgis_adapter_b200.engine.lora import read_adapter

    cfg = LlamaConfig(n_layers=3, hidden=2048, n_q_heads=16, n_kv_heads=4, ffn=4096, vocab=2048, max_model_len=256)
    eng = NativeEngine(ModelConfig(n_layers=cfg.n_layers, hidden=cfg.hidden, n_q_heads=cfg.n_q_heads, n_kv_heads=cfg.n_kv_heads, ffn=cfg.ffn,
                                   vocab=cfg.vocab, rope_theta=cfg.rope_theta, rms_eps=cfg.rms_eps, max_model_len=cfg.max_model_len),
                       max_loras=3, max_lora_rank=16, max_num_seqs=n, max_batched_tokens=2048, kv_cache_bytes=256 << 20)
    eng.load_weights(synthetic_weights(cfg, seed=1))
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


@pytest.mark.parametrize("n", [7, 40, 150])
def test_side_by_side_is_one_after_the_other(n, tmp_path):
    def run(pdl):
        os.makedirs(tmp_path / pdl)
        env = dict(os.environ, TGIS_PDL=pdl, PYTHONPATH=os.pathsep.join([HERE, os.path.dirname(HERE), os.environ.get("PYTHONPATH", "")]))
        p = subprocess.run([sys.executable, __file__, str(tmp_path / pdl), str(n)], env=env, capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-2000:]
        out = [line for line in p.stdout.splitlines() if line.startswith("out")]
        assert len(out) == 2 * n
        return out

    assert run("1") == run("0")


if __name__ == "__main__":
    from pathlib import Path

    child(Path(sys.argv[1]), int(sys.argv[2]))
