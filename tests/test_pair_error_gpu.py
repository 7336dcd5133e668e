"""The error word of the products on CTA pairs (csrc/gemm_pair.cu): it is there before the first step, whatever that step is."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

FIRST_STEP_IS_CAPTURED = """
import sys; sys.path.insert(0, {root!r})
from vllm_tgis_adapter_b200.engine import ponenex
from vllm_tgis_adapter_b200.engine.core import NativeEngine, cache_block_bytes, make_sampling_params
mc = ponenex.PRESETS["ponenex-tiny"]
texts = []
for graphs in (True, False):
    eng = NativeEngine(mc, max_num_seqs=2, max_batched_tokens=64, kv_cache_bytes=cache_block_bytes(mc) * 8, use_cuda_graphs=graphs)
    eng.load_weights(ponenex.synthetic_weights(mc, seed=5))
    texts.append([o.new_token for o in eng.generate_sync([[7]], make_sampling_params(max_tokens=4))[0]])
    eng.close()
assert len(texts[0]) == 4 and texts[0] == texts[1], texts
print("same tokens", texts[0])
"""


def test_the_first_launch_of_a_process_may_be_captured():
    """A one-token prompt is a decode-shaped step: with graphs on the first expert product of the process is captured."""
    r = subprocess.run([sys.executable, "-c", FIRST_STEP_IS_CAPTURED.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same tokens" in r.stdout, r.stdout + r.stderr
