"""The error word of the products on CTA pairs (csrc/gemm_pair.cu): it is there before the first step, whatever that step is, and
is looked at wherever their results are used.  The word is raised on the host, at a chosen launch."""
import ctypes as C
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import ROOT
from vllm_tgis_adapter_b200.engine import ponenex
from vllm_tgis_adapter_b200.engine.core import EngineError, NativeEngine, cache_block_bytes, make_sampling_params

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


@pytest.fixture
def lib():
    from vllm_tgis_adapter_b200.engine._lib import load_library

    lib = load_library()
    lib.tgis_k_pair_fault(0)
    yield lib
    lib.tgis_k_pair_fault(0)


def _engine():
    mc = ponenex.PRESETS["ponenex-tiny"]
    eng = NativeEngine(mc, max_num_seqs=300, max_batched_tokens=512, kv_cache_bytes=cache_block_bytes(mc) * 320)
    eng.load_weights(ponenex.synthetic_weights(mc, seed=5))
    return eng


TOKENS = [(7 * i) % 1000 for i in range(300)]


def _replay(eng):
    return eng.trace_step([("s", TOKENS, list(range(300)))], ["s"])


def _prompt_logprobs(eng):
    records = eng.generate_sync([TOKENS], make_sampling_params(max_tokens=1, prompt_logprobs=1))[0]
    return np.array([o.logprob for o in records if o.prompt_pos >= 0])


@pytest.mark.parametrize("work", [_replay, _prompt_logprobs])
def test_a_wait_that_runs_out_behind_the_step_is_reported(lib, work):
    """The head over the rows of a replay step and over a prompt's positions runs after the step's own end; with more rows than a
    token tile it is the last launch on CTA pairs.  Where that launch fails the call does."""
    eng = _engine()
    lib.tgis_k_pair_fault(0)
    good = work(eng)
    launches = lib.tgis_k_pair_fault(0)
    assert launches > 1 and len(good) >= 299
    lib.tgis_k_pair_fault(launches)
    with pytest.raises(EngineError, match="wait ran out"):
        work(eng)
    eng.close()


def test_a_wait_that_runs_out_inside_the_step_is_reported(lib):
    eng = _engine()
    lib.tgis_k_pair_fault(1)
    with pytest.raises(EngineError, match="wait ran out"):
        _replay(eng)
    eng.close()


def test_a_step_that_fails_leaves_the_callers_buffer_alone(lib, monkeypatch):
    eng, made = _engine(), []

    def full(shape, dtype):
        made.append(np.full(shape, 7.0, dtype))
        return made[-1]

    monkeypatch.setattr(np, "empty", full)
    lib.tgis_k_pair_fault(1)
    with pytest.raises(EngineError, match="wait ran out"):
        _replay(eng)
    assert len(made) == 1 and made[0].size > 4096 and bool((made[0] == 7.0).all())
    eng.close()


def test_kernel_hooks_report_it(lib):
    x, w, y = (torch.zeros(512, 512, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    ms = C.c_float()
    for expect in (0, -1, 0):
        lib.tgis_k_pair_fault(1 if expect else 0)
        assert lib.tgis_k_gemm(p(x), p(w), p(y), 300, 512, 512, 512, 0, 1, C.byref(ms), 0) == expect
        lib.tgis_k_pair_fault(1 if expect else 0)
        seg = torch.tensor([0, 300], device="cuda", dtype=torch.int32)
        assert lib.tgis_k_gemm_any(p(x), p(w), p(y), 1, 1, 1, 300, 512, 512, 512, 512, 512, 1, 0, 0, 0, p(seg), 1, 512 * 512, None, 1, 0, None, 0) == expect
