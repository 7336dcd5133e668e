"""Records of generated tokens (engine/core.py): whole native records at a time against the structure's own fields, and a call whose
records are made beside its steps -- all of them, in order, also what was reported before a step failed."""
import ctypes as C
import random
import time

import pytest

from vllm_tgis_adapter_b200.engine import _lib
from vllm_tgis_adapter_b200.engine.core import EngineError, NativeEngine, StepOutput, make_sampling_params


def _record(rng, rid, new=True):
    o = _lib.TgisStepOutput()
    o.request_id, o.n_new_tokens, o.token_id, o.logprob, o.rank = rid.encode(), int(new), rng.randrange(1 << 20), rng.uniform(-20, 0), rng.randrange(99)
    o.n_topn = rng.randrange(_lib.MAX_TOPN + 1)
    for j in range(_lib.MAX_TOPN):
        o.topn_ids[j], o.topn_logprobs[j] = rng.randrange(1 << 20), rng.uniform(-20, 0)
    o.finish_reason, o.stop_token_id, o.n_prompt_tokens, o.n_output_tokens = rng.randrange(4), -1, rng.randrange(99), rng.randrange(99)
    o.ts_arrival, o.ts_first_scheduled, o.ts_first_token, o.ts_last_token = (rng.random() for _ in range(4))
    o.prompt_pos = rng.choice([-1, 3])
    return o


def _by_field(o):
    return StepOutput(request_id=o.request_id.decode(), new_token=o.token_id if o.n_new_tokens else None, logprob=o.logprob, rank=o.rank,
                      topn=[(o.topn_ids[j], o.topn_logprobs[j]) for j in range(o.n_topn)], finish_reason=o.finish_reason, stop_token_id=o.stop_token_id,
                      n_prompt_tokens=o.n_prompt_tokens, n_output_tokens=o.n_output_tokens, ts_arrival=o.ts_arrival, ts_first_scheduled=o.ts_first_scheduled,
                      ts_first_token=o.ts_first_token, ts_last_token=o.ts_last_token, prompt_pos=o.prompt_pos, token_id=o.token_id)


class _Lib:
    """An engine whose steps add `per_step` records each, `fail_at`: the step that fails."""

    def __init__(self, steps, per_step, requests, fail_at=None):
        rng = random.Random(5)
        self.made = [[_record(rng, f"r{(s * per_step + i) % requests}", rng.random() < 0.9) for i in range(per_step)] for s in range(steps)]
        self.queue, self.fail_at, self.added = [], fail_at, []

    def tgis_engine_add_request(self, h, rid, arr, n, params):
        self.added.append(rid)
        return 0

    def tgis_engine_run_until_idle(self, h):
        for s, records in enumerate(self.made):
            if s == self.fail_at:
                return -1
            self.queue.extend(records)
            time.sleep(0.001)
        return len(self.made)

    def tgis_engine_poll(self, h, buf, cap, timeout):
        n = min(cap, len(self.queue))
        for i in range(n):
            C.memmove(C.byref(buf, i * C.sizeof(_lib.TgisStepOutput)), C.byref(self.queue.pop(0)), C.sizeof(_lib.TgisStepOutput))
        return n

    def tgis_last_error(self):
        return b"a step failed"

    tgis_engine_destroy = tgis_engine_stop = lambda self, *a: 0


def _engine(lib):
    eng = NativeEngine.__new__(NativeEngine)
    eng.lib, eng._h, eng._poll_buf, eng._unread = lib, None, (_lib.TgisStepOutput * 7)(), []
    return eng


def test_records_equal_their_fields():
    lib = _Lib(1, 40, 5)
    lib.queue = list(lib.made[0])
    eng, got = _engine(lib), []
    while more := eng.poll(0):
        got += more
    want = [_by_field(o) for o in lib.made[0]]
    assert got == want and [type(o.rank) for o in got] == [int] * 40 and all(type(v) is float for o in got for _, v in o.topn)


@pytest.mark.parametrize("max_tokens", [4, 400])   # (few tokens: no second thread)
def test_every_record_arrives_in_order(max_tokens):
    lib = _Lib(30, 9, 3)
    sp = make_sampling_params(max_tokens=max_tokens)
    res = _engine(lib).generate_sync([[1], [2], [3]], sp)
    flat = [_by_field(o) for step in lib.made for o in step]
    assert lib.added == [b"r0", b"r1", b"r2"] and not lib.queue
    assert res == [[o for o in flat if o.request_id == f"r{i}"] for i in range(3)]


@pytest.mark.parametrize("max_tokens", [4, 400])
def test_records_before_a_failure_stay_to_be_polled(max_tokens, monkeypatch):
    lib = _Lib(30, 9, 3, fail_at=20)
    monkeypatch.setattr(_lib, "last_error", lambda lib: "a step failed")
    eng, got = _engine(lib), []
    with pytest.raises(EngineError, match="a step failed"):
        eng.generate_sync([[1], [2], [3]], make_sampling_params(max_tokens=max_tokens))
    while more := eng.poll(0):
        got += more
    assert got == [_by_field(o) for step in lib.made[:20] for o in step]


@pytest.mark.parametrize("max_tokens", [4, 400])
def test_a_call_after_a_failure_takes_what_was_left_first(max_tokens, monkeypatch):
    """In the order in which they were reported, whether or not a second thread made the records."""
    lib = _Lib(30, 9, 3, fail_at=20)
    monkeypatch.setattr(_lib, "last_error", lambda lib: "a step failed")
    eng, sp = _engine(lib), make_sampling_params(max_tokens=max_tokens)
    with pytest.raises(EngineError, match="a step failed"):
        eng.generate_sync([[1], [2], [3]], sp)
    flat = [_by_field(o) for step in lib.made[:20] for o in step]
    lib.made, lib.fail_at = _Lib(12, 9, 3).made[5:], None
    flat += [_by_field(o) for step in lib.made for o in step]
    assert eng.generate_sync([[1], [2], [3]], sp) == [[o for o in flat if o.request_id == f"r{i}"] for i in range(3)]
