"""Scheduler and slot-state logic on CPU: admission under page reservations, lifecycle, finalize, refcount
conservation, overlap-vs-sequential equivalence, flags and request validation."""
import os

import pytest
import torch

from smcsd_b200.config import EngineArgs, env_flag
from smcsd_b200.io_types import GenerateRequest, ParticleOutput, RequestOutput, SamplingParams, validate_request
from smcsd_b200.runtime.scheduler import SMCScheduler


def _sched(**kw):
    base = dict(model_path="preset:tiny-target", draft_model_path="preset:tiny-draft", n_particles=4, gamma=3,
                dtype="float32", device="cpu", max_running_requests=2, draft_temperature=0.7, target_temperature=0.7)
    base.update(kw)
    return SMCScheduler(EngineArgs(**base).finalize())


def _req(rid, n=10, **sp):
    g = torch.Generator().manual_seed(hash(rid) % 1000)
    return GenerateRequest(rid, torch.randint(0, 4096, (n,), generator=g).tolist(), SamplingParams(**sp))


def test_admission_is_gated_by_slots_and_pages():
    s = _sched(max_running_requests=2, max_total_tokens=400)
    for i in range(4):
        s.add_request(_req(f"r{i}", max_new_tokens=20, ignore_eos=True))
    s.step()
    assert len(s.running) <= 2 and len(s.waiting) >= 2
    assert s.reserved_pages <= s.alloc.size
    outs = s.run_until_idle()
    done = [o for o in outs if isinstance(o, RequestOutput)]
    assert len(done) == 4 and all(o.completion_tokens == 20 for o in done)
    s.check_idle_invariants()
    s.alloc.check_conservation()


def test_request_larger_than_pool_is_aborted_not_hung():
    s = _sched(max_total_tokens=120)
    s.add_request(_req("big", n=30, max_new_tokens=500, ignore_eos=True))
    outs = s.run_until_idle()
    o = [x for x in outs if isinstance(x, RequestOutput)][0]
    assert o.aborted and "KV pages" in o.error


def test_queue_limit_and_abort():
    s = _sched(max_queued_requests=1)
    s.add_request(_req("a", max_new_tokens=30, ignore_eos=True))
    s.add_request(_req("b", max_new_tokens=30, ignore_eos=True))
    assert any(isinstance(o, RequestOutput) and o.aborted and "queue" in o.error for o in s.outbox)
    s.step()
    s.step()
    s.abort("a")
    outs = s.run_until_idle()
    assert any(isinstance(o, RequestOutput) and o.rid == "a" and o.aborted for o in outs)
    s.check_idle_invariants()


def test_prev_token_is_seeded_with_last_prompt_token():
    s = _sched()
    r = _req("x", n=7, max_new_tokens=9, ignore_eos=True)
    s.add_request(r)
    s.step()
    slots = s.state.row_slots[s.state.group_rows["x"]]
    assert all(int(s.state.prev_ids[i]) == r.input_ids[-1] for i in slots)
    assert all(int(s.state.seq_lens[i]) == 7 for i in slots)
    assert all(int(s.state.token_counts[i]) == 1 for i in slots)
    # fan-out shares the prompt pages: every prompt page is referenced once per particle
    pages = s.bt.table[slots[0], :7].long()
    assert (s.alloc.refcount[pages] == 4).all()
    s.run_until_idle()
    s.check_idle_invariants()


def test_finalize_reports_posterior_pick_and_particles():
    s = _sched()
    s.add_request(_req("p", max_new_tokens=11, ignore_eos=True))
    outs = s.run_until_idle()
    po = [o for o in outs if isinstance(o, ParticleOutput)][0]
    ro = [o for o in outs if isinstance(o, RequestOutput)][0]
    assert len(po.particle_output_ids) == 4 and 0 <= po.picked < 4
    assert ro.output_ids == po.particle_output_ids[po.picked]
    assert ro.finish_reason == {"type": "length", "length": 11}
    assert len(po.log_w_tilde) == 4 and isinstance(po.log_Z_hat, float)


def test_single_particle_never_resamples():
    s = _sched(n_particles=1)
    s.add_request(_req("one", max_new_tokens=15, ignore_eos=True))
    outs = s.run_until_idle()
    assert s.stats["resampled_groups"] == 0
    assert [o for o in outs if isinstance(o, RequestOutput)][0].completion_tokens == 15


def test_multinomial_resampling_runs_on_the_torch_path():
    s = _sched(resample_method="multinomial", resample_threshold=2.0)
    s.add_request(_req("m", max_new_tokens=13, ignore_eos=True))
    s.run_until_idle()
    assert s.stats["resampled_groups"] > 0
    s.check_idle_invariants()


def test_env_switch_beats_keyword_beats_default(monkeypatch):
    assert env_flag("SMC_X_UNSET", None, True) is True
    assert env_flag("SMC_X_UNSET", False, True) is False
    monkeypatch.setenv("SMC_DEFER_BONUS", "0")
    a = EngineArgs(model_path="a", draft_model_path="b", defer_bonus=True).finalize()
    assert a.defer_bonus is False
    monkeypatch.setenv("SMC_DEFER_BONUS", "1")
    assert EngineArgs(model_path="a", draft_model_path="b", defer_bonus=False).finalize().defer_bonus is True
    g = EngineArgs(model_path="a", draft_model_path="b", draft_temperature=0.0).finalize()
    assert g.cycle_graph is False           # greedy proposals take the eager path
    with pytest.raises(ValueError):
        EngineArgs(model_path="a", draft_model_path="b", power_alpha=0.0).finalize()


def test_request_validation_messages():
    ok = GenerateRequest("r", [1, 2, 3], SamplingParams(max_new_tokens=4))
    assert validate_request(ok, 128, 4) is None
    for field, val, word in [("image_data", object(), "multimodal"), ("input_embeds", [1.0], "input_embeds"),
                             ("grammar", "g", "grammar"), ("return_logprob", True, "return_logprob"),
                             ("return_hidden_states", True, "hidden"), ("return_routed_experts", True, "experts")]:
        r = GenerateRequest("r", [1, 2, 3], SamplingParams(max_new_tokens=4))
        setattr(r, field, val)
        assert word in validate_request(r, 128, 4)
    assert "stop regex" in validate_request(GenerateRequest("r", [1], SamplingParams(stop_regex="a+")), 128, 4)
    assert "context" in validate_request(GenerateRequest("r", [1] * 100, SamplingParams(max_new_tokens=100)), 128, 4)
    assert "empty" in validate_request(GenerateRequest("r", [], SamplingParams()), 128, 4)


def test_debug_records_are_appended(tmp_path, monkeypatch):
    import json
    path = tmp_path / "diag.jsonl"
    monkeypatch.setenv("SMC_DIAG_PATH", str(path))
    s = _sched()
    s.add_request(_req("d", max_new_tokens=6, ignore_eos=True))
    s.run_until_idle()
    rec = [json.loads(x) for x in path.read_text().splitlines()]
    assert rec and rec[0]["event"] == "finalize" and "pid" in rec[0] and "timestamp_ns" in rec[0]


def test_abort_of_a_group_whose_final_snapshot_is_pending():
    """With the overlapped loop a request's last cycle leaves one snapshot pending; an abort that arrives in that
    window must not release the group twice nor answer twice."""
    s = _sched(enable_overlap=True)
    s.add_request(_req("a", max_new_tokens=8, ignore_eos=True))       # gamma + 1 = 4 tokens per cycle: two cycles
    outs = []
    for _ in range(50):
        outs += s.step()
        if s.pending and "a" in s.running:
            s.abort("a")
            outs += list(s.outbox)
            s.outbox.clear()
    outs += s.run_until_idle()
    mine = [o for o in outs if isinstance(o, RequestOutput) and o.rid == "a"]
    assert len(mine) >= 1
    assert len([o for o in mine if o.finished]) == 1 or all(o.aborted for o in mine)
    s.check_idle_invariants()
    s.alloc.check_conservation()


def test_request_at_the_context_limit_survives_the_extra_overlap_cycle():
    """Two groups with overlap on: the one that ends on length gets one more cycle while the other keeps running;
    its block-table row must have room for it."""
    s = _sched(enable_overlap=True, max_running_requests=2)
    ctx = s.args.context_len if hasattr(s.args, "context_len") else s.bt.table.shape[1]
    gamma = s.args.gamma
    n = 12
    longest = ctx - n - 2 * (gamma + 1)
    assert validate_request(_req("x", n=n, max_new_tokens=longest + 1), ctx, gamma) is not None
    assert validate_request(_req("x", n=n, max_new_tokens=longest), ctx, gamma) is None
    if longest > 400:          # keep the CPU run short: the bound itself is checked above
        return
    s.add_request(_req("edge", n=n, max_new_tokens=longest, ignore_eos=True))
    s.add_request(_req("other", n=n, max_new_tokens=longest, ignore_eos=True))
    outs = s.run_until_idle()
    done = [o for o in outs if isinstance(o, RequestOutput)]
    assert len(done) == 2 and not any(o.aborted for o in done)
    s.check_idle_invariants()


def test_priority_is_refused_unless_switched_on_and_orders_the_queue():
    s = _sched()
    r = _req("p", max_new_tokens=8, ignore_eos=True)
    r.priority = 3
    s.add_request(r)
    assert any(isinstance(o, RequestOutput) and o.aborted and "priority" in o.error for o in s.outbox)
    for low_first, want in ((False, ["hi", "mid", "mid2", "lo", "none"]), (True, ["lo", "mid", "mid2", "hi", "none"])):
        s = _sched(enable_priority_scheduling=True, schedule_low_priority_values_first=low_first,
                   max_running_requests=1)
        for rid, prio in (("mid", 5), ("none", None), ("lo", 1), ("hi", 9), ("mid2", 5)):
            r = _req(rid, max_new_tokens=6, ignore_eos=True)
            r.priority = prio
            s.add_request(r)
        assert [g.rid for g in s.waiting] == want
        done = [o.rid for o in s.run_until_idle() if isinstance(o, RequestOutput) and o.finished]
        assert done == want                   # one group at a time: served in queue order
        s.check_idle_invariants()


def test_pause_holds_the_queue_and_continue_resumes():
    s = _sched()
    s.add_request(_req("a", max_new_tokens=12, ignore_eos=True))
    s.step()                                  # prefill
    s.step()
    cycles = s.stats["cycles"]
    assert s.pause_generation() and not s.pending
    s.add_request(_req("b", max_new_tokens=6, ignore_eos=True))
    for _ in range(5):
        assert all(not (isinstance(o, RequestOutput) and o.finished) for o in s.step())
    assert s.stats["cycles"] == cycles and len(s.waiting) == 1 and s.has_work()
    s.abort("b")                              # still possible while paused
    assert any(isinstance(o, RequestOutput) and o.rid == "b" and o.aborted for o in s.step())
    s.continue_generation()
    outs = s.run_until_idle()
    assert any(isinstance(o, RequestOutput) and o.rid == "a" and o.completion_tokens == 12 for o in outs)
    s.check_idle_invariants()


def test_materialize_failure_rolls_back_and_aborts_only_that_group():
    """The fan-out of one admitted group fails (injected on the host): that request comes back aborted with the
    message, its prompt pages and parent row are returned, and the other requests are served as usual."""
    s = _sched(max_running_requests=2)
    real = s.state.allocate_group

    def flaky(rid, **kw):
        if rid == "bad":
            raise RuntimeError("injected fan-out failure")
        return real(rid, **kw)
    s.state.allocate_group = flaky
    for rid in ("ok1", "bad", "ok2"):
        s.add_request(_req(rid, max_new_tokens=9, ignore_eos=True))
    outs = [o for o in s.run_until_idle() if isinstance(o, RequestOutput) and o.finished]
    by = {o.rid: o for o in outs}
    assert by["bad"].aborted and "injected" in by["bad"].error
    assert by["ok1"].completion_tokens == 9 and by["ok2"].completion_tokens == 9 and not by["ok1"].aborted
    s.check_idle_invariants()
    s.alloc.check_conservation()
    assert s.alloc.available() == s.alloc.size


def test_owned_pages_come_back_as_counted_ones_do():
    from smcsd_b200.memory.pools import PageAllocator
    a, b = PageAllocator(50, "cpu"), PageAllocator(50, "cpu")
    for alloc, free in ((a, a.dec_ref_and_free), (b, b.free_owned)):
        first, second = alloc.alloc(7), alloc.alloc(11)
        free(first[torch.tensor([3, 0, 6, 1, 2, 5, 4])])
        third = alloc.alloc(4)
        free(torch.empty(0, dtype=torch.int32))
        free(torch.cat([second, third]))
        alloc.check_conservation()
    assert torch.equal(a.free_stack, b.free_stack) and torch.equal(a.refcount, b.refcount) and a.available() == b.available() == 50


def test_fed_tokens_are_numbers_of_the_vocabulary():
    import numpy as np
    from smcsd_b200.runtime.feeder import _numbers
    for same in ([1, 2, 3], (1, 2, 3), torch.tensor([1, 2, 3]), [torch.tensor(1), torch.tensor(2), torch.tensor(3)], np.array([1, 2, 3]), range(1, 4)):
        assert _numbers(same).astype(np.int64).tolist() == [1, 2, 3]
    assert len(_numbers([])) == 0
    for bad in ([-0.5], [float("nan")], [1 << 70], [-1]):
        x = _numbers(bad)
        assert not ((x >= 0) & (x < 100)).all()


def test_bytes_to_the_device_of_ragged_prompt_passes_are_counted():
    from types import SimpleNamespace
    from smcsd_b200.ops.native_backend import NativeRunner
    from smcsd_b200.ops.ragged import Portion
    r = NativeRunner.__new__(NativeRunner)
    r.pass_bytes, r.device = 0, torch.device("cpu")
    seen = []
    nm = SimpleNamespace(T=32, BLOCK=8, bt=torch.zeros(4, 64, dtype=torch.int32), xa=torch.zeros(32, 16), forward_plan=lambda p: seen.append(p.keep[0].numel()))
    assert r._ragged_pass(nm, [Portion(0, 0, list(range(40))), Portion(1, 5, [3, 4])], [[], []]) is None
    assert len(seen) == 2 and r.pass_bytes == 4 * sum(seen) >= 3 * 4 * 42          # id, position and row of every token at least


@pytest.mark.parametrize("how", ["dec_ref_and_free", "free_owned"])
def test_pages_that_came_back_are_handed_out_ascending(how):
    from smcsd_b200.memory.pools import PageAllocator
    a = PageAllocator(100, "cpu")
    first, other = a.alloc(30), a.alloc(20)
    assert torch.equal(first, torch.arange(1, 31, dtype=torch.int32))
    getattr(a, how)(first[torch.randperm(30, generator=torch.Generator().manual_seed(0))])
    assert torch.equal(a.alloc(30), first) and torch.equal(other, torch.arange(31, 51, dtype=torch.int32))
    getattr(a, how)(torch.cat([other, first]))
    assert torch.equal(a.alloc(100), torch.arange(1, 101, dtype=torch.int32))


def test_fed_tokens_may_mix_numbers_and_tensors_of_one_element():
    from smcsd_b200.runtime.feeder import _numbers
    for mixed in ([1, torch.tensor(2), 3], [1, torch.tensor([2]), 3], [torch.tensor([1]), 2, torch.tensor(3)]):
        assert _numbers(mixed).tolist() == [1, 2, 3]
    with pytest.raises((TypeError, ValueError, RuntimeError)):
        _numbers([1, torch.tensor([2, 3])])


@pytest.mark.parametrize("nq,nkv,ks,longest,tiles,tc", [
    (8, 8, 2, 4112, 1, False), (8, 8, 1, 4256, 2, False), (8, 8, 1, 4256, 3, True), (16, 16, 2, 4112, 1, False), (32, 32, 2, 4112, 1, True), (8, 8, 1, 1000, 1, True), (32, 8, 2, 4112, 1, True),
    (16, 4, 8, 4112, 1, False), (16, 4, 2, 4112, 8, True), (16, 4, 8, 900, 1, True)])
def test_which_prompt_passes_take_the_tiled_attention(nq, nkv, ks, longest, tiles, tc):
    from types import SimpleNamespace
    from smcsd_b200.ops.native_backend import NativeRunner
    r = NativeRunner.__new__(NativeRunner)
    nm = SimpleNamespace(nq=nq, nkv=nkv, prompt_tokens=256 * nkv // nq, _ks=lambda blocks, E: ks)
    assert r._takes_tiles(nm, longest, 7, tiles) == tc
    nm.prompt_tokens = 0
    assert not r._takes_tiles(nm, longest, 7, tiles)
