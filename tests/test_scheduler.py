"""The scheduler's decisions, on the host: admission, portions under the token budget, decode
first, finishing and freeing, and what happens when pages run out."""
import pytest

import kirai_b200
from kirai_b200.cache import CacheManager
from kirai_b200.engine.scheduler import AdmissionError, Scheduler
from kirai_b200.parts.base import KVCacheNeed
from kirai_b200.sampling.params import SamplingParams
from kirai_b200.sampling import rng


def make(num_pages=64, page_size=4, num_slots=4, **kwargs):
    cache = CacheManager([KVCacheNeed(1, 8, None), KVCacheNeed(1, 8, 8)], page_size=page_size, num_pages=num_pages,
                         num_slots=num_slots, device=None)
    defaults = dict(max_batched_tokens=16, max_running=4, max_positions=512, default_max_new_tokens=64)
    defaults.update(kwargs)
    return cache, Scheduler(cache, **defaults)


def run(scheduler, cache, token_of=lambda request: 7, max_steps=10_000):
    """Drives the scheduler with a stand-in for the model; returns the trace of steps."""
    trace = []
    while scheduler.has_work():
        chosen = scheduler.schedule()
        assert chosen and sum(item.count for item in chosen) <= scheduler.max_batched_tokens
        for item in chosen:  # what the step function does with the pages
            assert item.first == item.request.pages.length == item.request.computed
            cache.commit(item.request.pages, item.count)
        sampled = [token_of(item.request) if item.sample else None for item in chosen]
        trace.append([(item.request.request_id, item.first, item.count, item.sample) for item in chosen])
        scheduler.update(chosen, sampled)
        cache.tables.check_consistency()
        assert len(trace) < max_steps
    return trace


def test_prompt_is_cut_to_the_budget_then_decodes():
    cache, scheduler = make()
    request = scheduler.add("a", list(range(37)), SamplingParams(temperature=0.0, max_new_tokens=3))
    trace = run(scheduler, cache)
    assert [step[0][1:] for step in trace] == [(0, 16, False), (16, 16, False), (32, 5, True), (37, 1, True), (38, 1, True)]
    assert request.output == [7, 7, 7] and request.finish_reason == "length"
    assert request.computed == 39  # the last sampled token is never run
    assert cache.free_pages() == [64, 64] and cache.tables.slots.free_slots == 4


def test_decode_goes_first_and_prompts_share_the_rest():
    cache, scheduler = make()
    scheduler.add("a", [1, 2, 3], SamplingParams(max_new_tokens=5, seed=1))
    trace_first = scheduler.schedule()
    for item in trace_first:
        cache.commit(item.request.pages, item.count)
    scheduler.update(trace_first, [9])
    scheduler.add("b", list(range(40)), SamplingParams(max_new_tokens=2, seed=1))
    chosen = scheduler.schedule()
    assert [(c.request.request_id, c.count, c.sample) for c in chosen] == [("a", 1, True), ("b", 15, False)]


def test_prefill_chunk_and_concurrency_limit():
    cache, scheduler = make(max_batched_tokens=64, prefill_chunk=8, max_running=2)
    for name in "abc":
        scheduler.add(name, list(range(20)), SamplingParams(max_new_tokens=1, seed=0))
    chosen = scheduler.schedule()
    assert [(c.request.request_id, c.count) for c in chosen] == [("a", 8), ("b", 8)]  # c waits: two may run
    assert len(scheduler.waiting) == 1


def test_stop_token_and_ignore_eos():
    cache, scheduler = make()
    stops = scheduler.add("s", [1, 2], SamplingParams(max_new_tokens=10, eos_token_id=7, seed=0))
    goes_on = scheduler.add("g", [1, 2], SamplingParams(max_new_tokens=4, eos_token_id=7, ignore_eos=True, seed=0))
    run(scheduler, cache)
    assert stops.output == [7] and stops.finish_reason == "stop"
    assert goes_on.output == [7] * 4 and goes_on.finish_reason == "length"


def test_admission_refuses_what_can_never_run():
    cache, scheduler = make(num_pages=8)
    with pytest.raises(AdmissionError):
        scheduler.add("long", list(range(500)), SamplingParams(max_new_tokens=20))  # beyond max_positions
    with pytest.raises(AdmissionError):
        scheduler.add("big", list(range(40)), SamplingParams(max_new_tokens=2))     # 41 tokens > 8 pages of 4
    with pytest.raises(AdmissionError):
        scheduler.add("many", [1], SamplingParams(max_new_tokens=65))               # above the configured maximum
    with pytest.raises(AdmissionError):
        scheduler.add("empty", [], SamplingParams())
    assert scheduler.add("fits", list(range(30)), SamplingParams(max_new_tokens=3)) is not None


def test_pages_run_out_youngest_is_evicted_and_recomputed():
    # 12 pages of 4 tokens.  Two requests of 17 prompt tokens (5 pages each) decode 12 tokens each: they need
    # 8 pages each in the end, 16 in all, so one must give way and come back.
    cache, scheduler = make(num_pages=12, max_batched_tokens=32)
    a = scheduler.add("a", list(range(17)), SamplingParams(max_new_tokens=12, seed=0))
    b = scheduler.add("b", list(range(100, 117)), SamplingParams(max_new_tokens=12, seed=0))
    counter = {"a": 0, "b": 0}

    def token_of(request):
        counter[request.request_id] += 1
        return counter[request.request_id]

    trace = run(scheduler, cache, token_of)
    assert scheduler.stats["preemptions"] >= 1 and b.preemptions >= 1 and a.preemptions == 0
    assert a.output == list(range(1, 13)) and b.output == list(range(1, 13))  # nothing lost, nothing sampled twice
    assert b.draws_used == 12
    # after eviction b was run again from position 0 with its prompt and what it had generated
    restarts = [entry for step in trace for entry in step if entry[0] == "b" and entry[1] == 0]
    assert len(restarts) == 1 + b.preemptions and restarts[-1][2] > 17
    assert cache.free_pages() == [12, 12]


def test_portion_shrinks_to_free_pages():
    cache, scheduler = make(num_pages=6, max_batched_tokens=64)
    scheduler.add("a", list(range(14)), SamplingParams(max_new_tokens=1, seed=0))   # 4 pages
    scheduler.add("b", list(range(20)), SamplingParams(max_new_tokens=1, seed=0))   # would need 5, 2 are free
    chosen = scheduler.schedule()
    assert [(c.request.request_id, c.count, c.sample) for c in chosen] == [("a", 14, True), ("b", 8, False)]


@pytest.mark.parametrize("native", [False, True])
def test_two_prompts_that_stall_each_other_in_mid_prompt(native):
    # 100 pages of 16 tokens; two prompts of 1,280 tokens (80 pages each) cut into portions of 256: after three steps
    # both hold pages, neither can finish its prompt and nobody decodes.  The younger one must give way.
    from kirai_b200.engine.scheduler import NativeScheduler

    cache = CacheManager([KVCacheNeed(1, 8, None)], page_size=16, num_pages=100, num_slots=4, device=None)
    scheduler = (NativeScheduler if native else Scheduler)(
        cache, max_batched_tokens=512, max_running=4, prefill_chunk=256, max_positions=4096, default_max_new_tokens=8)
    a = scheduler.add("a", list(range(1280)), SamplingParams(max_new_tokens=4, seed=0))
    b = scheduler.add("b", list(range(1280)), SamplingParams(max_new_tokens=4, seed=0))
    trace = run(scheduler, cache)
    assert a.preemptions == 0 and b.preemptions >= 1 and scheduler.stats["preemptions"] == b.preemptions
    assert len(a.output) == 4 and len(b.output) == 4 and a.finish_reason == b.finish_reason == "length"
    assert cache.free_pages() == [100]
    # while a request waits for pages in mid-prompt nobody new is admitted: b comes back only after a has finished
    # its prompt or freed pages, and is then recomputed from its first token
    restarts = [entry for step in trace for entry in step if entry[0] == "b" and entry[1] == 0]
    assert len(restarts) == 1 + b.preemptions


def test_abort_frees_everything():
    cache, scheduler = make()
    request = scheduler.add("a", list(range(10)), SamplingParams(max_new_tokens=5, seed=0))
    waiting = scheduler.add("b", list(range(10)), SamplingParams(max_new_tokens=5, seed=0))
    chosen = scheduler.schedule()
    for item in chosen:
        cache.commit(item.request.pages, item.count)
    scheduler.update(chosen, [1, 1])
    scheduler.abort(request)
    scheduler.abort(waiting)
    assert request.finish_reason == "aborted" and not scheduler.has_work()
    assert cache.free_pages() == [64, 64] and cache.tables.slots.free_slots == 4


def test_draws_are_a_function_of_seed_and_count():
    values = [rng.draw(5, k) for k in range(1000)]
    assert all(0.0 <= v < 1.0 for v in values) and len(set(values)) > 990
    assert values[:3] == [rng.draw(5, 0), rng.draw(5, 1), rng.draw(5, 2)] and rng.draw(6, 0) != values[0]
    assert 0.45 < sum(values) / len(values) < 0.55


def test_sampling_params_ranges():
    for bad in (dict(temperature=-0.1), dict(temperature=2.5), dict(temperature=float("nan")), dict(top_p=0.0),
                dict(top_p=1.5), dict(max_new_tokens=0)):
        with pytest.raises(ValueError):
            SamplingParams(**bad)
    assert SamplingParams(temperature=0.0).greedy and SamplingParams().top_p == 1.0 and SamplingParams().temperature == 1.0


def test_decode_plan_prefers_the_balanced_kernel_only_for_uneven_or_badly_filled_batches():
    """The host-side choice between the two decode attention kernels (no GPU needed: it is arithmetic)."""
    import kirai_b200  # noqa: F401
    from kirai_b200.csrc.ops import decode_plan

    assert decode_plan([4096], 8)[0] is False                      # one request: the split kernel has the lower fixed cost
    assert decode_plan([4096] * 8, 8)[0] is False                  # equal lengths that fill one wave
    uneven = [1024, 7168, 2048, 6000, 3000, 5000, 4000, 1500]
    assert decode_plan(uneven, 8)[0] is True                       # the longest request would set the split kernel's time
    assert decode_plan([n for n in uneven], 8, window=512)[0] is False  # a window makes them equal again
    balanced, splits = decode_plan([100_000] + [500] * 15, 8)
    assert balanced is True and splits >= 1
    assert decode_plan([], 8) == (False, 1)


def test_decode_crowd_plan_follows_the_measured_batches():
    """More (request, kv head) pairs than SMs: CTAs of 8 warps where a long request would set the time of smaller ones or one wave
    holds the batch, of 4 warps for many alike, ranges for a few very long ones; nothing else is taken."""
    from kirai_b200.csrc.ops import decode_crowd_plan

    assert decode_crowd_plan([1000] * 18, 8) is None                        # 144 CTAs fit the SMs
    assert decode_crowd_plan([1000] * 64, 8, head_dim=256) is None and decode_crowd_plan([1000] * 64, 8, group=16) is None
    assert decode_crowd_plan([1000] * 513, 8) is None and decode_crowd_plan([], 8) is None
    assert decode_crowd_plan([1000] * 32, 8) == (4, 1) and decode_crowd_plan([1000] * 64, 8) == (4, 1)
    uneven = [3000 - 2500 * i // 19 for i in range(20)]
    assert decode_crowd_plan(uneven, 8) == (8, 1)
    assert decode_crowd_plan(uneven, 8, reach=256) == (4, 1)                # a window makes them equal
    assert decode_crowd_plan([6000 - 5950 * i // 23 for i in range(24)], 8) == (4, 3)
    assert decode_crowd_plan([200_000] + [100] * 30, 8) is None             # equal ranges for all SMs


def test_products_with_chosen_experts_are_taken_where_they_were_measured_faster():
    """Every measured step whose two ways differ by more than a twentieth: (experts, top, width, expert size, rows behind the
    experts, tokens, us whole, first product chosen, both)."""
    import kirai_b200  # noqa: F401
    from kirai_b200.csrc.ops import linear_chosen_pays

    measured = [
        (16, 2, 4096, 1536, 0, 1, 102, 56, 32), (16, 2, 4096, 1536, 0, 3, 100, 68, 52), (16, 2, 4096, 1536, 0, 8, 101, 79, 71),
        (16, 2, 4096, 1536, 0, 12, 103, 93, 92), (16, 2, 4096, 1536, 0, 20, 110, 113, 116), (16, 2, 4096, 1536, 0, 32, 112, 117, 122),
        (16, 2, 4096, 1536, 0, 64, 121, 129, 135), (16, 2, 4096, 1536, 1536, 3, 111, 75, 60), (16, 2, 4096, 1536, 1536, 12, 114, 100, 96),
        (16, 2, 4096, 1536, 1536, 64, 129, 136, 142), (8, 2, 4096, 2048, 0, 1, 73, 47, 33), (8, 2, 4096, 2048, 0, 3, 73, 60, 55),
        (8, 2, 4096, 2048, 0, 12, 73, 75, 80), (8, 2, 4096, 2048, 0, 64, 85, 89, 94), (64, 4, 2048, 768, 0, 1, 102, 64, 35),
        (64, 4, 2048, 768, 0, 3, 103, 67, 48), (64, 4, 2048, 768, 0, 8, 104, 77, 73), (64, 4, 2048, 768, 0, 12, 105, 85, 90),
        (64, 4, 2048, 768, 0, 16, 107, 97, 108), (64, 4, 2048, 768, 0, 32, 123, 125, 147), (64, 4, 2048, 768, 0, 64, 139, 168, 197),
        (128, 8, 2048, 768, 0, 1, 191, 113, 57), (128, 8, 2048, 768, 0, 8, 195, 135, 125), (128, 8, 2048, 768, 0, 12, 197, 153, 158),
        (128, 8, 2048, 768, 0, 16, 201, 170, 189), (128, 8, 2048, 768, 0, 32, 229, 230, 274), (128, 8, 2048, 768, 0, 64, 273, 358, 416),
    ]
    for experts, top, width, ff, behind, tokens, whole, first, both in measured:
        share = 1.0 - (1.0 - top / experts) ** tokens
        up = linear_chosen_pays(tokens, experts, share, experts * 2 * ff + 2 * behind, width, 4 * experts * ff * width, False)
        down = linear_chosen_pays(tokens, experts, share, width, experts * ff + behind, 2 * experts * ff * width, True)
        if abs(first - whole) > 0.05 * whole:
            assert up == (first < whole), (experts, tokens)
        if abs(both - first) > 0.05 * whole:
            assert down == (both < first), (experts, tokens)
    assert not linear_chosen_pays(1, 8, 0.125, 2048, 64, 8 * 2 * 128 * 64 * 2, False)  # a small layer has nothing to save


def test_captured_steps_plan_for_the_heads_that_the_layers_have():
    """A captured step of more pairs than SMs takes the plan that an eager one takes: the crowd's kernel only where it serves the
    layers' groups and heads, and beside layers that it does not serve the plan that those would have without it."""
    from types import SimpleNamespace

    import kirai_b200  # noqa: F401
    from kirai_b200.csrc import ops
    from kirai_b200.engine.graphs import DecodeGraphs
    from kirai_b200.parts.attention import GQAttention
    from kirai_b200.parts.base import KVCacheNeed

    fake_ops = SimpleNamespace(decode_plan=ops.decode_plan, decode_crowd_plan=ops.decode_crowd_plan,
                               decode_crowd_serves=getattr(ops, "decode_crowd_serves", None), sm_count=lambda device: 148,
                               decode_cluster_room=lambda device, head_dim, group=4: (lambda cluster: 148 // cluster))

    def plan(needs, lens):
        cache = CacheManager(needs, page_size=16, num_pages=4, num_slots=1, device=None)
        graphs = DecodeGraphs(SimpleNamespace(rt=SimpleNamespace(ops=fake_ops, device="cuda:0"), cache=cache))
        return graphs._plan(lens)

    def attention(q_heads, kv_heads, head_dim, **more):
        return GQAttention("", 64, q_heads, kv_heads, head_dim, None, **more).cache_need()

    lens = [100 + 3000 * i // 63 for i in range(64)]
    crowd = ops.decode_crowd_plan(lens, 8)
    assert crowd is not None and ops.decode_plan(lens, 4)[0] is True
    assert plan([attention(32, 8, 128)] * 3, lens) == (False, 0, crowd)
    assert plan([attention(64, 4, 128)], lens) == (True, 0, None)            # 16 query heads to a kv head
    assert plan([attention(32, 8, 128), attention(32, 8, 256)], lens)[2] == crowd
    for other in (attention(128, 8, 128, window=4096), attention(16, 8, 256, window=4096), attention(8, 1, 128, window=4096)):
        both = plan([attention(32, 8, 128), other], lens)
        assert both == ((True, 0, crowd) if ops.decode_plan(lens, 8)[0] else (False, ops.decode_plan(lens, 8)[1], crowd))
    assert plan([attention(32, 8, 128), attention(128, 8, 128)], lens)[2] is None  # one pool, the larger group counts
    shared = attention(32, 8, 128).also_read_by(attention(128, 8, 128))                # a layer that reads another's pages
    assert shared == attention(32, 8, 128) and shared.group == 16 and plan([shared], lens)[2] is None
    assert attention(32, 8, 128).also_read_by(KVCacheNeed(8, 128, None)).group is None
    assert plan([KVCacheNeed(8, 128, None)], lens)[2] is None                # a mixer that does not say its group
    assert plan([attention(32, 8, 128)], [1000] * 18) == (False, ops.decode_plan([1000] * 18, 8)[1], None)


def test_a_step_plans_its_decode_attention_once_for_layers_alike(monkeypatch):
    """Layers of the same heads and reach share one plan of the step; other heads, another reach and changed lengths are
    planned for themselves, and the answers are those of the plans."""
    from types import SimpleNamespace

    from kirai_b200.csrc import ops

    calls = []
    crowd_plan, plan = ops.decode_crowd_plan, ops.decode_plan
    monkeypatch.setattr(ops, "decode_crowd_plan", lambda *a, **k: calls.append("crowd") or crowd_plan(*a, **k))
    monkeypatch.setattr(ops, "decode_plan", lambda *a, **k: calls.append("plan") or plan(*a, **k))
    room = lambda cluster: 148 // cluster  # noqa: E731
    for lens in ([1000] * 32, [200_000] + [100] * 30, [700, 900]):
        batch = SimpleNamespace(start_positions=[n - 1 for n in lens] + [5], query_lens=[1] * len(lens) + [9], decode_plans={})
        crowd = crowd_plan(lens, 8)
        expected = (crowd, False if crowd else plan(lens, 8, room=room)[0], max(lens))
        calls.clear()
        for _ in range(36):
            assert ops._decode_choice(batch, len(lens), 8, None, 148, room, 128, 4) == expected
        assert len(calls) <= 2
        assert ops._decode_choice(batch, len(lens), 8, 64, 148, room, 128, 4)[0] == crowd_plan(lens, 8, 64)
        assert ops._decode_choice(batch, len(lens), 2, None, 148, room, 256, 16) == (None, plan(lens, 2, room=room, head_dim=256, group=16)[0], max(lens))
        batch.start_positions[0] += 100_000
        assert ops._decode_choice(batch, len(lens), 8, None, 148, room, 128, 4)[2] == lens[0] + 100_000
        del batch.decode_plans
        assert ops._decode_choice(batch, len(lens), 8, None, 148, room, 128, 4)[2] == lens[0] + 100_000


def test_decode_plan_over_random_batches_respects_the_kernels_limits():
    """Whatever the batch, the planner names a split count that the decode kernel takes (1 to 64 ranges, never more
    ranges than key tiles), and ranges are merged inside the kernel only where the device said the clusters fit and
    the other CTAs' rows fit the first one's slots."""
    import random

    import kirai_b200  # noqa: F401
    from kirai_b200.csrc.ops import DECODE_CLUSTER_RANGES, decode_pair_merges, decode_plan, decode_splits

    rnd = random.Random(4)
    for _ in range(300):
        sms = rnd.choice([16, 66, 132, 148])
        counts = {1: sms, 2: sms // 2, 3: rnd.randint(0, sms // 3), 4: rnd.randint(0, sms // 4), 5: rnd.randint(0, sms // 5)}
        room = lambda cluster: counts.get(cluster, 0)  # noqa: E731
        kv_heads, group, head_dim = rnd.choice([1, 2, 8]), rnd.choice([1, 3, 4, 8, 16]), rnd.choice([64, 128, 256])
        lens = [rnd.randint(1, rnd.choice([40, 5000, 40000])) for _ in range(rnd.randint(1, 70))]
        window = rnd.choice([None, None, 512])
        balanced, splits = decode_plan(lens, kv_heads, window, sms=sms, room=room, head_dim=head_dim, group=group)
        longest = max(min(n, window) if window else n for n in lens)
        assert isinstance(balanced, bool) and 1 <= splits <= min(64, -(-longest // 16))
        assert splits == decode_splits(len(lens), kv_heads, longest, sms=sms, room=room, head_dim=head_dim, group=group)
        pairs = len(lens) * kv_heads
        for ranges in range(1, 9):
            merges = decode_pair_merges(pairs, ranges, head_dim, room, group)
            if merges:
                assert 2 <= ranges <= DECODE_CLUSTER_RANGES and pairs <= counts[ranges] and head_dim <= 128
                assert (ranges - 1) * group <= 16


def drive_random_workload(scheduler_class, seed):
    """A random workload (arrivals over time, stop tokens, aborts, few pages and slots) through a scheduler; the
    trace of every decision and of what was left at the end."""
    import random

    rnd = random.Random(seed)
    page_size, num_pages, slots = rnd.choice([2, 4, 8]), rnd.randint(6, 40), rnd.randint(1, 5)
    cache = CacheManager([KVCacheNeed(1, 8, None), KVCacheNeed(1, 8, 8)], page_size=page_size, num_pages=num_pages,
                         num_slots=slots, device=None)
    scheduler = scheduler_class(cache, max_batched_tokens=rnd.choice([4, 16, 33]), max_running=rnd.randint(1, 5), max_positions=512,
                                default_max_new_tokens=64, prefill_chunk=rnd.choice([None, 3, 8]))
    arrivals = [(rnd.randint(1, 40), rnd.randint(1, 12), rnd.randint(0, 30)) for _ in range(rnd.randint(1, 12))]
    trace, step, added = [], 0, 0
    while scheduler.has_work() or added < len(arrivals):
        while added < len(arrivals) and arrivals[added][2] <= step:
            prompt_len, new_tokens, _ = arrivals[added]
            added += 1
            try:
                scheduler.add(f"r{added}", list(range(prompt_len)), SamplingParams(temperature=0.0, max_new_tokens=new_tokens, eos_token_id=5))
            except AdmissionError:
                trace.append(("refused", added))
        step += 1
        if not scheduler.has_work():
            continue
        chosen = scheduler.schedule()  # always finds something to run: it raises if it is stuck
        for item in chosen:
            assert item.first == item.request.pages.length == item.request.computed
            cache.commit(item.request.pages, item.count)
        sampled = [(5 if rnd.random() < 0.05 else 7) if item.sample else None for item in chosen]
        trace.append([(item.request.request_id, item.first, item.count, item.sample) for item in chosen])
        trace.append(("finished", sorted(r.request_id for r in scheduler.update(chosen, sampled))))
        if rnd.random() < 0.03 and scheduler.running:
            victim = rnd.choice(scheduler.running)
            scheduler.abort(victim)
            trace.append(("abort", victim.request_id))
        cache.tables.check_consistency()
        assert step < 5000
    trace.append(("left", cache.free_pages(), cache.tables.slots.free_slots, dict(scheduler.stats)))
    return trace, scheduler.stats["preemptions"]


def test_native_scheduler_decides_as_the_python_model_does():
    """The scheduler in native code (the one the engine uses) against the Python class, step by step, on random
    workloads that admit, cut prompts, evict, recompute, stop, abort and refuse."""
    from kirai_b200.engine.scheduler import NativeScheduler

    evictions = 0
    for seed in range(150):
        expected, preempted = drive_random_workload(Scheduler, seed)
        got, _ = drive_random_workload(NativeScheduler, seed)
        assert got == expected, f"seed {seed}"
        evictions += preempted
    assert evictions > 20  # the workloads do run out of pages


@pytest.mark.parametrize("tokens,good", [([0, 5, 99], True), ([3, -1], False), ([100], False), ([5] * 40 + [1 << 70], False), ((7, 8), True)])
def test_a_steps_tokens_are_checked_as_an_array(tokens, good):
    from kirai_b200.engine.batch import StepEntry
    from kirai_b200.engine.step import StepError, check_entries

    cache = CacheManager([KVCacheNeed(1, 8, None)], page_size=4, num_pages=64, num_slots=2, device=None)
    entries = [StepEntry(cache.open("a"), tokens, [])]
    if good:
        assert check_entries(entries, 100, None)[0].tolist() == list(tokens)
    else:
        with pytest.raises(StepError, match="outside vocab size 100"):
            check_entries(entries, 100, None)
