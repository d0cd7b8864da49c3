"""The arena and its regions, the workspace's lifetimes, the sizing of the storage and its errors, without a device."""
import pytest
import torch

from cpmcu_b200.cache import Cache, CacheFull
from cpmcu_b200.memory import ALIGN, Arena, PoolExhausted, Staging, Workspace, plan_storage
from cpmcu_b200.parts.base import CacheNeeds
from tests import configs, dinutar_cases, kipizen_cases, reravik_cases


def test_regions_are_carved_in_order_and_name_themselves_when_full():
    arena = Arena(64 * 1024, "cpu")
    w = arena.carve("weights", 10_000)
    c = arena.carve("cache", 40_000)
    assert w.offset == 0 and c.offset == w.size and w.size % ALIGN == 0
    a = w.tensor((100,), torch.float32)
    b = w.tensor((3, 5), torch.bfloat16, zero=True)
    assert a.data_ptr() % ALIGN == 0 and b.data_ptr() % ALIGN == 0 and b.data_ptr() >= a.data_ptr() + 400
    assert float(b.float().abs().sum()) == 0.0
    a.fill_(7.0)
    assert arena.buffer[:400].view(torch.float32).tolist() == [7.0] * 100            # a view of the one allocation
    with pytest.raises(PoolExhausted, match="region 'weights'") as e:
        w.tensor((10_000,), torch.float32, what="a tensor too many")
    assert e.value.region == "weights" and "a tensor too many" in str(e.value)
    with pytest.raises(PoolExhausted, match="region 'arena'"):
        arena.carve("more", 30_000)
    assert arena.report()["weights"][1] == w.peak


def test_workspace_frames_alternate_and_the_step_is_checked_before_it_runs():
    arena = Arena(1 << 20, "cpu")
    ws = Workspace(arena.carve("workspace", 4096), [arena.carve("frame0", 8192), arena.carve("frame1", 8192)],
                   sized_tokens=64, sized_seqs=4)
    ws.begin_step()
    x = ws.alloc((16,), torch.float32)                       # persistent: lives through the step
    ws.begin_layer(0)
    f0 = ws.alloc((100,), torch.float32)
    f0.fill_(1.0)
    ws.begin_layer(1)
    f1 = ws.alloc((100,), torch.float32)
    f1.fill_(2.0)
    assert float(f0.sum()) == 100.0                          # layer 0's output is intact while layer 1 runs
    ws.begin_layer(2)
    g0 = ws.alloc((100,), torch.float32)
    assert g0.data_ptr() == f0.data_ptr() and float(f1.sum()) == 200.0      # layer 2 takes layer 0's place, not layer 1's
    ws.end_layers()
    y = ws.alloc((16,), torch.float32)
    assert y.data_ptr() > x.data_ptr()
    with pytest.raises(PoolExhausted, match="region 'frame1'"):
        ws.begin_layer(3)
        ws.alloc((4096,), torch.float32)
    ws.require(64, 4)
    with pytest.raises(PoolExhausted, match="128 tokens.*sized for 64"):
        ws.require(128, 1)                                   # a chunk larger than the workspace was sized for
    with pytest.raises(PoolExhausted, match="sequences"):
        ws.require(8, 8)
    assert ws.peaks()[1] >= 400


def test_plan_storage_says_what_does_not_fit():
    def cache_bytes(tokens):                                 # 1 KiB per token and a table that grows with it
        return tokens * 1024 + tokens // 64 * 4 * 10

    tokens, total = plan_storage(10 << 20, 2 << 20, 1 << 20, cache_bytes, None)
    assert tokens % 64 == 0 and cache_bytes(tokens) <= (10 << 20) - (3 << 20) and cache_bytes(tokens + 128) > (7 << 20) - 64 * ALIGN - 200_000
    tokens, total = plan_storage(None, 2 << 20, 1 << 20, cache_bytes, 1000)
    assert tokens == 960 and total >= (3 << 20) + cache_bytes(960)
    with pytest.raises(PoolExhausted, match="region 'cache'.*two pages"):            # memory_limit too small for any cache
        plan_storage((3 << 20) + 64 * ALIGN + 50_000, 2 << 20, 1 << 20, cache_bytes, None)
    with pytest.raises(PoolExhausted, match="region 'weights'"):
        plan_storage(1 << 20, 2 << 20, 1 << 20, cache_bytes, None)
    with pytest.raises(PoolExhausted, match="region 'workspace'"):
        plan_storage(5 << 19, 2 << 20, 1 << 20, cache_bytes, None)
    with pytest.raises(PoolExhausted, match="do not fit the memory limit"):
        plan_storage(4 << 20, 2 << 20, 1 << 20, cache_bytes, 4096)


def test_workspace_is_measured_by_the_models_own_forward_pass():
    from cpmcu_b200.ops.dry import measure_workspace
    from cpmcu_b200.registry import architecture

    arch = architecture("MiniCPMForCausalLM")
    sizes = {}
    for name, cfgd in (("a", configs.tiny_a()), ("b", configs.tiny_b())):
        spec = arch.model_spec(arch.config_class.from_dict(cfgd))
        for chunk in (64, 256):
            p, f, notes = measure_workspace(spec, torch.bfloat16, chunk, 4, 1024)
            assert notes == [] and p > 0 and f > 0
            sizes[(name, chunk)] = (p, f)
        # four times the tokens: up to four times the frame (per-token tensors, plus padding and scratch that do not grow)
        if name == "a":
            assert 2.0 < sizes[(name, 256)][1] / sizes[(name, 64)][1] < 4.5
        else:       # the sparse model's largest tensor is the block selection's scratch for steps of few tokens
            assert sizes[(name, 256)][1] >= sizes[(name, 64)][1]
    p32, f32, _ = measure_workspace(arch.model_spec(arch.config_class.from_dict(configs.tiny_a())), torch.float32, 64, 4, 1024)
    assert f32 > sizes[("a", 64)][1]
    # a frame holds at least the widest tensor of a layer: the gate_up product of 64 tokens
    assert sizes[("a", 64)][1] >= 64 * 176 * 2


def _need(spec, dtype, portions, max_kv_len, chunk, max_batch):
    """Bytes (persistent, frame) that one step asks for."""
    from cpmcu_b200.cache import Cache as AnyCache
    from cpmcu_b200.models.model import Model
    from cpmcu_b200.ops.dry import DryOps, dry_context

    ops = DryOps(dtype)
    model = Model(spec, ops)
    model.load_weights({name: torch.empty(w.shape, device="meta", dtype=torch.int32 if w.role == "table" else dtype)
                        for name, w in model.weight_specs().items()})
    cache = AnyCache(model.cache_needs(), max_tokens=16384, dtype=dtype, device="meta", n_slots=max_batch + 1, max_seq_tokens=16384,
                     max_step_tokens=chunk)
    ops.workspace.begin_step()
    n = sum(portions)
    ctx = dry_context(portions, max_kv_len, cache, all(q == 1 for q in portions))
    rows = ops.empty(n, dtype=torch.int32)
    ops.empty(8 * n + 4 * len(portions) + 64, dtype=torch.int32)
    model.forward(ctx, rows)
    return ops.workspace.peaks()


@pytest.mark.parametrize("arch_name,config,chunk,max_batch", [
    ("Kipizen", kipizen_cases.config_wide_state, 300, 64), ("Kipizen", kipizen_cases.config_wide_state, 2048, 64),
    ("Kipizen", kipizen_cases.config_wide_state, 2048, 5), ("Kipizen", kipizen_cases.config_d, 64, 200),
    ("Dinutar", dinutar_cases.config_d, 300, 64), ("Dinutar", dinutar_cases.config_a, 2048, 33), ("Reravik", reravik_cases.config_a, 300, 5),
    ("MiniCPMForCausalLM", configs.tiny_b, 300, 64), ("MiniCPMForCausalLM", configs.tiny_e, 64, 200),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_no_step_needs_more_than_the_workspace_is_measured_for(arch_name, config, chunk, max_batch, dtype):
    """Steps of portions as uneven as they come, of fewer tokens than a chunk, over short and long histories, and decode steps
    between the buckets, against what storage gives a frame (the measured bytes, a twentieth and 1 MiB more)."""
    from cpmcu_b200.ops.dry import measure_workspace
    from cpmcu_b200.registry import architecture

    arch = architecture(arch_name)
    spec = arch.model_spec(arch.config_class.from_dict(config()))
    persistent, frame, notes = measure_workspace(spec, dtype, chunk, max_batch, 16384)
    assert notes == []
    given = (int(persistent * 1.05) + (1 << 20), int(frame * 1.05) + (1 << 20))
    bucket = 1
    while bucket < max_batch:
        bucket *= 2
    steps = []
    for n in {chunk, chunk - 1, chunk // 2 + 3, min(chunk, 254), min(chunk, 95), min(chunk, 61)}:
        for seqs in {1, 2, max_batch, bucket, (bucket + 1) // 2}:
            ones = min(seqs, n) - 1
            steps.append([1] * ones + [n - ones])                                        # one long portion among single tokens
            few = min(seqs, n // 8)
            if few > 1:
                steps.append([8] * (few - 1) + [n - 8 * (few - 1)])
            if seqs * 65 <= n:
                steps.append([65] * (seqs - 1) + [n - 65 * (seqs - 1)])                    # a tile and one token each
            if seqs <= n:
                steps.append([n // seqs + (i < n % seqs) for i in range(seqs)])
    steps += [[1] * n for n in {1, 3, max_batch, bucket, max(1, bucket - 1), (bucket * 3 + 3) // 4}]
    for portions in steps:
        for kv in (max(portions), 4000, 16384):
            need = _need(spec, dtype, portions, max(kv, max(portions)), chunk, bucket)
            assert need[0] <= given[0] and need[1] <= given[1], (portions[:3], max(portions), len(portions), kv)


def test_cache_inside_regions():
    needs = [CacheNeeds(kv_heads=2, head_dim=16), CacheNeeds(kv_heads=1, head_dim=32, state={"s": ((8,), torch.float32)})]
    counting = Arena(None, None)
    st, pg = counting.carve("state", None), counting.carve("cache", None)
    Cache(needs, max_tokens=64 * 8, dtype=torch.float32, device="meta", n_slots=4, state_region=st, page_region=pg)
    assert pg.peak >= 8 * 64 * (2 * 2 * 16 + 2 * 32) * 4 and st.peak >= 2 * 4 * 8 * 4
    arena = Arena(st.peak + pg.peak + 64 * ALIGN, "cpu")
    c = Cache(needs, max_tokens=64 * 8, dtype=torch.float32, device="cpu", n_slots=4,
              state_region=arena.carve("state", st.peak + 16 * ALIGN), page_region=arena.carve("cache", pg.peak + 16 * ALIGN))
    lo, hi = arena.buffer.data_ptr(), arena.buffer.data_ptr() + arena.total
    for lane in c.lanes:
        for t in (lane.k, lane.v, lane.page_table, *lane.state.values()):
            assert lo <= t.data_ptr() < hi
    s = c.open_sequence()
    c.reserve(s, 200)
    c.set_length(s, 200)
    c.check_consistent()
    with pytest.raises(CacheFull):
        c.reserve(s, 64 * 9)
    small = Arena(1 << 20, "cpu")
    with pytest.raises(PoolExhausted, match="region 'cache'.*key-value pages"):
        Cache(needs, max_tokens=64 * 64, dtype=torch.float32, device="cpu", n_slots=4,
              state_region=small.carve("state", 1 << 16), page_region=small.carve("cache", 1 << 18))


def test_guard_words_show_which_region_was_overrun():
    arena = Arena(64 * 1024, "cpu", guards=True)
    a = arena.carve("frame0", 1024)
    b = arena.carve("frame1", 1024)
    assert b.offset == a.offset + a.size + ALIGN            # a guard lies between them
    t = a.tensor((256,), torch.float32)
    t.fill_(1.0)
    arena.check_guards()
    arena.buffer[a.offset + a.size + 3] = 0                 # one byte past frame0's end
    with pytest.raises(RuntimeError, match="behind region 'frame0'.*byte 3"):
        arena.check_guards()


def test_opened_slots_are_cleared_together_and_others_left():
    """Neighbouring and scattered slots: their state is zeros, the rest of the state as it was."""
    c = Cache([CacheNeeds(state={"s": ((3,), torch.float32)})], max_tokens=64 * 8, dtype=torch.float32, device="cpu", n_slots=7)
    first = c.open_sequences(6)
    assert first == [0, 1, 2, 3, 4, 5]
    state = c.lanes[0].state["s"]
    state.fill_(5.0)
    for s in (1, 3, 4):
        c.close_sequence(s)
    assert c.open_sequences(3) == [1, 3, 4]
    assert [float(r.sum()) for r in state] == [15.0, 0.0, 15.0, 0.0, 0.0, 15.0, 15.0]


@pytest.mark.parametrize("n,sizes", [(5, [3]), (5, [2, 2]), (3, [5]), (0, [1]), (4, []), (6, [2, 0, 5])])
def test_staged_copies_need_parts_of_the_sources_size(n, sizes):
    """Refused before anything is copied, as a plain copy between unequal shapes is."""
    parts = [torch.full((m,), 7, dtype=torch.int32) for m in sizes]
    with pytest.raises(RuntimeError, match=f"{n} numbers"):
        Staging(torch.device("cpu")).copy(torch.arange(n, dtype=torch.int32), parts)
    assert all(p.tolist() == [7] * p.numel() for p in parts)


@pytest.mark.parametrize("at,nbytes,shape", [(0, 16, (100,)), (0, 400, (99,)), (3600, 512, (128,)), (4096, 4, (1,)), (3840, 256, (65,))])
def test_a_view_lies_inside_the_arena_and_is_as_long_as_its_shape(at, nbytes, shape):
    arena = Arena(4096, "cpu")
    with pytest.raises(RuntimeError):
        arena.view(at, nbytes, shape, torch.float32, False)
    assert arena.view(3840, 256, (64,), torch.float32, True).tolist() == [0.0] * 64           # the last bytes
    assert arena.view(4096, 0, (0, 3), torch.bfloat16, True).shape == (0, 3)


def test_a_groups_page_table_is_brought_up_to_date_by_itself():
    """A group may be asked without the cache around it, as ever."""
    c = Cache([CacheNeeds(kv_heads=1, head_dim=4)], max_tokens=64 * 8, dtype=torch.float32, device="cpu", n_slots=2)
    for slot, tokens in zip(c.open_sequences(2), (130, 64)):
        c.reserve(slot, tokens)
    c.groups[0].sync()
    assert [row.tolist()[:3] for row in c.groups[0].page_table] == [c.groups[0].pages_of_slot[0], c.groups[0].pages_of_slot[1] + [0, 0]]
