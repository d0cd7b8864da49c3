"""The decode runner against the plain implementation at the level of logits.

Generation, the command line, the smoke run and the benchmark reach the model through
``DecodeRunner`` (fixed device buffers per bucket, padding entries, optionally a CUDA graph),
not through ``Stepper.step``.  Here the runner is fed the tokens of given sequences and the
logits of every step are compared with the plain implementation's: with and without a graph,
in 32-bit and in bfloat16, with buckets that hold padding entries, a bucket of 64, and batches
that shrink twice as sequences end."""
import pytest
import torch

from tests import configs, helpers

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
CONFIGS = {"tiny_a": (configs.tiny_a, 0), "tiny_b": (configs.tiny_b, 1), "tiny_e": (configs.tiny_e, 4)}


def _stepper(folder, dtype, max_tokens, chunk=64, n_slots=None):
    from cpmcu_b200.cache import Cache
    from cpmcu_b200.engine import Stepper
    from cpmcu_b200.loading import load_model

    _, cfg, model = load_model(folder, dtype)
    cache = Cache(model.cache_needs(), max_tokens, DT[dtype], "cuda:0", n_slots=n_slots, max_step_tokens=chunk)
    return cfg, Stepper(model, cache, chunk_tokens=chunk)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["tiny_a", "tiny_b", "tiny_e"])
def test_runner_logits_with_padding_and_shrinking_batches(model_folders, name, dtype, graph):
    """Three sequences in a bucket of four (one padding entry); they end after 5, 12 and 20 decode steps, so the
    runner is restarted on two (a full bucket of two) and on one."""
    make, seed = CONFIGS[name]
    folder = model_folders(name, make(), seed, dtype)
    cfg, st = _stepper(folder, dtype, 64 * 16)
    lens, extra = (70, 9, 33), (5, 20, 12)
    seqs = [helpers.random_ids(cfg.vocab_size, L + e, 50 + L) for L, e in zip(lens, extra)]
    helpers.record_blocks(st)                    # eager steps leave their block choices: every sparse row is compared
    rows_seen = []

    def check(i, rows, positions, blocks):
        assert positions == list(range(lens[i] - 1, lens[i] + extra[i]))
        helpers.check_rows(rows, folder, seqs[i], positions, dtype, label=(name, i), blocks=blocks)
        rows_seen.append(len(positions))

    steps = helpers.runner_parity(st, seqs, lens, check, graph)
    assert steps == 20 and sum(rows_seen) == 3 + sum(extra)
    st.cache.check_consistent()
    assert st.cache.tokens_held() == 0


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_runner_logits_bucket_of_64(model_folders, dtype, graph):
    """64 short sequences of tiny A in one bucket; 24 leave after two steps (40 live in a bucket of 64), 20 more
    after four (20 live in a bucket of 32), the rest after six."""
    folder = model_folders("tiny_a", configs.tiny_a(), 0, dtype)
    cfg, st = _stepper(folder, dtype, 64 * 70, n_slots=70)
    lens = [3 + (7 * i) % 38 for i in range(64)]
    extra = [2 if i < 24 else 4 if i < 44 else 6 for i in range(64)]
    seqs = [helpers.random_ids(cfg.vocab_size, L + e, 900 + i) for i, (L, e) in enumerate(zip(lens, extra))]
    count = [0]

    def check(i, rows, positions, blocks):
        helpers.check_rows(rows, folder, seqs[i], positions, dtype, label=i)
        count[0] += len(positions)

    assert helpers.runner_parity(st, seqs, lens, check, graph) == 6
    assert count[0] == 64 + sum(extra)
    st.cache.check_consistent()


@pytest.mark.parametrize("sizes", [[5, 0, 7], [8192, 1], [70_000, 3, 20_000]])
def test_staged_copies_arrive_whole_behind_a_busy_stream(sizes):
    """Three times round the ring of pinned buffers while the stream is busy: every copy holds what the host array held when it was
    queued, in arrays smaller than a buffer, as large and larger."""
    from cpmcu_b200.memory import Staging

    staging, n = Staging(torch.device("cuda:0")), sum(sizes)
    a = torch.randn(4096, 4096, device="cuda:0")
    outs = []
    for i in range(3 * Staging.BUFFERS + 1):
        a = torch.tanh(a @ a)                                  # milliseconds of work in front of each copy
        host = torch.arange(n, dtype=torch.int32) * (i + 1)
        parts = [torch.zeros(s, dtype=torch.int32, device="cuda:0") for s in sizes]
        staging.copy(host, parts)
        host.zero_()                                           # the caller's array is its own again
        outs.append(parts)
    for i, parts in enumerate(outs):
        assert torch.equal(torch.cat(parts).cpu(), torch.arange(n, dtype=torch.int32) * (i + 1)), i


def test_a_staged_copy_that_fails_leaves_its_buffer_to_the_copies_before_it():
    """The second of two parts has another shape and is refused: the first part's copy is queued by then, and its buffer
    is not written again before that copy is over."""
    from cpmcu_b200.memory import Staging

    staging, n = Staging(torch.device("cuda:0")), 4096
    staging.copy(torch.zeros(1, dtype=torch.int32), [torch.empty(1, dtype=torch.int32, device="cuda:0")])
    torch.cuda.synchronize()
    a = torch.randn(8192, 8192, device="cuda:0")
    for _ in range(8):
        a = torch.tanh(a @ a)                                  # tens of milliseconds of work in front of the copies
    first = torch.zeros(n, dtype=torch.int32, device="cuda:0")
    with pytest.raises(RuntimeError):
        staging.copy(torch.arange(n + 6, dtype=torch.int32), [first, torch.empty(2, 3, dtype=torch.int32, device="cuda:0")])
    for _ in range(Staging.BUFFERS):                           # once round the ring, over the same buffer
        staging.copy(torch.full((n,), -1, dtype=torch.int32), [torch.empty(n, dtype=torch.int32, device="cuda:0")])
    assert torch.equal(first.cpu(), torch.arange(n, dtype=torch.int32))


def test_a_staged_copy_is_refused_under_capture():
    """As a copy out of ordinary memory is: a replay would read a buffer that holds other copies' numbers by then.  The ring goes on."""
    from cpmcu_b200.memory import Staging

    staging, part = Staging(torch.device("cuda:0")), torch.zeros(5, dtype=torch.int32, device="cuda:0")
    for i in range(3):
        staging.copy(torch.full((5,), i, dtype=torch.int32), [part])
        with pytest.raises(RuntimeError, match="captured"):
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                part.add_(0)
                staging.copy(torch.full((5,), 9, dtype=torch.int32), [part])
        assert part.tolist() == [i] * 5
