"""The kernel library without a device: every call returns at once and every tensor is a
tensor without storage.

Running the model's own forward pass on it costs microseconds and touches no memory, but it
asks the workspace for exactly the tensors a real step asks for, in the same order and with
the same lifetimes.  That is how the step workspace of the arena is sized: not by a formula
kept beside the model, but by the model's code itself (cpmcu_b200.memory.Workspace counts the
bytes).  The reference sizes its activation area by adding up the layers' ``init_output_ptr``
offsets for ``chunk_length`` tokens (src/model/model.cuh:103-120).
"""
from __future__ import annotations

from typing import List, Optional, Sequence, Tuple

import torch

from ..memory import Arena, Workspace
from ..parts.base import StepContext
from .ops import BF16, F32, Ops, PREFILL_TILE_ROWS


class _NoLibrary:
    """Stands in for the compiled library: every entry point "launches" successfully."""

    @staticmethod
    def cpm_decode_attention_scratch_floats(n_seqs, n_heads, n_kv, d, n_splits):
        return n_seqs * n_kv * ((n_heads // n_kv + 15) // 16) * n_splits * (16 * d + 32)

    @staticmethod
    def cpm_decode_attention_blocks_per_sm(d):
        return 2 if d == 64 else 1

    @staticmethod
    def cpm_select_blocks_scratch_floats(n_tokens, n_kv, max_entries, n_slices):
        return n_tokens * n_kv * (max_entries * 16 + n_slices * 32)

    @staticmethod
    def cpm_latent_attention_scratch_floats(n_tokens, n_heads, rank, n_splits):
        return 0 if n_splits <= 1 else n_tokens * ((n_heads + 15) // 16) * n_splits * 16 * (rank + 2)

    @staticmethod
    def cpm_mingru_summary_floats(n_tiles, width):
        return n_tiles * 3 * width

    @staticmethod
    def cpm_retention_tiles_scratch_floats(n_tiles, heads, d, dv):
        return n_tiles * heads * d * dv

    @staticmethod
    def cpm_retention_step_sizes(d, dv):
        return 1

    @staticmethod
    def cpm_moe_expert_product_kernels(*args):
        return 1

    @staticmethod
    def cpm_sink_attention_bf16_sizes(d, dv):
        return int(d in (32, 64, 96, 128) and dv in (32, 64, 96, 128))

    @staticmethod
    def cpm_listed_attention_tcgen05_max_pages():
        return 11808

    def __getattr__(self, name):
        return lambda *args: 0


class DryOps(Ops):
    def __init__(self, dtype: torch.dtype, sm_count: int = 148):
        if dtype not in (torch.float32, torch.bfloat16):
            raise ValueError(f"compute dtype must be float32 or bfloat16, got {dtype}")
        self.dtype = dtype
        self.code = F32 if dtype == torch.float32 else BF16
        self.device = torch.device("meta")
        self.lib = _NoLibrary()
        self.element_size = 4 if dtype == torch.float32 else 2
        self.sm_count = sm_count
        self.arrivals = None
        self.use_tcgen05 = self.use_tcgen05_attention = self.use_tcgen05_listed = self.use_tcgen05_sink = True
        self.tcgen05_pair = False
        arena = Arena(None, None)
        self.workspace = Workspace(arena.carve("persistent", None), [arena.carve("frame0", None), arena.carve("frame1", None)])
        self.weights = None

    # no device, no checks
    @staticmethod
    def _stream():
        return 0

    def _act(self, t, what):
        return t

    @staticmethod
    def _i32(t, what):
        return t

    @staticmethod
    def _f32(t, what):
        return t

    def set_page_limit(self, n_pages):
        pass

    def _library_bmm(self, a, w, c):          # (the fp32 form has no kernel for tensors without storage)
        pass

    kept_bytes = 0      # what the parts asked to keep for good, each tensor rounded up to the arena's alignment

    def keep(self, t):
        from ..memory import round_up
        self.kept_bytes += round_up(t.numel() * t.element_size())
        return t

    def result(self, *shape, dtype=None):
        return torch.empty(*shape, dtype=dtype or self.dtype, device="meta")


def measure_weights(spec, dtype: torch.dtype) -> int:
    """Bytes of the tensors a model's parts keep for good once loaded (fused and widened copies included, which the
    declared shapes do not show), counted by loading tensors without storage; vectors as 32-bit, the most they can be."""
    from ..models.model import Model

    ops = DryOps(dtype)
    model = Model(spec, ops)
    model.load_weights({name: torch.empty(w.shape, device="meta",
                                          dtype=torch.int32 if w.role == "table" else (dtype if w.role == "matrix" else torch.float32))
                        for name, w in model.weight_specs().items()})
    return ops.kept_bytes


def _meta(n: int) -> torch.Tensor:
    return torch.empty(n, dtype=torch.int32, device="meta")


def dry_context(q_lens: Sequence[int], max_kv_len: int, cache, decode: bool, captured: bool = False,
                n_tiles: Optional[int] = None) -> StepContext:
    """A step that brings ``q_lens`` tokens of its sequences, on tensors without storage.  ``n_tiles``: as many query tiles
    instead of the portions' own (a recorded step has room for those of any portions, and takes its longest to be all tokens)."""
    n_tokens, n_seqs = sum(q_lens), len(q_lens)
    ctx = StepContext(
        n_tokens=n_tokens, n_seqs=n_seqs, is_decode=decode, captured=captured, q_lens=[n_tokens] if captured and not decode else list(q_lens),
        kv_lens=[] if captured else [max_kv_len] * n_seqs, slots=[] if captured else list(range(n_seqs)),
        max_q_len=n_tokens if captured and not decode else max(q_lens), max_kv_len=max_kv_len, token_ids=_meta(n_tokens),
        positions=_meta(n_tokens), token_seq=_meta(n_tokens), cu_q=_meta(n_seqs + 1), kv_len_dev=_meta(n_seqs), slot_dev=_meta(n_seqs),
        cache=cache)
    if n_tiles is None:
        n_tiles = sum((n + PREFILL_TILE_ROWS - 1) // PREFILL_TILE_ROWS for n in q_lens)
    ctx.q_tiles = (_meta(n_tiles), _meta(n_tiles), n_tiles)
    ctx.extras["step_begun"] = True
    return ctx


def _evenly(n_tokens: int, n_seqs: int) -> List[int]:
    base, extra = divmod(n_tokens, n_seqs)
    return [base + (1 if i < extra else 0) for i in range(n_seqs)]


def _most_tiles(n_tokens: int, most_seqs: int, longest: int) -> List[int]:
    """The portions of a step of ``n_tokens`` tokens that need most query tiles while one of them has ``longest`` tokens or more: as many
    sequences of one token as there may be, and the rest."""
    ones = max(0, min(most_seqs - 1, n_tokens - longest))
    return [1] * ones + [n_tokens - ones]


def _half_full_tiles(n_tokens: int, most_seqs: int) -> List[int]:
    """The same while the tiles are half full on average (what ``Ops.recurrence_by_tiles`` asks for)."""
    ones = 0
    while ones + 1 < most_seqs and 32 * (ones + 1 + (n_tokens - ones - 1 + PREFILL_TILE_ROWS - 1) // PREFILL_TILE_ROWS) <= n_tokens:
        ones += 1
    return [1] * ones + [n_tokens - ones]


def workspace_steps(max_step_tokens: int, max_batch: int, max_seq_tokens: int, packed_pieces: int = 0, sm_count: int = 148):
    """The steps a workspace is measured with: (portions, keys of the longest sequence, decode, captured, query tiles or None).

    Which step needs most room differs from part to part.  Most tensors grow with the step's tokens; the scratch of parts that go
    by query tiles with their number, which is largest when one portion is long and the others have one token (as many of these as
    the part's rule allows); the scratch of
    shared-out keys, and the plain copies that narrow products make, are largest just below the number of tokens where a
    kernel that needs none takes over (or the last step down of the number of shares); block-sparse attention needs other tensors below its threshold than above.
    ``max_batch`` counts up to the next power of two, as the workspace lets steps through.  ``packed_pieces``: sequences of a recorded
    chunk of several prompts (0: none is recorded)."""
    T, b = int(max_step_tokens), 1
    while b < max_batch:
        b *= 2
    steps = []
    # (a step of an eighth of the tokens fits wherever the full one does, whatever its scratch)
    for n in sorted({T, max(1, T // 2)} | {p for p in (512, 256, 255, 3 * sm_count // 2, 128, 95, 64, 63) if T > p > T // 8}):
        if n in (T, max(1, T // 2)):
            steps.append((_evenly(n, min(n, max_batch)), max_seq_tokens, False, False, None))
        uneven = {tuple(_most_tiles(n, b, longest)) for longest in (Ops.RETENTION_TILE_MIN_TOKENS, Ops.MINGRU_TILE_MIN_TOKENS)}
        uneven.add(tuple(_half_full_tiles(n, b)))
        for portions in sorted(uneven - {(n,)}):
            steps.append((list(portions), max_seq_tokens, False, False, None))
        for kv in {min(max(n, k), max_seq_tokens) for k in (0, 8192)} | {max_seq_tokens}:
            steps.append(([n], kv, False, False, None))
    if packed_pieces:
        steps.append(([T], max_seq_tokens, False, True, None))
        if b >= packed_pieces + 1 and T > packed_pieces:
            steps.append((_evenly(T, packed_pieces + 1), max_seq_tokens, False, True, T // PREFILL_TILE_ROWS + packed_pieces))
    for size in sorted({b, max(1, b // 2), max(1, b // 4), min(b, 8), 1}):      # captured decode steps; eager ones of as many sequences
        steps.append(([1] * size, max_seq_tokens, True, True, None))
    steps.append(([1] * max(1, b - 1), 1, True, False, None))
    for size in sorted({max_batch, b, max(1, b - 1)}):
        steps.append(([1] * size, max_seq_tokens, True, False, None))
    return steps


def measure_workspace(spec, dtype: torch.dtype, max_step_tokens: int, max_batch: int, max_seq_tokens: int,
                      sm_count: int = 148) -> Tuple[int, int, List[str]]:
    """(bytes of the persistent part, bytes of one frame, notes) that the steps of a model need at most: prompts of up to
    ``max_step_tokens`` packed tokens and decode steps of up to ``max_batch`` sequences (see ``workspace_steps``), each run once on
    tensors without storage.  A part that cannot run that way (it reads values on the host) is left out of the
    measurement; what it allocates comes from torch's allocator anyway, and the note says so."""
    from ..cache import Cache
    from ..engine.step import MAX_GRAPH_PIECES
    from ..models.model import Model

    ops = DryOps(dtype, sm_count)
    model = Model(spec, ops)
    model.load_weights({name: torch.empty(w.shape, device="meta", dtype=torch.int32 if w.role == "table" else dtype)
                        for name, w in model.weight_specs().items()})
    per_seq = max(64, int(max_seq_tokens))
    cache = Cache(model.cache_needs(), max_tokens=per_seq, dtype=dtype, device="meta", n_slots=max(2, max_batch + 1),
                  max_seq_tokens=per_seq, max_step_tokens=max_step_tokens)
    recorded = model.recordable_prompt()
    notes: List[str] = []
    for q_lens, kv, decode, captured, n_tiles in workspace_steps(max_step_tokens, max_batch, per_seq, MAX_GRAPH_PIECES if recorded else 0, sm_count):
        n_tokens = sum(q_lens)
        ops.workspace.begin_step()
        try:
            ctx = dry_context(q_lens, kv, cache, decode, captured, n_tiles)
            rows = ops.empty(n_tokens, dtype=torch.int32)                  # the step's descriptor: ids, positions, ...
            ops.empty(8 * n_tokens + 4 * len(q_lens) + 64, dtype=torch.int32)
            model.forward(ctx, rows)
        except Exception as e:                                            # a part that needs real values
            note = f"a part could not be measured without a device ({type(e).__name__}: {str(e)[:80]})"
            if note not in notes:
                notes.append(note)
    persistent, frame = ops.workspace.peaks()
    return persistent, frame, notes
