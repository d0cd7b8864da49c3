"""The norms of whole rows at the borders of their kernels, against 64-bit results: rows in registers (one, two and four groups of four
columns a thread, a last group that is not full, one warp and sixteen), rows in shared memory (too wide, or too many of them),
and the 32-bit path's promise that a row does not depend on what else is in the step."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
# fp32: sums of up to 8,196 squares and one division: a few roundings of 2^-24 of values up to five standard deviations; bf16: one rounding of a
# result up to eight
TOL = {"float32": 2e-5, "bfloat16": 8 * 2.0 ** -8}
# widths around one, two and four groups a thread (2,048, 4,096, 8,192); row counts around the limits for many wide rows
SIZES = [(3, 132), (5, 2044), (5, 2048), (5, 2052), (4, 4096), (3, 4100), (3, 6148), (4, 8192), (3, 8196), (512, 2048), (513, 2048), (200, 8192),
         (201, 8192), (600, 4096)]


def _ops(dtype):
    from cpmcu_b200.ops.ops import Ops
    return Ops(DT[dtype], "cuda:0")


def _layer_norm(x, w, b):
    m = x.mean(-1, keepdim=True)
    return (x - m) / ((x - m).pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w + b


def _rms_norm(x, w):
    return x / (x.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w


def _near(got, want, dtype):
    assert float((got.double() - want).abs().max()) < TOL[dtype]


def _operands(rows, hidden, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows * 10000 + hidden)
    x = torch.randn(rows, hidden, generator=g, device="cuda") * 2 + 0.5
    a, a2 = ((torch.randn(rows, hidden, generator=g, device="cuda")).to(DT[dtype]) for _ in range(2))
    vectors = [torch.rand(hidden, generator=g, device="cuda") * 0.8 + 0.2 for _ in range(2)] + \
              [torch.rand(hidden, generator=g, device="cuda") * 0.4 - 0.2 for _ in range(2)]
    return x, a, a2, *vectors


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,hidden", SIZES)
def test_norms_behind_sums(dtype, rows, hidden):
    ops = _ops(dtype)
    x, a, a2, w, w2, b, b2 = _operands(rows, hidden, dtype)
    X, A, A2, W, W2, B, B2 = (t.double() for t in (x, a, a2, w, w2, b, b2))
    s = x.clone()
    y = ops.add_rmsnorm(s, a, 0.4, w, 1e-5)
    _near(s, X + 0.4 * A, "float32")
    _near(y, _rms_norm(X + 0.4 * A, W), dtype)
    s = x.clone()
    y, y2 = ops.layernorm(s, w, b, 1e-5, None, a, 0.4, a2, (w2, b2))
    _near(s, X + 0.4 * (A + A2), "float32")
    _near(y, _layer_norm(X + 0.4 * (A + A2), W, B), dtype)
    _near(y2, _layer_norm(X + 0.4 * (A + A2), W2, B2), dtype)
    _near(ops.layernorm(x.clone(), w, None, 1e-5, torch.tensor([rows - 1, 0], dtype=torch.int32, device="cuda")), _layer_norm(X, W, 0.0)[[rows - 1, 0]], dtype)
    s = x.clone()
    y = ops.post_norm(s, a, 1.5, w2, w, 1e-5)
    want = _rms_norm(1.5 * X + W2 * A, W)
    _near(s, want, "float32")
    _near(y, want, dtype)
    s = x.clone()
    y = ops.post_norm_add(s, a, w, b, 1e-5, (w2, b2))
    want = X + _layer_norm(A, W, B)
    _near(s, want, "float32")
    _near(y, _layer_norm(want, W2, B2), dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,hidden", [s for s in SIZES if s[0] > 2])
def test_layer_norm_with_token_shift(dtype, rows, hidden):
    """Three sequences: one goes on from a carried row, one begins in a slot that holds rubbish, one brings a single token."""
    from types import SimpleNamespace

    ops = _ops(dtype)
    x, _, _, w, mix, b, _ = _operands(rows, hidden, dtype)
    X, W, M, B = (t.double() for t in (x, w, mix, b))
    cut = (rows - 1) // 2 or 1
    cu = [0, cut, rows - 1, rows]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts, slots = [4, 0, 9], [3, 1, 0]
    ctx = SimpleNamespace(positions=i32([s + i for s, lo, hi in zip(starts, cu, cu[1:]) for i in range(hi - lo)]), cu_q=i32(cu), slot_dev=i32(slots),
                          token_seq=i32([j for j, (lo, hi) in enumerate(zip(cu, cu[1:])) for _ in range(hi - lo)]))
    state = torch.randn(5, hidden, device="cuda")
    before = state.clone()
    y = ops.layernorm_shift(ctx, x, w, b, 1e-5, mix, state)
    h = _layer_norm(X, W, B)
    prev = torch.cat([h[:1], h[:-1]])
    for s, slot, lo in zip(starts, slots, cu):
        prev[lo] = before[slot].double() if s else 0.0
    _near(y, h + (prev - h) * M, dtype)
    for slot, hi in zip(slots, cu[1:]):
        _near(state[slot], h[hi - 1], "float32")
    assert torch.equal(state[[2, 4]], before[[2, 4]])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("S,W", [(1, 132), (2, 1024), (2, 2048), (3, 2044), (4, 1024), (4, 2048), (4, 2052), (5, 1024)])
@pytest.mark.parametrize("rows", [3, 513])
def test_streams_blended_and_normed(dtype, S, W, rows):
    ops = _ops(dtype)
    g = torch.Generator(device="cuda").manual_seed(S * W)
    X = torch.randn(rows, S, W, generator=g, device="cuda")
    y = torch.randn(rows, W, generator=g, device="cuda").to(DT[dtype])
    mix, out, read, gain = (torch.randn(*n, generator=g, device="cuda") * 0.4 for n in ((S, S), (S,), (S,), (1,)))
    now, total = X.clone(), torch.empty(rows, W, device="cuda")
    h = ops.hyper_step(now, write=(y, mix, out), read=(read, gain), eps=1e-5, total=total)
    want = torch.einsum("sr,tsw->trw", mix.double(), X.double()) + out.double()[None, :, None] * y.double()[:, None]
    _near(now, want, "float32")
    _near(total, want.sum(1), "float32")
    _near(h, _rms_norm(torch.einsum("s,tsw->tw", read.double(), want), gain.double()), dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tokens,heads,dv,group", [(3, 3, 44, 3), (3, 2, 64, 1), (2, 4, 128, 1), (2, 16, 128, 16), (2, 33, 64, 33), (2, 32, 256, 32), (300, 2, 1024, 1), (200, 3, 1024, 1)])
@pytest.mark.parametrize("act", ["sigmoid", "silu"])
def test_norm_over_heads_with_a_gate_on_whole_loads(dtype, tokens, heads, dv, group, act):
    """The gate is a slice of a wider row that begins on a 16-byte boundary, and (the same numbers) one that does not."""
    ops = _ops(dtype)
    g = torch.Generator(device="cuda").manual_seed(heads * dv)
    o = torch.randn(tokens, heads, dv, generator=g, device="cuda") * 3
    wide = torch.randn(tokens, heads * dv + 8, generator=g, device="cuda")
    weight = torch.rand(group * dv, generator=g, device="cuda") * 0.5
    gate = wide[:, 4:4 + heads * dv].double()
    want = _rms_norm(o.double().view(tokens, heads // group, group * dv), weight.double()).reshape(tokens, -1)
    want = want * (torch.sigmoid(gate) if act == "sigmoid" else gate * torch.sigmoid(gate))
    _near(ops.gated_group_norm(o, wide[:, 4:4 + heads * dv], weight, 1e-5, group, act), want, dtype)
    shifted = torch.randn(tokens, heads * dv + 9, device="cuda")
    shifted[:, 5:5 + heads * dv] = wide[:, 4:4 + heads * dv]
    _near(ops.gated_group_norm(o, shifted[:, 5:5 + heads * dv], weight, 1e-5, group, act), want, dtype)


@pytest.mark.parametrize("hidden", [1024, 2048, 4096, 8192])
def test_a_row_of_the_32_bit_path_does_not_depend_on_the_step(hidden):
    """The same bits alone and among 700 rows, in every norm of a row."""
    ops = _ops("float32")
    x, a, a2, w, w2, b, b2 = _operands(700, hidden, "float32")
    some = [0, 13, 699]
    for f in (lambda x, a, a2: (ops.add_rmsnorm(x, a, 0.4, w, 1e-5),), lambda x, a, a2: ops.layernorm(x, w, b, 1e-5, None, a, 0.4, a2, (w2, b2)),
              lambda x, a, a2: (ops.post_norm(x, a, 1.5, w2, w, 1e-5),), lambda x, a, a2: (ops.post_norm_add(x, a, w, b, 1e-5, (w2, b2)),),
              lambda x, a, a2: (ops.gated_group_norm(x.view(-1, 1, hidden), a, w, 1e-5, 1, "silu"),),
              lambda x, a, a2: (ops.hyper_step(torch.stack([x, a], 1), read=(w[:2].contiguous(), w[:1].contiguous()), eps=1e-5),)):
        whole = f(x.clone(), a, a2)
        for i in some:
            alone = f(x[i:i + 1].clone(), a[i:i + 1].contiguous(), a2[i:i + 1].contiguous())
            assert all(torch.equal(one[0], many[i]) for one, many in zip(alone, whole))
