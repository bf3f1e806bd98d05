"""The recurrences of prompts in chunks of tokens against the same recurrences token by token."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def ops():
    from fieldrun_b200.csrc import ops as o
    return o


def i32(values):
    return torch.tensor(np.asarray(values), dtype=torch.int32, device=DEV)


def tables(lengths, size):
    seqs, lo, hi, first = [], [], [], [0]
    for b, n in enumerate(lengths):
        for t in range(0, n, size):
            seqs.append(b), lo.append(t), hi.append(min(t + size, n))
        first.append(len(seqs))
    return tuple(i32(x) for x in (seqs, lo, hi, first))


def norm_error(got, want):
    assert torch.isfinite(got).all()
    return ((got.double() - want.double()).norm() / want.double().norm().clamp_min(1e-30)).item()


# Both ways are float32 sums of the same terms; a state's decays are multiplied one after the other over the whole prompt
# (about a rounding each: some hundred times 2^-24 for 300 tokens), or 16 and 64 at a time.
LIMIT = 300 * 2.0 ** -24


@pytest.mark.parametrize("decay", ["mild", "strong", "extreme", "mixed"])
@pytest.mark.parametrize("heads,dim,vdim,rank,dtype", [(3, 128, 128, 32, "float32"), (2, 64, 64, 16, "float32"), (2, 128, 64, 4, "float32"),
                                                       (1, 64, 128, 64, "float32"), (3, 128, 128, 32, "bfloat16")])
def test_gated_linear_attention_in_chunks(heads, dim, vdim, rank, dtype, decay):
    """Chunks of 64, 16 k + r and one token, sequences that go on from a state at odd and even positions, decays of a chunk from
    nearly one to exp(-10000)."""
    gen = torch.Generator(device=DEV).manual_seed(dim + vdim)
    lengths, starts, slots = [300, 64, 17, 1, 129], [0, 3, 10, 7, 64], [4, 0, 2, 1, 3]
    tokens, width = sum(lengths), 2 * heads * (dim + vdim) + rank
    offsets = (0, heads * dim, 2 * heads * dim, 2 * heads * dim + heads * vdim, 2 * heads * (dim + vdim))
    kind = getattr(torch, dtype)
    proj = torch.randn(tokens, width, device=DEV, generator=gen)
    a2 = (torch.randn(heads * dim, rank, device=DEV, generator=gen) * 0.3).to(kind)
    bias = torch.randn(heads * dim, device=DEV, generator=gen) + {"mild": 3.0, "strong": -20.0, "extreme": -150.0, "mixed": 0.0}[decay]
    if decay == "mixed":
        bias *= 20.0
    norm = torch.randn(vdim, device=DEV, generator=gen)
    state = torch.randn(5, 2, heads, dim, vdim, device=DEV, generator=gen)
    sizes = dict(heads=heads, dim=dim, vdim=vdim, tau=1.0 if decay == "extreme" else 16.0, q_scale=dim ** -0.5, eps=1e-6)
    cu = i32(np.concatenate([[0], np.cumsum(lengths)]))
    results = []
    for chunked in (False, True):
        kept, out = state.clone(), torch.full((tokens, heads * vdim), float("nan"), device=DEV, dtype=kind)
        args = (proj, offsets, a2, bias, norm, kept, i32(slots), i32(starts), cu, out)
        if chunked:
            assert ops().gla_chunks_take(dim, vdim, rank, width, offsets)
            chunks = tables(lengths, 64)
            scratch = torch.full((ops().gla_chunks_scratch_floats(chunks[0].numel(), tokens, heads, dim, vdim),), float("nan"), device=DEV)
            ops().gla_chunks(*args, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().gla_scan(*args, **sizes)
        results.append((out, kept))
    assert norm_error(results[1][0].float(), results[0][0].float()) < (LIMIT if dtype == "float32" else 2.0 ** -9)
    for n, start, slot in zip(lengths, starts, slots):
        assert norm_error(results[1][1][slot, (start + n) & 1], results[0][1][slot, (start + n) & 1]) < LIMIT
        if n % 2:
            assert torch.equal(results[1][1][slot, start & 1], state[slot, start & 1])       # the copy it began from is left alone


class Tables:
    def __init__(self, lengths, starts, slots):
        self.num_seqs, self.max_q_len = len(lengths), max(lengths)
        self.seq_slot, self.seq_start = i32(slots), i32(starts)
        self.cu_q_len = i32(np.concatenate([[0], np.cumsum(lengths)]))
        self.tok_seq = i32(np.repeat(np.arange(len(lengths)), lengths))


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("channels,typed,biased", [(4, True, True), (520, False, True), (1028, True, False)])
def test_convolution_of_four_channels_a_thread_equals_one_channel_a_thread(taps, channels, typed, biased):
    """Sequences that end inside a run of eight rows, and shorter ones than the window; the same sums in the same order."""
    gen = torch.Generator(device=DEV).manual_seed(channels)
    lengths, starts, slots = [77, 1, 2, 3, 60, 8], [0, 5, 4, 7, 2, 0], [5, 3, 1, 0, 2, 4]
    tokens = sum(lengths)
    rows = torch.randn(tokens, channels, device=DEV, generator=gen)
    weights, bias, in_bias = (torch.randn(*shape, device=DEV, generator=gen) for shape in ((channels, taps), (channels,), (channels,)))
    results = []
    for offset in (4, 3):                                        # 3: the rows do not begin on 16 bytes
        shifted = torch.zeros(tokens, channels + 8, device=DEV)
        shifted[:, offset:offset + channels] = rows
        state = torch.ones(6, 2, (taps - 1) * channels, device=DEV)
        out32 = torch.full((tokens, channels), float("nan"), device=DEV)
        out = torch.zeros(tokens, channels, device=DEV, dtype=torch.bfloat16) if typed else None
        ops().causal_conv(shifted, offset, channels, weights, bias if biased else None, Tables(lengths, starts, slots), state, 0, out32, out,
                          in_bias=in_bias if biased else None, activation="silu")
        results.append((out32, state, out))
    assert torch.isfinite(results[0][0]).all()
    for a, b in zip(*results):
        assert a is None or torch.equal(a, b)


@pytest.mark.parametrize("lengths", [[2900, 1, 33, 3, 300], [1000, 2, 900, 31]])
def test_convolution_of_long_runs_of_rows(lengths):
    """Runs of 32 rows a thread and of 16, sequences that begin and end inside them, sums beyond 80 in size (another form of silu), a state
    at any offset: the same bits as one channel a thread."""
    channels, taps, starts, slots = 6144, 4, [3, 0, 6, 1, 8][:len(lengths)], [4, 0, 2, 1, 3][:len(lengths)]
    gen = torch.Generator(device=DEV).manual_seed(len(lengths))
    tokens = sum(lengths)
    rows = torch.randn(tokens, channels, device=DEV, generator=gen)
    rows[::50] *= 100.0
    weights, bias = torch.randn(channels, taps, device=DEV, generator=gen), torch.randn(channels, device=DEV, generator=gen)
    before = torch.randn(5, 2, 3 + (taps - 1) * channels, device=DEV, generator=gen)
    results = []
    for offset in (4, 3):
        shifted = torch.zeros(tokens, channels + 8, device=DEV)
        shifted[:, offset:offset + channels] = rows
        state, out32 = before.clone(), torch.full((tokens, channels), float("nan"), device=DEV)
        ops().causal_conv(shifted, offset, channels, weights, bias, Tables(lengths, starts, slots), state, 3, out32, activation="silu")
        results.append((out32, state))
    assert torch.isfinite(results[0][0]).all() and torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("decay", ["mild", "strong", "extreme", "mixed"])
@pytest.mark.parametrize("heads,groups,n,vdim", [(4, 2, 128, 64), (2, 1, 64, 64), (2, 2, 128, 128), (3, 1, 64, 128)])
def test_state_space_in_chunks(heads, groups, n, vdim, decay):
    """Chunks of 128, 16 k + r and one token, sequences that go on from a state at odd and even positions, decays of a token from
    nearly one to exp(-50)."""
    gen = torch.Generator(device=DEV).manual_seed(n + vdim + heads)
    lengths, starts, slots = [300, 128, 17, 1, 257], [0, 3, 10, 7, 64], [4, 0, 2, 1, 3]
    tokens, inner = sum(lengths), heads * vdim
    proj = torch.randn(tokens, inner + heads + heads % 2, device=DEV, generator=gen)
    proj[:, inner:] += {"mild": -4.0, "strong": 2.0, "extreme": 8.0, "mixed": 0.0}[decay]
    if decay == "mixed":
        proj[:, inner:] *= 5.0
    xbc = torch.randn(tokens, inner + 2 * groups * n, device=DEV, generator=gen) * 0.3
    dt_bias, a_log, d = torch.randn(heads, device=DEV, generator=gen) * 0.2, torch.randn(heads, device=DEV, generator=gen) * 0.5, torch.ones(heads, device=DEV)
    state = torch.randn(5, 2, 4 + heads * n * vdim + 8, device=DEV, generator=gen)
    sizes = dict(heads=heads, vdim=vdim, n=n, groups=groups)
    tabs = Tables(lengths, starts, slots)
    results = []
    for chunked in (False, True):
        kept, out = state.clone(), torch.full((tokens, inner), float("nan"), device=DEV)
        args = (proj, 0, inner, xbc, inner, inner + groups * n, dt_bias, a_log, d, tabs, kept, 4, out)
        if chunked:
            assert ops().state_space_chunks_take(z_offset=0, row=proj.shape[1], xbc_offsets=(xbc.shape[1], inner), state=kept, state_offset=4, **sizes)
            chunks = tables(lengths, 128)
            scratch = torch.full((ops().state_space_chunks_scratch_floats(chunks[0].numel(), **sizes),), float("nan"), device=DEV)
            ops().state_space_chunks(*args, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().state_space_scan(*args, **sizes)
        results.append((out, kept))
    assert norm_error(results[1][0], results[0][0]) < LIMIT
    for length, start, slot in zip(lengths, starts, slots):
        copy = (start + length) & 1
        assert norm_error(results[1][1][slot, copy, 4:-8], results[0][1][slot, copy, 4:-8]) < LIMIT
        results[1][1][slot, copy, 4:-8] = state[slot, copy, 4:-8]
    assert torch.equal(results[1][1], state)                     # nothing else was written


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(2, 1, 128, 128), (2, 1, 64, 64), (2, 2, 128, 64), (1, 1, 64, 128)])
def test_values_of_the_delta_rule_at_any_offset(heads, kv_heads, dim, vdim):
    """Values that begin on 16 bytes, on 8, and on 4 alone (read two columns at a time or one): the same bits."""
    gen = torch.Generator(device=DEV).manual_seed(dim + vdim)
    lengths, starts, slots = [130, 1, 63, 64], [0, 3, 10, 6], [3, 0, 2, 1]
    tokens, qk, inner = sum(lengths), kv_heads * dim, heads * vdim
    rows, proj = torch.randn(tokens, 2 * qk + inner, device=DEV, generator=gen), torch.randn(tokens, 2 * heads + inner, device=DEV, generator=gen)
    a_log, dt_bias, norm = (torch.randn(n, device=DEV, generator=gen) * 0.2 + 1.0 for n in (heads, heads, vdim))
    state = torch.randn(4, 2, heads * dim * vdim, device=DEV, generator=gen)
    chunks = tables(lengths, 64)
    results = []
    for shift in (0, 2, 1):
        conv = torch.full((tokens, 2 * qk + inner + 4), float("nan"), device=DEV)
        conv[:, :2 * qk], conv[:, 2 * qk + shift:2 * qk + shift + inner] = rows[:, :2 * qk], rows[:, 2 * qk:]
        kept, out, raw = state.clone(), torch.full((tokens, inner), float("nan"), device=DEV), torch.full((tokens, inner), float("nan"), device=DEV)
        scratch = torch.full((ops().delta_chunks_scratch_floats(chunks[0].numel(), heads, dim, vdim),), float("nan"), device=DEV)
        ops().delta_chunks(conv, 0, qk, 2 * qk + shift, proj, 0, heads, 2 * heads, a_log, dt_bias, norm, Tables(lengths, starts, slots), kept, 0, out,
                           raw=raw, chunks=chunks, scratch=scratch, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, eps=1e-6)
        results.append((out, kept))
    assert torch.isfinite(results[0][0]).all()
    for out, kept in results[1:]:
        assert torch.equal(out, results[0][0]) and torch.equal(kept, results[0][1])


@pytest.mark.parametrize("decay", ["mild", "strong", "extreme", "mixed"])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,dtype", [(4, 2, 128, 128, "float32"), (2, 1, 64, 64, "float32"), (2, 2, 128, 64, "float32"),
                                                           (1, 1, 64, 128, "float32"), (4, 1, 128, 128, "bfloat16")])
def test_gated_delta_rule_in_chunks(heads, kv_heads, dim, vdim, dtype, decay):
    """Chunks of 64, 16 k + r and one token, sequences that go on from a state at odd and even positions, decays of a token from
    nearly one to exp(-50), keys that repeat one another (the substitution's hardest case) and a key of zeros."""
    gen = torch.Generator(device=DEV).manual_seed(dim + vdim + heads)
    lengths, starts, slots = [300, 64, 17, 1, 129], [0, 3, 10, 7, 64], [4, 0, 2, 1, 3]
    tokens, qk, inner = sum(lengths), kv_heads * dim, heads * vdim
    conv = torch.randn(tokens, 2 * qk + inner, device=DEV, generator=gen)
    conv[70:100, qk:2 * qk] = conv[70, qk:2 * qk] * torch.where(torch.arange(30, device=DEV) % 3 == 1, -1.0, 2.0)[:, None]
    conv[110, qk:2 * qk] = 0.0
    proj = torch.randn(tokens, 2 * heads + inner, device=DEV, generator=gen)
    proj[:, :heads] += 2.0                                       # beta close to one
    proj[:, heads:2 * heads] += {"mild": -4.0, "strong": 2.0, "extreme": 8.0, "mixed": 0.0}[decay]
    if decay == "mixed":
        proj[:, heads:2 * heads] *= 5.0
    a_log, dt_bias = torch.randn(heads, device=DEV, generator=gen) * 0.5, torch.randn(heads, device=DEV, generator=gen) * 0.2
    norm = torch.randn(vdim, device=DEV, generator=gen)
    state = torch.randn(5, 2, 2 + heads * dim * vdim + 6, device=DEV, generator=gen)
    sizes = dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, eps=1e-6)
    tabs = Tables(lengths, starts, slots)
    results = []
    for chunked in (False, True):
        kept, out = state.clone(), torch.full((tokens, inner), float("nan"), device=DEV, dtype=getattr(torch, dtype))
        raw = torch.full((tokens, inner), float("nan"), device=DEV)
        args = (conv, 0, qk, 2 * qk, proj, 0, heads, 2 * heads, a_log, dt_bias, norm, tabs, kept, 2, out)
        if chunked:
            assert ops().delta_chunks_take(dim, vdim, (conv.shape[1], qk), kept, 2)
            chunks = tables(lengths, 64)
            scratch = torch.full((ops().delta_chunks_scratch_floats(chunks[0].numel(), heads, dim, vdim),), float("nan"), device=DEV)
            ops().delta_chunks(*args, raw=raw, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().gated_delta_rule(*args, raw=raw, **sizes)
        results.append((out, kept, raw))
    assert norm_error(results[1][0].float(), results[0][0].float()) < (LIMIT if dtype == "float32" else 2.0 ** -9)
    for n, start, slot in zip(lengths, starts, slots):
        copy = (start + n) & 1
        assert norm_error(results[1][1][slot, copy, 2:-6], results[0][1][slot, copy, 2:-6]) < LIMIT
        results[1][1][slot, copy, 2:-6] = state[slot, copy, 2:-6]
    assert torch.equal(results[1][1], state)                     # nothing else was written


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,width,groups", [(3, 4, 1), (2, 4096, 1), (5, 4100, 1), (2, 9000, 2), (5, 2304, 9), (3, 1024, 1), (1, 1028, 1),
                                               (7, 780, 3)])
def test_group_norm_of_four_columns_a_thread(rows, width, groups, dtype):
    """Parts inside, at and beyond what a block keeps in registers, against 64 bits and against one column a thread."""
    gen = torch.Generator(device=DEV).manual_seed(width)
    store = torch.randn(rows * width + 1, device=DEV, generator=gen)
    weight = torch.randn(width, device=DEV, generator=gen)
    results = []
    for place in (0, 1):                                         # 1: the rows do not begin on 16 bytes
        x = store[place:place + rows * width].copy_(store[:rows * width].clone()).view(rows, width)
        out = torch.full((rows, width), float("nan"), device=DEV, dtype=getattr(torch, dtype))
        ops().group_rms_norm(x, weight, out, groups, 1e-6)
        parts = x.double().view(rows, groups, -1)
        want = (parts / (parts.square().mean(-1, keepdim=True) + 1e-6).sqrt()).view(rows, width) * weight.double()
        # a rounding each of the root, the quotient and two products, and the sum's (a few: 128 threads each add up to 72 squares)
        bound = want.abs() * (2.0 ** -20 if dtype == "float32" else 2.0 ** -8)
        assert ((out.double() - want).abs() <= bound).all()
        results.append(out)
    assert norm_error(results[0].float(), results[1].float()) < (2.0 ** -20 if dtype == "float32" else 2.0 ** -8)


# ------------------------------------------------------------------------------- numbers that are not finite, one strong decay

INF, NAN = float("inf"), float("nan")
LENGTHS, STARTS, SLOTS = [300, 64, 17, 1, 129], [0, 3, 10, 7, 64], [4, 0, 2, 1, 3]
AT = [int(c) for c in np.concatenate([[0], np.cumsum(LENGTHS)])]


def gla_case():
    """heads x dim x vdim 2 x 64 x 64, decay rank 8: the inputs by name (views of the projection's rows), and run(chunked)."""
    heads, dim, vdim, rank = 2, 64, 64, 8
    gen = torch.Generator(device=DEV).manual_seed(1)
    tokens, width = AT[-1], 2 * heads * (dim + vdim) + rank
    offsets = (0, heads * dim, 2 * heads * dim, 2 * heads * dim + heads * vdim, 2 * heads * (dim + vdim))
    proj = torch.randn(tokens, width, device=DEV, generator=gen)
    a2, bias = torch.randn(heads * dim, rank, device=DEV, generator=gen) * 0.3, torch.randn(heads * dim, device=DEV, generator=gen) + 2.0
    norm, state = torch.randn(vdim, device=DEV, generator=gen), torch.randn(5, 2, heads, dim, vdim, device=DEV, generator=gen)
    views = {n: proj[:, a:b] for n, a, b in zip(("q", "k", "v", "gate", "decay"), offsets, (*offsets[1:], width))}
    sizes = dict(heads=heads, dim=dim, vdim=vdim, tau=16.0, q_scale=dim ** -0.5, eps=1e-6)

    def run(chunked):
        kept, out = state.clone(), torch.full((tokens, heads * vdim), NAN, device=DEV)
        args = (proj, offsets, a2, bias, norm, kept, i32(SLOTS), i32(STARTS), i32(AT), out)
        if chunked:
            chunks = tables(LENGTHS, 64)
            scratch = torch.full((ops().gla_chunks_scratch_floats(chunks[0].numel(), tokens, heads, dim, vdim),), NAN, device=DEV)
            ops().gla_chunks(*args, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().gla_scan(*args, **sizes)
        return out, kept.view(5, 2, -1)

    def exact():
        q, k, v, gate, inside = (views[m].double() for m in ("q", "k", "v", "gate", "decay"))
        alpha = torch.exp(torch.nn.functional.logsigmoid(inside @ a2.double().T + bias.double()) / 16.0).view(tokens, heads, dim, 1)
        q, k, v = (z.view(tokens, heads, *shape) for z, shape in ((q, (dim, 1)), (k, (dim, 1)), (v, (1, vdim))))
        outs, states = [], []
        for row, length in enumerate(LENGTHS):
            kept = state[SLOTS[row], STARTS[row] & 1].double()
            for t in range(AT[row], AT[row] + length):
                kept = kept * alpha[t] + k[t] * v[t]
                outs.append((kept * q[t]).sum(1) * dim ** -0.5)
            states.append(kept)
        o = torch.stack(outs)
        o = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-6) * norm.double()
        return o * torch.nn.functional.silu(gate).view(tokens, heads, vdim), states
    return views, run, exact


def state_space_case(n=64, vdim=64):
    heads, groups = 4, 2
    gen = torch.Generator(device=DEV).manual_seed(2)
    tokens, inner = AT[-1], heads * vdim
    proj, xbc = torch.randn(tokens, inner + heads, device=DEV, generator=gen), torch.randn(tokens, inner + 2 * groups * n, device=DEV, generator=gen) * 0.3
    proj[:, inner:] -= 3.0
    dt_bias, a_log, d = (torch.randn(heads, device=DEV, generator=gen) * 0.2 + c for c in (0.0, 0.0, 1.0))
    state = torch.randn(5, 2, heads * n * vdim, device=DEV, generator=gen)
    views = {"x": xbc[:, :inner], "b": xbc[:, inner:inner + groups * n], "c": xbc[:, inner + groups * n:], "gate": proj[:, :inner], "decay": proj[:, inner:]}
    sizes, tabs = dict(heads=heads, vdim=vdim, n=n, groups=groups), Tables(LENGTHS, STARTS, SLOTS)

    def run(chunked):
        kept, out = state.clone(), torch.full((tokens, inner), NAN, device=DEV)
        args = (proj, 0, inner, xbc, inner, inner + groups * n, dt_bias, a_log, d, tabs, kept, 0, out)
        if chunked:
            chunks = tables(LENGTHS, 128)
            scratch = torch.full((ops().state_space_chunks_scratch_floats(chunks[0].numel(), **sizes),), NAN, device=DEV)
            ops().state_space_chunks(*args, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().state_space_scan(*args, **sizes)
        return out, kept

    def exact():
        step = torch.nn.functional.softplus(views["decay"].double() + dt_bias.double())
        decay, x = torch.exp(-a_log.double().exp() * step), views["x"].double().view(tokens, heads, vdim)
        b, c = (views[m].double().view(tokens, groups, n).repeat_interleave(heads // groups, 1) for m in "bc")
        outs, states = [], []
        for row, length in enumerate(LENGTHS):
            kept = state[SLOTS[row], STARTS[row] & 1].double().view(heads, n, vdim)
            for t in range(AT[row], AT[row] + length):
                kept = kept * decay[t][:, None, None] + b[t][:, :, None] * (step[t][:, None] * x[t])[:, None]
                outs.append((kept * c[t][:, :, None]).sum(1) + d.double()[:, None] * x[t])
            states.append(kept)
        return (torch.stack(outs).view(tokens, inner) * torch.nn.functional.silu(views["gate"].double())).view(tokens, heads, vdim), states
    return views, run, exact


def delta_case(vdim=64):
    heads, kv_heads, dim = 4, 2, 64
    gen = torch.Generator(device=DEV).manual_seed(3)
    tokens, qk, inner = AT[-1], kv_heads * dim, heads * vdim
    conv, proj = torch.randn(tokens, 2 * qk + inner, device=DEV, generator=gen), torch.randn(tokens, 2 * heads + inner, device=DEV, generator=gen)
    proj[:, heads:2 * heads] -= 3.0
    a_log, dt_bias, norm = (torch.randn(*shape, device=DEV, generator=gen) * 0.2 + c for shape, c in (((heads,), 0.0), ((heads,), 0.0), ((vdim,), 1.0)))
    state = torch.randn(5, 2, heads * dim * vdim, device=DEV, generator=gen)
    views = {"q": conv[:, :qk], "k": conv[:, qk:2 * qk], "v": conv[:, 2 * qk:], "beta": proj[:, :heads], "decay": proj[:, heads:2 * heads],
             "gate": proj[:, 2 * heads:]}
    sizes, tabs = dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, eps=1e-6), Tables(LENGTHS, STARTS, SLOTS)

    def run(chunked):
        kept, out = state.clone(), torch.full((tokens, inner), NAN, device=DEV)
        raw = torch.full((tokens, inner), NAN, device=DEV)
        args = (conv, 0, qk, 2 * qk, proj, 0, heads, 2 * heads, a_log, dt_bias, norm, tabs, kept, 0, out)
        if chunked:
            chunks = tables(LENGTHS, 64)
            scratch = torch.full((ops().delta_chunks_scratch_floats(chunks[0].numel(), heads, dim, vdim),), NAN, device=DEV)
            ops().delta_chunks(*args, raw=raw, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().gated_delta_rule(*args, raw=raw, **sizes)
        return out, kept

    def exact():
        q, k = (views[m].double().view(tokens, kv_heads, dim) for m in "qk")
        q, k = ((z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(heads // kv_heads, 1) for z in (q, k))
        v, beta = views["v"].double().view(tokens, heads, vdim), torch.sigmoid(views["beta"].double())
        decay = torch.exp(-a_log.double().exp() * torch.nn.functional.softplus(views["decay"].double() + dt_bias.double()))
        outs, states = [], []
        for row, length in enumerate(LENGTHS):
            kept = state[SLOTS[row], STARTS[row] & 1].double().view(heads, dim, vdim)
            for t in range(AT[row], AT[row] + length):
                kept = kept * decay[t][:, None, None]
                u = beta[t][:, None] * (v[t] - (kept * k[t][:, :, None]).sum(1))
                kept = kept + k[t][:, :, None] * u[:, None]
                outs.append((kept * q[t][:, :, None]).sum(1) * dim ** -0.5)
            states.append(kept)
        o = torch.stack(outs)
        o = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-6) * norm.double()
        return o * torch.nn.functional.silu(views["gate"].double()).view(tokens, heads, vdim), states
    return views, run, exact


# with 128 value columns the chain along the chunks runs on tcgen05
CASES = {"gla": gla_case, "state space": state_space_case, "state space 128": lambda: state_space_case(128, 128), "delta": delta_case, "delta 128": lambda: delta_case(128)}


NAMES = [("gla", n) for n in ("q", "k", "v", "decay")] + [(c, n) for c in ("state space", "state space 128") for n in ("x", "b", "c", "decay")] + [
    (c, n) for c in ("delta", "delta 128") for n in ("q", "k", "v", "beta", "decay")]


@pytest.mark.parametrize("case,name,number", [(*c, n) for c in NAMES for n in (INF, NAN)] + [("state space", "x", 3.4028234e38),
                                                                                             ("state space 128", "x", 3.4028234e38),
                                                                                             ("delta", "v", 3.4028234e38),
                                                                                             ("delta 128", "v", 3.4028234e38)])
def test_a_token_that_is_not_finite_reaches_no_token_before_it(case, name, number):
    """One entry of a token in the middle of a chunk, of a chunk's last block and of a short sequence: the heads of the outputs and the
    entries of the states that it makes infinities or NaNs of are those that it does token by token, and the tokens before it keep
    theirs.  (The largest float32 rounds to an infinity when it is cut in parts; here no product with it is one.)"""
    views, run = CASES[case]()[:2]
    hit = [AT[0] + 70, AT[0] + 170, AT[1] + 5, AT[2] + 15]
    for t in hit:
        views[name][t, 1] = number
    want, got = run(False), run(True)
    clean = torch.ones(AT[-1], dtype=torch.bool, device=DEV)                 # rows that no such number has come into
    for row, begin in enumerate(AT[:-1]):
        first = min((t for t in hit if begin <= t < AT[row + 1]), default=AT[row + 1])
        clean[first:AT[row + 1]] = False
    assert want[0][clean].isfinite().all() and norm_error(got[0][clean], want[0][clean]) < LIMIT
    heads = [out.view(AT[-1], -1, 64).isfinite().all(2) for out in (want[0], got[0])]
    assert torch.equal(*heads)
    pairs = [(got[0].view(AT[-1], -1, 64)[heads[0]], want[0].view(AT[-1], -1, 64)[heads[0]])]
    for row, slot in enumerate(SLOTS):
        copy = (STARTS[row] + LENGTHS[row]) & 1
        a, b = got[1][slot, copy], want[1][slot, copy]
        assert torch.equal(a.isfinite(), b.isfinite())
        pairs.append((a[b.isfinite()], b[b.isfinite()]))
    for a, b in pairs:
        if b.numel():
            assert norm_error(a, b) < LIMIT


@pytest.mark.parametrize("case,strong", [(c, s) for c in ("state space", "state space 128", "delta", "delta 128") for s in (-20.0, -200.0, -2000.0)] +
                         [("delta", -INF), ("delta 128", -INF)])
def test_one_strong_decay_among_mild_ones(case, strong):
    """Tokens that all but clear the state (logarithm of the decay down to about -2,000, and a decay of zero), one in each of some blocks,
    at the starts of chunks and blocks among them, the others mild: against 64 bits, every token's head by itself.  A weight between
    tokens behind such a one that is made from sums reaching across it has lost 2,000 2^-24 of its size.  The limit: 128 entries of
    a sum over the states and 64 of a sum over tokens, a rounding each, on results that are at least an eighth of what they are sums of."""
    views, run, exact = CASES[case]()
    for t in (3, 64, 80, 127, 128, 145, 200, 299):
        views["decay"][t] = -strong
    want, states = exact()
    got, kept = run(True)
    error = (got.double().view_as(want) - want).norm(dim=-1) / want.norm(dim=-1)
    print(case, strong, "outputs", error.max().item(), "token by token", ((run(False)[0].double().view_as(want) - want).norm(dim=-1) / want.norm(dim=-1)).max().item())
    assert error.max() < 8 * 192 * 2.0 ** -24
    for row, slot in enumerate(SLOTS):
        state = kept[slot, (STARTS[row] + LENGTHS[row]) & 1].double().view_as(states[row])
        assert ((state - states[row]).norm(dim=(1, 2)) / states[row].norm(dim=(1, 2))).max() < 300 * 2.0 ** -24


# by name: the tokens made large, those whose decay clears the state, and the rows of zeros in front
SETTINGS = {
    "a large token, cleared by a decay": ({20: 1.0}, (30, 80), 0),
    "a large first token, cleared by a decay": ({0: 1.0, 64: 1.0}, (8, 70), 0),
    "a large token behind zeros": ({20: 1.0}, (), 9),
    "a large token behind small ones": ({50: 1.0, 140: 1.0}, (), 0),
    "a large last token": ({63: 1.0, 127: 1.0}, (64, 128), 0),
}


@pytest.mark.parametrize("setting", SETTINGS)
@pytest.mark.parametrize("case,name", [(c, n) for c in ("state space", "state space 128") for n in "xb"] + [("delta", "v"), ("delta 128", "v")])
@pytest.mark.parametrize("power", [8, 16, 19, 22, 26, 30, 36, 50, 66])
def test_a_large_token_costs_no_other_token_its_digits(case, name, setting, power):
    """Tokens 2^power larger than the others, with a decay of e^-200 behind them, or behind eight rows of zeros and none, or behind small ones:
    against 64 bits, every token's head by itself, as in the test before; the states' columns too, behind the last token."""
    views, run, exact = CASES[case]()
    large, cleared, zeros = SETTINGS[setting]
    for begin in AT[:-1]:
        end = AT[AT.index(begin) + 1]
        for t in large:
            if begin + t < end:
                views[name][begin + t] *= 2.0 ** power
        for t in cleared:
            if begin + t < end:
                views["decay"][begin + t] = 200.0
        views[name][begin:min(begin + zeros, end)] = 0.0
    want, states = exact()
    plain, kept_plain = run(False)
    got, kept = run(True)
    size = want.norm(dim=-1)
    error, least = (((t.double().view_as(want) - want).norm(dim=-1) / size)[size > 0] for t in (got, plain))
    assert torch.equal(got.view_as(want)[size == 0], plain.view_as(want)[size == 0])
    print(case, name, setting, power, "outputs", error.max().item(), "token by token", least.max().item())
    assert (error <= 8 * 192 * 2.0 ** -24 + 4 * least).all()
    for row, slot in enumerate(SLOTS):
        copy = (STARTS[row] + LENGTHS[row]) & 1
        a, b, c = (z.double().view_as(states[row]) for z in (kept[slot, copy], kept_plain[slot, copy], states[row]))
        off, least = ((z - c).norm(dim=1) / c.norm(dim=1) for z in (a, b))         # a column each
        assert (off <= 8 * 192 * 2.0 ** -24 + 4 * least).all(), (off.max(), least.max())


@pytest.mark.parametrize("case", CASES)
def test_chunks_are_as_near_to_64_bits_as_tokens(case):
    """Outputs and states against a recurrence in 64 bits: a chunk's sums, of operands of 22 bits, are off by less than twice what the
    roundings of the decays and sums token by token come to.  (Left on the tensor cores, whose adder cuts off, they were off by up to
    six times that.)"""
    views, run, exact = CASES[case]()
    want, states = exact()
    errors = []
    for chunked in (False, True):
        out, kept = run(chunked)
        errors.append([norm_error(out.view_as(want), want)] + [norm_error(kept[slot, (start + n) & 1].view_as(state), state)
                                                               for slot, start, n, state in zip(SLOTS, STARTS, LENGTHS, states)])
    assert all(b < 2 * a + 2.0 ** -25 for a, b in zip(*errors)), errors


# ------------------------------------------------------------------------------------------- the choice, through the parts

def mixer_spec(kind, heads, dim, vdim):
    from fieldrun_b200.config.plan import PartSpec
    args = {"hidden_size": 256, "num_heads": heads, "norm_eps": 1e-6}
    if kind == "gated_linear_attention":
        args.update(head_dim=dim, value_dim=vdim, decay_rank=8, tau=16.0)
        names = ("q_proj", "k_proj", "v_proj", "gate_proj", "decay_in", "decay_out", "decay_bias", "out_norm", "o_proj")
    elif kind == "gated_delta_rule":
        args.update(num_kv_heads=heads // 2, head_dim=dim, value_dim=vdim, conv=4)
        names = ("q_proj", "k_proj", "v_proj", "beta_proj", "decay_proj", "gate_proj", "q_conv", "k_conv", "v_conv", "a_log", "dt_bias", "norm", "o_proj")
    else:
        args.update(value_dim=vdim, state=dim, groups=2, norm_groups=1, conv=4)
        names = ("in_proj", "conv", "conv_bias", "dt_bias", "a_log", "d", "norm", "o_proj")
    return PartSpec(kind, args, {n: "r/" + n for n in names})


def mixer(kind, heads, dim, vdim, dtype):
    from fieldrun_b200.parts import build_part

    class Source:
        def fetch(self, need):
            gen = torch.Generator(device=DEV).manual_seed(sum(need.name.encode()))
            value = torch.randn(need.shape, device=DEV, generator=gen) * (need.shape[-1] ** -0.5 if need.role == "matrix" else 0.3)
            return value.to(getattr(torch, dtype)) if need.role == "matrix" else value

    part = build_part("mixer", mixer_spec(kind, heads, dim, vdim), getattr(torch, dtype))
    part.load(Source())
    return part


@pytest.mark.parametrize("lengths", [[63], [64], [127, 5], [128], [191], [192, 5], [129, 300], [2] * 7 + [256], [1500]])
@pytest.mark.parametrize("kind", ["gated_linear_attention", "gated_delta_rule", "scalar_decay_state_space"])
def test_a_prompt_has_the_same_results_on_either_side_of_the_choice(kind, lengths, monkeypatch):
    """Steps below, at and beyond the lengths where the chunks begin to pay: what the part picks, chunks and token by token."""
    from fieldrun_b200.cache import SequenceCache
    from fieldrun_b200.engine.context import StepContext, Workspace
    part = mixer(kind, 8, 64, 64, "float32")
    act = torch.randn(sum(lengths), 256, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4))

    def run(chunks):
        if chunks is not None:
            monkeypatch.setattr(type(part), "chunks_pay", lambda self, ctx: chunks)
        cache = SequenceCache([part.cache_need()], max_tokens=64 * len(lengths) + sum(lengths), num_slots=len(lengths), dtype=torch.float32, device=DEV)
        part.prepare(cache.max_tokens, DEV)
        slots = [cache.alloc() for _ in lengths]
        cache.begin_step(slots, lengths)
        ctx = StepContext(Workspace(DEV), torch.float32, slots, [0] * len(lengths), lengths)
        update = part.forward(ctx, act, cache.line(0), True)
        states = cache.line(0).state.view(len(lengths), 2, -1)
        return update.clone(), [states[b, n & 1].clone() for b, n in enumerate(lengths)], part.chunks_pay(ctx)

    picked, chunked, plain = run(None), run(True), run(False)
    same = chunked if picked[2] else plain
    assert torch.equal(picked[0], same[0]) and all(torch.equal(a, b) for a, b in zip(picked[1], same[1]))
    assert norm_error(chunked[0], plain[0]) < LIMIT
    for a, b in zip(chunked[1], plain[1]):
        assert norm_error(a, b) < LIMIT


def test_short_steps_and_decode_steps_go_token_by_token_and_long_prompts_in_chunks():
    from fieldrun_b200.engine.context import StepContext, Workspace
    for kind in ("gated_linear_attention", "gated_delta_rule", "scalar_decay_state_space"):
        part, space = mixer(kind, 16, 64, 64, "bfloat16"), Workspace(DEV)
        pays = lambda lengths: part.chunks_pay(StepContext(space, torch.bfloat16, range(len(lengths)), [0] * len(lengths), lengths))
        assert not any(pays(lengths) for lengths in ([1], [1] * 64, [30], [63] * 8, [5] * 63 + [64]))
        assert all(pays(lengths) for lengths in ([2048], [2048] * 4, [1024] + [16] * 4))


def test_gated_linear_attention_takes_a_norm_weight_at_any_offset():
    """The output norm's weight as a view that does not begin on eight bytes: the results of the same weight at a boundary."""
    heads, dim, vdim, rank, tokens = 2, 64, 64, 8, 130
    gen = torch.Generator(device=DEV).manual_seed(5)
    offsets = (0, heads * dim, 2 * heads * dim, 3 * heads * dim, 4 * heads * dim)
    proj = torch.randn(tokens, offsets[4] + rank, device=DEV, generator=gen)
    a2, bias = torch.randn(heads * dim, rank, device=DEV, generator=gen), torch.randn(heads * dim, device=DEV, generator=gen)
    store, results = torch.randn(vdim + 1, device=DEV, generator=gen), []
    for norm in (store[1:], store[1:].clone()):
        state, out = torch.zeros(1, 2, heads, dim, vdim, device=DEV), torch.empty(tokens, heads * vdim, device=DEV)
        chunks = tables([tokens], 64)
        ops().gla_chunks(proj, offsets, a2, bias, norm, state, i32([0]), i32([0]), i32([0, tokens]), out, heads=heads, dim=dim, vdim=vdim, tau=16.0,
                         q_scale=0.125, eps=1e-6, chunks=chunks,
                         scratch=torch.empty(ops().gla_chunks_scratch_floats(chunks[0].numel(), tokens, heads, dim, vdim), device=DEV))
        results.append(out)
    assert torch.equal(*results)


def test_state_space_steps_on_either_side_of_the_line():
    """Below 128 tokens none; up to 191 those that are about twice as fast; from 192 on wherever chunks cost less."""
    from fieldrun_b200.engine.context import StepContext, Workspace
    space = Workspace(DEV)
    for heads, n, vdim, some, none in ((64, 128, 64, ([128] * 16, [191] * 16, [192], [192] * 16), ([127] * 64, [128], [130] * 16, [191])),
                                       (16, 128, 128, ([128] * 32, [191], [192]), ([127] * 64, [128] * 4)), (8, 64, 64, ([192],), ([128], [191]))):
        part = mixer("scalar_decay_state_space", heads, n, vdim, "bfloat16")
        pays = lambda lengths: part.chunks_pay(StepContext(space, torch.bfloat16, range(len(lengths)), [0] * len(lengths), lengths))
        assert [pays(lengths) for lengths in some] == [True] * len(some) and [pays(lengths) for lengths in none] == [False] * len(none)


# the chunks of 64 tokens that have such a number: the first and the last of a sequence, neighbours, all
@pytest.mark.parametrize("hits", [[0], [1, 2], [11], [0, 5, 11], list(range(12))])
@pytest.mark.parametrize("case,name", [(c, "x") for c in ("state space", "state space 128")] + [("delta 128", "v")])
@pytest.mark.parametrize("number", [2.0 ** 50, NAN])
def test_prompts_taken_token_by_token_after_all(case, name, hits, number, monkeypatch):
    """A large token cleared four tokens on, against 64 bits; and NaNs in one entry, cleared by nothing: where token by token has them."""
    import sys
    lengths, starts, slots = [719, 768, 300], [0, 3, 10], [1, 0, 2]
    for what, value in (("LENGTHS", lengths), ("STARTS", starts), ("SLOTS", slots), ("AT", [0, *(int(c) for c in np.cumsum(lengths))])):
        monkeypatch.setattr(sys.modules[__name__], what, value)
    views, run, exact = CASES[case]()
    for begin, length in zip(AT, lengths):
        for chunk in hits:
            t = 64 * chunk + 20
            if t + 4 < length:
                if number == number:
                    views[name][begin + t] *= number
                    views["decay"][begin + t + 4] = 200.0
                else:
                    views[name][begin + t, 3] = number
    got, kept = run(True)
    plain, kept_plain = run(False)
    if number != number:
        assert torch.equal(got.isfinite(), plain.isfinite()) and got.isnan().any()
        fine = plain.isfinite()
        assert norm_error(got[fine], plain[fine]) < LIMIT
    else:
        want, _ = exact()
        error, least = ((t.double().view_as(want) - want).norm(dim=-1) / want.norm(dim=-1) for t in (got, plain))
        assert (error <= 8 * 192 * 2.0 ** -24 + 4 * least).all()
    for length, start, slot in zip(lengths, starts, slots):
        a, b = kept[slot, (start + length) & 1], kept_plain[slot, (start + length) & 1]
        assert torch.equal(a.isfinite(), b.isfinite()) and norm_error(a[b.isfinite()], b[b.isfinite()]) < LIMIT


@pytest.mark.parametrize("case,name", [("state space 128", "x"), ("delta 128", "v")])
def test_one_number_that_is_not_finite_does_not_make_a_prompt_slow(case, name, monkeypatch):
    """Prompts of 2,048 tokens, one with an infinity in the middle, or with a large token that a decay clears: less than twelve times as
    long as without (the prompt token by token with one thread a column took 46 times as long)."""
    import sys
    for what, value in (("LENGTHS", [2048] * 5), ("STARTS", [0] * 5), ("SLOTS", [0, 1, 2, 3, 4]), ("AT", [2048 * i for i in range(6)])):
        monkeypatch.setattr(sys.modules[__name__], what, value)
    views, run, _ = CASES[case]()

    def shortest():
        times = []
        for _ in range(5):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            run(True)
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times[1:])

    clean = shortest()
    for rows in (slice(0, 9), slice(500, 520), slice(2048, 2120)):               # rows of zeros are results, not a loss of digits
        for what in ("x", "c") if name == "x" else ("q", "k", "v"):
            views[what][rows] = 0.0
    assert shortest() < 2 * clean
    views[name][1000] *= 1e12
    views["decay"][1004] = 200.0
    assert shortest() < 12 * clean
    views[name][1000, 1] = INF
    assert shortest() < 12 * clean


GATES = {"subnormal": (1e-45, 1e-38), "tiny": (1e-38, 1e-8), "small": (1e-8, 0.1), "about one": (0.1, 4.0), "some": (4.0, 20.0), "large": (20.0, 60.0),
         "up to 80": (60.0, 79.9999), "around 80": (79.5, 80.5), "beyond": (80.0, 200.0)}


def gates_of(size, sign, tokens, width):
    """A million of that size and sign for 4,096 x 256, zeros, infinities and NaNs among them."""
    gen = torch.Generator(device=DEV).manual_seed(7)
    low, high = GATES[size]
    spread = torch.rand(tokens, width, device=DEV, generator=gen, dtype=torch.float64)
    gates = (sign * torch.exp(spread * np.log(high / low)) * low).float()
    for row, odd in ((70, INF), (200, -INF), (330, NAN), (460, 0.0), (590, -0.0), (720, 500.0), (850, -500.0)):
        gates[row, ::7] = odd
    return gates


def same_bits(plain, got, gates):
    assert torch.equal(plain.isnan(), got.isnan()) and plain.isnan().any()
    differ = (plain.view(torch.int32) != got.view(torch.int32)) & ~plain.isnan()
    assert not differ.any(), (differ.sum().item(), gates[differ][:5].tolist(), plain[differ][:5].tolist(), got[differ][:5].tolist())


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("size", GATES)
def test_gates_have_the_bits_of_the_division(size, sign):
    """x and D of one and a B of zeros: the outputs are z / (1 + exp(-z)), in chunks by a reciprocal and one correction below 80, token by
    token by a division."""
    heads, groups, n, vdim, tokens = 4, 1, 64, 64, 4096
    inner = heads * vdim
    proj = torch.zeros(tokens, inner + heads, device=DEV)
    proj[:, :inner] = gates_of(size, sign, tokens, inner)
    xbc = torch.ones(tokens, inner + 2 * groups * n, device=DEV)
    xbc[:, inner:] = 0.0
    zeros, ones = torch.zeros(heads, device=DEV), torch.ones(heads, device=DEV)
    sizes, tabs, results = dict(heads=heads, vdim=vdim, n=n, groups=groups), Tables([tokens], [0], [0]), []
    for chunked in (False, True):
        state, out = torch.zeros(1, 2, heads * n * vdim, device=DEV), torch.full((tokens, inner), NAN, device=DEV)
        args = (proj, 0, inner, xbc, inner, inner + groups * n, zeros, zeros, ones, tabs, state, 0, out)
        if chunked:
            chunks = tables([tokens], 128)
            scratch = torch.full((ops().state_space_chunks_scratch_floats(chunks[0].numel(), **sizes),), NAN, device=DEV)
            ops().state_space_chunks(*args, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().state_space_scan(*args, **sizes)
        results.append(out)
    same_bits(*results, proj[:, :inner])


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("size", GATES)
def test_gates_of_linear_attention_have_the_bits_of_the_division(size, sign):
    """Decays of zero, one entry of q and k, values of one and no epsilon: every normed output is one, and the results are the gates."""
    heads, dim, vdim, rank, tokens = 4, 64, 64, 4, 4096
    qk, inner = heads * dim, heads * vdim
    offsets = (0, qk, 2 * qk, 2 * qk + inner, 2 * qk + 2 * inner)
    proj = torch.zeros(tokens, offsets[4] + rank, device=DEV)
    proj[:, 0:2 * qk:dim] = 1.0
    proj[:, offsets[2]:offsets[3]] = 1.0
    gates = proj[:, offsets[3]:offsets[4]]
    gates[:] = gates_of(size, sign, tokens, inner)
    a2, bias, norm = torch.zeros(qk, rank, device=DEV), torch.full((qk,), -1000.0, device=DEV), torch.ones(vdim, device=DEV)
    sizes, results = dict(heads=heads, dim=dim, vdim=vdim, tau=1.0, q_scale=1.0, eps=0.0), []
    for chunked in (False, True):
        state, out = torch.zeros(1, 2, heads, dim, vdim, device=DEV), torch.full((tokens, inner), NAN, device=DEV)
        args = (proj, offsets, a2, bias, norm, state, i32([0]), i32([0]), i32([0, tokens]), out)
        if chunked:
            chunks = tables([tokens], 64)
            scratch = torch.full((ops().gla_chunks_scratch_floats(chunks[0].numel(), tokens, heads, dim, vdim),), NAN, device=DEV)
            ops().gla_chunks(*args, chunks=chunks, scratch=scratch, **sizes)
        else:
            ops().gla_scan(*args, **sizes)
        results.append(out)
    same_bits(*results, gates)
