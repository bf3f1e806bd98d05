"""The float32 path's own kernels against the general ones, at the edges of their tiles and over all forms that they take."""
import numpy as np
import pytest
import torch

from fieldrun_b200.engine.context import StepContext, Workspace

pytestmark = pytest.mark.gpu

DEV = "cuda"


def ops():
    from fieldrun_b200.csrc import ops as o
    return o


def i32(values):
    return torch.tensor(np.asarray(values), dtype=torch.int32, device=DEV)


def paged(starts, lengths, k_heads, v_heads, dim, vdim, seed):
    """Pages in a scrambled order, filled with numbers to the end, for sequences that hold starts + lengths tokens."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    need = [(s + n + 63) // 64 for s, n in zip(starts, lengths)]
    order = np.random.default_rng(seed).permutation(sum(need) + 3)
    keys = torch.randn(len(order), k_heads, 64, dim, device=DEV, generator=gen)
    values = torch.randn(len(order), v_heads, vdim, 64, device=DEV, generator=gen)
    table = np.full((len(starts), max(need)), -1, dtype=np.int32)
    at = 0
    for row, count in enumerate(need):
        table[row, :count] = order[at:at + count]
        at += count
    return keys, values, i32(table), gen


FORMS = {
    "plain": {},
    "window": dict(window=70),
    "window beside first tokens": dict(window=37, keep_first=5),
    "chunks, sinks, gates": dict(chunk=48, sinks=True, gate=True),
    "slopes": dict(slopes=True),
    "cap": dict(softcap=3.0),
}
SHAPES = [(6, 2, 32, 32, 1), (8, 8, 64, 64, 1), (12, 2, 128, 128, 1), (9, 1, 96, 96, 1), (8, 4, 64, 128, 2), (6, 3, 12, 20, 1), (2, 1, 100, 7, 1)]


def options(form, heads, tokens, gen):
    made = dict(window=None)
    made.update({k: v for k, v in FORMS[form].items() if v is not True})
    if FORMS[form].get("sinks"):
        made["sinks"] = torch.randn(heads, device=DEV, generator=gen)
    if FORMS[form].get("slopes"):
        made["slopes"] = torch.rand(heads, device=DEV, generator=gen) * 0.2
    if FORMS[form].get("gate"):
        made["gate"] = torch.randn(tokens, heads + 3, device=DEV, generator=gen)
    return made


def check(got, want, keys):
    """Both sides are float32 sums of at most `keys` weighted values, whose weights carry the rounding of a product of at most
    128 entries: the difference stays below (128 + keys / 8) roundings of the largest result."""
    error = (got - want).abs().max().item() / want.abs().max().item()
    assert torch.isfinite(got).all() and error < (128 + keys / 8) * 2.0 ** -24, error


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps", SHAPES)
def test_prompts_in_tiles_equal_the_general_kernel(heads, kv_heads, dim, vdim, maps, form):
    assert ops().attention_f32_tiles_take(dim, vdim)
    starts, lengths = [0, 3, 0, 130, 64], [1, 64, 65, 200, 127]
    keys, values, table, gen = paged(starts, lengths, kv_heads, kv_heads // maps, dim, vdim, 3)
    tokens = sum(lengths)
    q = torch.randn(tokens, heads * dim, device=DEV, generator=gen)
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, v_dim=vdim, scale=dim ** -0.5, maps=maps,
                  **options(form, heads, tokens, gen))
    pos = np.concatenate([s + np.arange(n) for s, n in zip(starts, lengths)])
    want, got = (torch.full((tokens, heads * vdim), float("nan"), device=DEV) for _ in range(2))
    ops().attention_generic(q, keys, values, table, i32(pos), i32(np.repeat(np.arange(5), lengths)), want, **common)
    tiles = [(b, q0) for b, n in enumerate(lengths) for q0 in range(0, n, 128)]
    ops().attention_f32_tiles(q, keys, values, table, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), i32(range(5)), i32(starts),
                              i32(lengths), i32(np.concatenate([[0], np.cumsum(lengths)])), got, **common)
    check(got, want, 330)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps", [s for s in SHAPES if s[2] % 32 == 0] + [(10, 1, 64, 64, 1), (20, 1, 32, 32, 1)])
def test_single_tokens_in_chunks_equal_the_general_kernel(heads, kv_heads, dim, vdim, maps, form):
    assert ops().attention_f32_token_takes(dim, vdim)
    lengths = [1, 64, 65, 256, 257, 700]
    keys, values, table, gen = paged([0] * 6, lengths, kv_heads, kv_heads // maps, dim, vdim, 4)
    q = torch.randn(6, heads * dim, device=DEV, generator=gen)
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, v_dim=vdim, scale=dim ** -0.5, maps=maps,
                  **options(form, heads, 6, gen))
    pos, slots = i32([n - 1 for n in lengths]), i32(range(6))
    want, got = (torch.full((6, heads * vdim), float("nan"), device=DEV) for _ in range(2))
    ops().attention_generic(q, keys, values, table, pos, slots, want, **common)
    chunks = 4                                                    # more than the longest sequence needs
    part_o = torch.full((6, heads, chunks, vdim), float("nan"), device=DEV)
    part_ml = torch.full((6, heads, chunks, 2), float("nan"), device=DEV)
    ops().attention_f32_token(q, keys, values, table, pos, slots, part_o, part_ml, got, max_chunks=chunks, **common)
    check(got, want, 700)


@pytest.mark.parametrize("paired,limit", [(True, 0.0), (True, 2.0), (False, 0.0)])
@pytest.mark.parametrize("features,inner", [(1, 4), (7, 96), (16, 128), (17, 132), (48, 1024), (130, 3072)])
def test_rows_equal_the_general_kernel(features, inner, paired, limit):
    """Tiles of 1 to 8 rows, experts without rows, features and inner sizes that fill no warp or run.  Both sides round the
    products of `inner` terms of size one: their sums differ by less than inner roundings of the largest."""
    gen = torch.Generator(device=DEV).manual_seed(features + inner)
    counts = [1, 0, 2, 3, 8, 5, 11]
    offsets = np.concatenate([[0], np.cumsum(counts)])
    total = int(offsets[-1])
    w = torch.randn(len(counts), (2 if paired else 1) * features, inner, device=DEV, generator=gen) * inner ** -0.5
    x = torch.randn(9, inner, device=DEV, generator=gen)
    source = i32(np.random.default_rng(1).integers(0, 9, size=total))
    tiles = [(e, offsets[e] + r) for e, n in enumerate(counts) for r in range(0, n, 8)]
    lists = (i32([t[0] for t in tiles] + [0]), i32([t[1] for t in tiles] + [0]), i32([len(tiles)]), i32(offsets), len(tiles) + 1)
    want, got = (torch.full((total, features), float("nan"), device=DEV) for _ in range(2))
    ops().expert_gemm_generic(w, x, source, *lists, want, paired=paired, gate_limit=limit)
    ops().rows_f32(w, x, source, *lists, got, paired=paired, gate_limit=limit)
    assert torch.isfinite(got).all()
    assert (got - want).abs().max() < 4 * max(inner, 16) * 2.0 ** -24 * max(want.abs().max().item(), 1.0)


# Groups of eight weight rows a block, runs of the inner size a warp: one run of several warps and blocks an SM (three groups), of eight warps
# and one block; two, three and four runs (three groups; five for seven and eight rows, whose blocks come in pairs); five runs and more (one
# block an SM; six and four warps of several, three groups and more).  The last block's last group is never whole.
@pytest.mark.parametrize("features,inner", [(1, 4), (7, 96), (130, 132), (43013, 100), (14501, 132), (7205, 516), (3077, 1024), (3077, 1536), (3077, 3072),
                                            (3077, 4100), (3077, 6144), (74, 6200), (7205, 6200), (9597, 6200), (3077, 12300)])
def test_dense_rows_of_every_number(features, inner):
    """Parts of the inner size that fill no run, one to many of them, shares of a block that end inside eight weight rows; inputs and results
    behind the last row stay as they are.  Sums of `inner` terms of size one: off by less than inner roundings of the largest.  A row's bits
    do not depend on the other rows."""
    gen = torch.Generator(device=DEV).manual_seed(features + inner)
    w = torch.randn(features, inner, device=DEV, generator=gen) * inner ** -0.5
    all_rows = torch.randn(8, inner, device=DEV, generator=gen)
    want = all_rows.double() @ w.double().T
    alone = torch.empty(8, features, device=DEV)
    for row in range(8):
        ops().dense_rows_f32(w, all_rows[row:row + 1], alone[row:row + 1])
    for rows in range(1, 9):
        x = torch.full((rows + 1, inner), float("nan"), device=DEV)
        x[:rows] = all_rows[:rows]
        got = torch.full((rows + 1, features), 7.0, device=DEV)
        ops().dense_rows_f32(w, x[:rows], got[:rows], weights_final=rows % 2 == 0)
        assert (got[:rows] - want[:rows]).abs().max() < 2 * max(inner, 16) * 2.0 ** -24 * max(want.abs().max().item(), 1.0)
        assert torch.equal(got[:rows], alone[:rows])
        assert (got[rows] == 7.0).all()


@pytest.mark.parametrize("features,inner", [(65536, 1024), (65544, 1024), (131073, 516)])
def test_a_row_of_a_float32_product_is_the_same_in_any_company(features, inner):
    """The largest weight that the dense products' kernel takes, and larger ones."""
    from fieldrun_b200.parts.linear import DENSE_ROWS_ENTRIES, linear, require_true_float32
    require_true_float32()
    assert (features * inner <= DENSE_ROWS_ENTRIES) == (features == 65536)
    gen = torch.Generator(device=DEV).manual_seed(features)
    w, x = torch.randn(features, inner, device=DEV, generator=gen) * inner ** -0.5, torch.randn(8, inner, device=DEV, generator=gen)
    together, want = linear(x, w), x.double() @ w.double().T
    assert (together - want).abs().max() < 2 * inner * 2.0 ** -24 * want.abs().max()
    for first, rows in ((0, 1), (7, 1), (3, 2), (0, 5), (1, 7)):
        assert torch.equal(linear(x[first:first + rows], w), together[first:first + rows])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_products_of_a_weight_that_the_kernel_before_wrote(dtype):
    from fieldrun_b200.parts.linear import linear, require_true_float32
    require_true_float32()
    gen = torch.Generator(device=DEV).manual_seed(3)
    drawn, x = torch.randn(8192, 3072, device=DEV, generator=gen).to(dtype), torch.randn(4, 3072, device=DEV, generator=gen).to(dtype)
    w, once = drawn.clone(), linear(x, drawn)
    torch.cuda.synchronize()
    for power in range(12):
        torch.mul(drawn, 2.0 ** power, out=w)
        assert torch.equal(linear(x, w), once * 2.0 ** power)


def split_product(w, x, lists=None, max_tiles=0, source=None, gated=False, limit=0.0):
    """w [E, F, K] times the rows of x (of ``source``) by the tensor cores' float32 products."""
    count = len(source) if source is not None else x.shape[0]
    parts = torch.full((2, count, w.shape[2]), float("nan"), dtype=torch.float16, device=DEV)
    scale, out = torch.full((count,), float("nan"), device=DEV), torch.full((count, w.shape[1]), float("nan"), device=DEV)
    ops().products_f32(w, ops().weight_scales(w), x, parts, scale, out, x_rows=source, gated=gated, gate_limit=limit, lists=lists,
                       max_tiles=max_tiles)
    ops().tc_status_check(out.device)
    return out


def relative(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("rows,features,inner", [(1, 1, 8), (16, 128, 64), (17, 130, 72), (128, 256, 256), (129, 100, 264), (300, 384, 1000),
                                                 (64, 512, 3072), (1000, 640, 6144)])
def test_split_products_are_as_exact_as_float32(rows, features, inner):
    """Tails of the rows, features and inner size, more items than blocks, chunks of 256 entries that end early.  The products
    carry 22 bits, and the sums of 256 entries that are cut off are added rounded: errors of a few 2^-23 of the size that a sum of
    entries of random signs has."""
    gen = torch.Generator(device=DEV).manual_seed(rows + inner)
    x = torch.randn(rows, inner, device=DEV, generator=gen) * torch.exp(3 * torch.randn(rows, 1, device=DEV, generator=gen))
    w = torch.randn(1, features, inner, device=DEV, generator=gen) * torch.exp(3 * torch.randn(1, features, 1, device=DEV, generator=gen))
    x[rows // 2] *= 0.0 if rows > 1 else 1.0
    got, want = split_product(w, x), x.double() @ w[0].double().T
    size = x.double().norm(dim=1, keepdim=True) * w[0].double().norm(dim=1)[None]
    assert ((got.double() - want).abs() <= 8 * 2.0 ** -23 * size).all()


@pytest.mark.parametrize("rows,features,inner", [(1500, 6144, 2048), (1930, 4100, 200), (161, 21000, 320), (40, 40000, 64)])
def test_split_products_of_several_items_a_block(rows, features, inner):
    """A block goes on from item to item with its rings and accumulators at any place, while
    the item before is written: the same bounds as for a single item."""
    gen = torch.Generator(device=DEV).manual_seed(rows)
    x, w = torch.randn(rows, inner, device=DEV, generator=gen), torch.randn(1, features, inner, device=DEV, generator=gen)
    for _ in range(3):
        got, want = split_product(w, x), x.double() @ w[0].double().T
        size = x.double().norm(dim=1, keepdim=True) * w[0].double().norm(dim=1)[None]
        assert ((got.double() - want).abs() <= 8 * 2.0 ** -23 * size).all()


@pytest.mark.parametrize("limit", [0.0, 1.5])
def test_split_products_of_experts(limit):
    """Expert lists: gathered rows, tiles of 1 to 160 rows, each output of one tile alone, an expert without rows and some of several tiles,
    the gated second half."""
    gen = torch.Generator(device=DEV).manual_seed(5)
    counts, hidden, width = [1, 0, 130, 128, 15, 400, 159, 160, 161, 320], 96, 72
    offsets = np.concatenate([[0], np.cumsum(counts)])
    total = int(offsets[-1])
    w13 = torch.randn(len(counts), 2 * width, hidden, device=DEV, generator=gen) * hidden ** -0.5
    w2 = torch.randn(len(counts), hidden, width, device=DEV, generator=gen)
    x = torch.randn(50, hidden, device=DEV, generator=gen)
    source = i32(np.random.default_rng(1).integers(0, 50, size=total))
    tiles = [(e, offsets[e] + r) for e, n in enumerate(counts) for r in range(0, n, ops().PRODUCTS_F32_TILE)]
    lists = (i32([t[0] for t in tiles] + [0]), i32([t[1] for t in tiles] + [0]), i32([len(tiles)]), i32(offsets))
    both = split_product(w13, x, lists, len(tiles) + 1, source)
    got = split_product(w2, both, lists, len(tiles) + 1, gated=True, limit=limit)
    rows = x.double()[source.long()]
    for e, n in enumerate(counts):
        if n == 0:
            continue
        part = slice(int(offsets[e]), int(offsets[e + 1]))
        assert relative(both[part], rows[part] @ w13[e].double().T) < 4 * 2.0 ** -23
        gate, up = both[part].double().split(width, dim=1)
        if limit:
            gate = gate.clamp_max(limit)
            unit = gate * torch.sigmoid(1.702 * gate) * (up.clamp(-limit, limit) + 1)
        else:
            unit = torch.nn.functional.silu(gate) * up
        assert relative(got[part], unit @ w2[e].double().T) < 6 * 2.0 ** -23      # the unit's own rounding besides


def test_split_products_keep_infinities_nans_and_far_exponents():
    gen = torch.Generator(device=DEV).manual_seed(6)
    x, w = torch.randn(140, 72, device=DEV, generator=gen), torch.randn(1, 130, 72, device=DEV, generator=gen)
    x[3, 5], x[133, 0], x[7, 1] = float("inf"), float("nan"), 3e38
    x[8] *= 1e-30
    x[9] *= 1e-42
    w[0, 129, 2], w[0, 1, 3] = -float("inf"), float("nan")
    w[0, 4] *= 1e-20
    w[0, 5] *= 1e30
    got, want = split_product(w, x), torch.stack([(x[r][None] * w[0]).sum(1) for r in range(140)])
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    fine = want.isfinite() & (want.abs() > 1e-36)                 # results that float32 holds to its full precision
    size = x.double().abs() @ w[0].double().abs().T
    assert ((got.double() - want.double()).abs() <= 1e-5 * size + 2e-43)[fine].all()


@pytest.mark.parametrize("top_k", [1, 3, 4, 8, 9])
@pytest.mark.parametrize("width", [4, 96, 1028, 3072])
def test_weighted_sums_of_four_columns_equal_those_of_one(width, top_k):
    """The same sums in the same order: the bits of rows that lie one float off, which take a column a thread."""
    gen = torch.Generator(device=DEV).manual_seed(width + top_k)
    y, weights = torch.randn(7 * top_k, width, device=DEV, generator=gen), torch.rand(7, top_k, device=DEV, generator=gen)
    rows = torch.randperm(7 * top_k, device=DEV, generator=gen).to(torch.int32)
    results = []
    for shift in (0, 1):
        held = torch.zeros(y.numel() + 4, device=DEV)
        shifted = held[shift:shift + y.numel()].view_as(y)
        shifted.copy_(y)
        out = torch.full((7, width), float("nan"), device=DEV)
        ops().expert_combine(shifted, weights, rows, out)
        results.append(out)
    assert torch.isfinite(results[0]).all() and torch.equal(*results)


def plant(keys, values, table, row, position, key=None, value=None):
    """A number in one entry of the key, or in one or every entry of the value, of a sequence's token."""
    page, at = int(table[row, position // 64]), position % 64
    if key is not None:
        keys[page, :, at, 1] = key
    if value is not None:
        values[page, :, :3, at] = value


def same_but_for_rounding(got, want, keys):
    """NaNs and infinities in the same places, and everything else as close as ever."""
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    fine = want.isfinite()
    assert fine.any() and not fine.all()
    check(got[fine], want[fine], keys)


INF, NAN = float("inf"), float("nan")


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps", [SHAPES[0], SHAPES[2], SHAPES[3], SHAPES[4]])
def test_values_that_a_token_does_not_see_do_not_reach_it(heads, kv_heads, dim, vdim, maps, form):
    """Single tokens: numbers that are not finite behind a sequence's last token (what an earlier sequence left in the page), and,
    where a window or a chunk ends, before the first key seen.  One that is seen reaches the result as in the general kernel."""
    lengths = [1, 64, 65, 256, 257, 700, 130]
    count = len(lengths)
    keys, values, table, gen = paged([0] * count, lengths, kv_heads, kv_heads // maps, dim, vdim, 8)
    for row, n in enumerate(lengths):
        for at in range(n, (n + 63) // 64 * 64):
            plant(keys, values, table, row, at, NAN, NAN if at % 2 else INF)
    for row in (4, 5):
        plant(keys, values, table, row, lengths[row] - 72, NAN, INF)     # hidden by the windows and the chunks, seen without
    plant(keys, values, table, 6, 129, value=INF)                        # seen by all
    plant(keys, values, table, 6, 128, key=3.4e38)
    q = torch.randn(count, heads * dim, device=DEV, generator=gen)
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, v_dim=vdim, scale=dim ** -0.5, maps=maps,
                  **options(form, heads, count, gen))
    pos, slots = i32([n - 1 for n in lengths]), i32(range(count))
    want, got = (torch.full((count, heads * vdim), NAN, device=DEV) for _ in range(2))
    ops().attention_generic(q, keys, values, table, pos, slots, want, **common)
    part_o, part_ml = torch.full((count, heads, 3, vdim), NAN, device=DEV), torch.full((count, heads, 3, 2), NAN, device=DEV)
    ops().attention_f32_token(q, keys, values, table, pos, slots, part_o, part_ml, got, max_chunks=3, **common)
    same_but_for_rounding(got, want, 700)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps", [SHAPES[0], SHAPES[2], SHAPES[4], SHAPES[5], SHAPES[6]])
def test_infinities_and_nans_reach_the_queries_that_see_them(heads, kv_heads, dim, vdim, maps, form):
    """Prompts: a token's value, key or query that is not finite, or so large that a part of it is not, changes the results of the
    queries that see it and of no others; what lies behind a sequence's last token changes none."""
    starts, lengths = [0, 3, 0, 130, 64], [1, 64, 65, 200, 127]
    keys, values, table, gen = paged(starts, lengths, kv_heads, kv_heads // maps, dim, vdim, 9)
    tokens, ends = sum(lengths), [s + n for s, n in zip(starts, lengths)]
    for row, n in enumerate(ends):
        for at in range(n, (n + 63) // 64 * 64):
            plant(keys, values, table, row, at, NAN, NAN if at % 2 else INF)
    plant(keys, values, table, 1, 40, value=INF)
    plant(keys, values, table, 2, 63, value=NAN)
    plant(keys, values, table, 2, 64, value=-3.4028234e38)               # rounds to an infinity as a part
    plant(keys, values, table, 3, 100, key=INF, value=-INF)
    plant(keys, values, table, 3, 300, key=NAN)
    plant(keys, values, table, 4, 100, key=3.4028234e38)
    q = torch.randn(tokens, heads * dim, device=DEV, generator=gen)
    q[tokens - 10, 2], q[tokens - 5, 1] = INF, NAN
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, v_dim=vdim, scale=dim ** -0.5, maps=maps,
                  **options(form, heads, tokens, gen))
    pos = np.concatenate([s + np.arange(n) for s, n in zip(starts, lengths)])
    want, got = (torch.full((tokens, heads * vdim), NAN, device=DEV) for _ in range(2))
    ops().attention_generic(q, keys, values, table, i32(pos), i32(np.repeat(np.arange(5), lengths)), want, **common)
    tiles = [(b, q0) for b, n in enumerate(lengths) for q0 in range(0, n, 128)]
    ops().attention_f32_tiles(q, keys, values, table, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), i32(range(5)), i32(starts),
                              i32(lengths), i32(np.concatenate([[0], np.cumsum(lengths)])), got, **common)
    same_but_for_rounding(got, want, 330)


@pytest.mark.parametrize("inner", [8, 256, 3072])
@pytest.mark.parametrize("spread", [0, 20, 60])
def test_split_products_of_rows_whose_entries_lie_far_apart(inner, spread):
    """Entries over 2^spread either way in every row of both operands, rows and weight rows with a single entry that is not zero, and an
    entry 2^40 above the rest that the weights leave out: every output within 2^-21 (two operands of 22 bits, and the product of their
    small parts) and a float32 sum's roundings of the sum of its terms' sizes, which no norm of a row hides."""
    gen = torch.Generator(device=DEV).manual_seed(inner + spread)
    x, w = torch.randn(40, inner, device=DEV, generator=gen), torch.randn(1, 150, inner, device=DEV, generator=gen)
    x, w = (t * torch.exp2((torch.rand(t.shape, device=DEV, generator=gen) * 2 - 1) * spread) for t in (x, w))
    for r in range(8):
        x[r], x[r, r] = 0.0, 1.7 * 2.0 ** -r
    for f in range(64):
        w[0, f], w[0, f, f % inner] = 0.0, 1.3
    x[20:30, 0], w[0, 100:, 0] = 2.0 ** 40, 0.0
    x[31], w[0, 99] = 0.0, 0.0
    got, want = split_product(w, x).double(), x.double() @ w[0].double().T
    size = x.double().abs() @ w[0].double().abs().T
    assert ((got - want).abs() <= (2.0 ** -21 + inner ** 0.5 * 2.0 ** -24) * size).all()
    assert (got[31] == 0).all() and (got[:, 99] == 0).all()


@pytest.mark.parametrize("factor", [1e9, 1e-9, 0.0])
def test_split_products_of_weights_written_after_their_scales(factor):
    """Scales are made when weights are loaded; weights of another size written in their place later give the products of the new ones."""
    gen = torch.Generator(device=DEV).manual_seed(7)
    x, w = torch.randn(30, 264, device=DEV, generator=gen), torch.randn(1, 140, 264, device=DEV, generator=gen)
    w[0, 0] = 0.0
    scales = ops().weight_scales(w)
    w.mul_(factor)
    w[0, 0, 3] = 1.0
    w[0, 1, 1] = INF
    parts, scale = torch.empty(2, 30, 264, dtype=torch.float16, device=DEV), torch.empty(30, device=DEV)
    out = torch.empty(30, 140, device=DEV)
    ops().products_f32(w, scales, x, parts, scale, out)
    ops().tc_status_check(out.device)
    want, fine = x.double() @ w[0].double().T, w[0].isfinite().all(1)
    assert torch.equal(out[:, 1].double(), want[:, 1])                       # an infinity, as the entries of x give it its sign
    assert ((out.double() - want).abs()[:, fine] <= 2.0 ** -20 * (x.double().abs() @ w[0].double().abs().T)[:, fine]).all()


@pytest.mark.parametrize("tokens", [3, 700])
def test_experts_take_rows_at_any_offset(tokens):
    """Rows that do not begin on 16 bytes, few of them (the stream over the weights) and many (the split products)."""
    from fieldrun_b200.config.plan import PartSpec
    from fieldrun_b200.engine.context import StepContext, Workspace
    from fieldrun_b200.parts import build_part

    class Source:
        def fetch(self, need):
            gen = torch.Generator(device=DEV).manual_seed(sum(need.name.encode()))
            return torch.randn(need.shape, device=DEV, generator=gen) * need.shape[-1] ** -0.5

    hidden = 512
    part = build_part("feed_forward", PartSpec("routed_experts", {"hidden_size": hidden, "num_experts": 4, "top_k": 2, "expert_width": 256,
                                                                  "renormalize": True},
                                               {"router": "r", "w_gate": "{e}g", "w_up": "{e}u", "w_down": "{e}d"}), torch.float32)
    part.load(Source())
    assert part.on_split_products(2 * tokens) == (tokens == 700)
    ctx = StepContext(Workspace(DEV), torch.float32, [0], [0], [tokens])
    rows = torch.randn(tokens, hidden, device=DEV)
    shifted = torch.zeros(rows.numel() + 1, device=DEV)[1:].view_as(rows).copy_(rows)
    assert torch.equal(part.forward(ctx, shifted, rows).clone(), part.forward(ctx, rows, rows))


@pytest.mark.parametrize("heads,kv_heads,dim", [(6, 2, 32), (8, 8, 64), (12, 2, 128), (6, 3, 12)])
def test_float32_attention_is_as_near_to_64_bits_as_the_general_kernel(heads, kv_heads, dim):
    """Prompts in tiles and single tokens in chunks against a softmax in 64 bits: off by no more than twice what the general kernel's
    roundings come to on the same inputs."""
    starts, lengths = [0, 130], [300, 129]
    keys, values, table, gen = paged(starts, lengths, kv_heads, kv_heads, dim, dim, 11)
    tokens = sum(lengths)
    q = torch.randn(tokens, heads * dim, device=DEV, generator=gen)
    pos = np.concatenate([s + np.arange(n) for s, n in zip(starts, lengths)])
    slots, common = np.repeat(np.arange(2), lengths), dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, scale=dim ** -0.5, window=None)
    exact = torch.empty(tokens, heads, dim, dtype=torch.float64, device=DEV)
    for row in range(2):
        held, mine = starts[row] + lengths[row], slice(*(int(c) for c in np.searchsorted(slots, [row, row + 1])))
        pages = table[row, :(held + 63) // 64].long()
        k = keys[pages].double().permute(1, 0, 2, 3).reshape(kv_heads, -1, dim)[:, :held].repeat_interleave(heads // kv_heads, 0)
        v = values[pages].double().permute(1, 0, 3, 2).reshape(kv_heads, -1, dim)[:, :held].repeat_interleave(heads // kv_heads, 0)
        scores = q[mine].double().view(-1, heads, dim).transpose(0, 1) @ k.transpose(1, 2) * dim ** -0.5
        hidden = torch.arange(held, device=DEV)[None] > torch.as_tensor(pos[mine], device=DEV)[:, None]
        exact[mine] = (scores.masked_fill(hidden, -INF).softmax(-1) @ v).transpose(0, 1)
    exact = exact.view(tokens, heads * dim)
    general, tiles = (torch.full((tokens, heads * dim), NAN, device=DEV) for _ in range(2))
    ops().attention_generic(q, keys, values, table, i32(pos), i32(slots), general, **common)
    cut = [(b, q0) for b, n in enumerate(lengths) for q0 in range(0, n, 128)]
    ops().attention_f32_tiles(q, keys, values, table, i32([t[0] for t in cut]), i32([t[1] for t in cut]), i32(range(2)), i32(starts), i32(lengths),
                              i32(np.concatenate([[0], np.cumsum(lengths)])), tiles, **common)
    limit = 2 * relative(general, exact)
    assert relative(tiles, exact) < limit
    if ops().attention_f32_token_takes(dim, dim):
        last = [lengths[0] - 1, tokens - 1]
        token, part_o, part_ml = (torch.full(shape, NAN, device=DEV) for shape in ((2, heads * dim), (2, heads, 2, dim), (2, heads, 2, 2)))
        ops().attention_f32_token(q[last], keys, values, table, i32(pos[last]), i32(range(2)), part_o, part_ml, token, max_chunks=2, **common)
        assert relative(token, exact[last]) < limit


TC_SHAPES = [(8, 8, 64, 64, 1), (12, 2, 128, 128, 1), (8, 4, 64, 128, 2), (3, 1, 128, 128, 1)]


def attention_on_tcgen05(q, keys, values, table, starts, lengths, out, **common):
    """Prompts by the tcgen05 kernel, its scratch full of NaNs before."""
    kv_heads, maps, dim, vdim = common["num_kv_heads"], common.get("maps", 1), common["head_dim"], common.get("v_dim") or common["head_dim"]
    assert ops().attention_f32_tc_takes(dim, vdim, common["scale"])
    pages = StepContext(Workspace(DEV), torch.float32, range(len(starts)), starts, lengths).visible_pages(
        common.get("window"), common.get("chunk"), common.get("keep_first", 0))
    scratch = torch.full((ops().attention_f32_tc_scratch(pages, kv_heads, dim, vdim, maps) + 64,), NAN, device=DEV)
    tiles = [(b, q0) for b, n in enumerate(lengths) for q0 in range(0, n, 128)]
    ops().attention_f32_tc(q, keys, values, table, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), i32(range(len(lengths))), i32(starts),
                           i32(lengths), i32(np.concatenate([[0], np.cumsum(lengths)])), scratch[:-64], pages, out, **common)
    ops().tc_status_check(out.device)
    assert scratch[-64:].isnan().all() and not scratch[:-64].isnan().all()


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps", TC_SHAPES)
@pytest.mark.parametrize("starts,lengths", [([0, 3, 0, 130, 64], [1, 64, 65, 200, 127]), ([0, 700, 64], [620, 150, 1]), ([0] * 70, [1, 2, 64, 65, 129] * 14)])
def test_prompts_on_tcgen05_equal_the_general_kernel(heads, kv_heads, dim, vdim, maps, form, starts, lengths):
    """One page to a dozen, tiles of 1 to 128 queries, more sequences than a warp has lanes; the bounds of the tiles on mma.sync."""
    keys, values, table, gen = paged(starts, lengths, kv_heads, kv_heads // maps, dim, vdim, 3)
    tokens = sum(lengths)
    q = torch.randn(tokens, heads * dim, device=DEV, generator=gen)
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, v_dim=vdim, scale=dim ** -0.5, maps=maps,
                  **options(form, heads, tokens, gen))
    pos = np.concatenate([s + np.arange(n) for s, n in zip(starts, lengths)])
    want, got = (torch.full((tokens, heads * vdim), NAN, device=DEV) for _ in range(2))
    ops().attention_generic(q, keys, values, table, i32(pos), i32(np.repeat(np.arange(len(starts)), lengths)), want, **common)
    attention_on_tcgen05(q, keys, values, table, starts, lengths, got, **common)
    check(got, want, 850)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps", TC_SHAPES[:3])
def test_infinities_and_nans_on_tcgen05_reach_the_queries_that_see_them(heads, kv_heads, dim, vdim, maps, form):
    """As for the tiles on mma.sync; and queries and keys too large for parts, and pages far apart in size."""
    starts, lengths = [0, 3, 0, 130, 64], [1, 64, 65, 200, 127]
    keys, values, table, gen = paged(starts, lengths, kv_heads, kv_heads // maps, dim, vdim, 9)
    tokens, ends = sum(lengths), [s + n for s, n in zip(starts, lengths)]
    values[int(table[3, 0])] *= 1e-30
    values[int(table[3, 1])] *= 1e25
    keys[int(table[2, 0])] *= 1e-25
    for row, n in enumerate(ends):
        for at in range(n, (n + 63) // 64 * 64):
            plant(keys, values, table, row, at, NAN, NAN if at % 2 else INF)
    plant(keys, values, table, 1, 40, value=INF)
    plant(keys, values, table, 2, 63, value=NAN)
    plant(keys, values, table, 2, 64, value=-3.4028234e38)
    plant(keys, values, table, 3, 100, key=INF, value=-INF)
    plant(keys, values, table, 3, 300, key=NAN)
    plant(keys, values, table, 4, 100, key=3.4028234e38)
    q = torch.randn(tokens, heads * dim, device=DEV, generator=gen)
    q[tokens - 10, 2], q[tokens - 5, 1], q[tokens - 20] = INF, NAN, q[tokens - 20] * 1e-30
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, v_dim=vdim, scale=dim ** -0.5, maps=maps,
                  **options(form, heads, tokens, gen))
    pos = np.concatenate([s + np.arange(n) for s, n in zip(starts, lengths)])
    want, got = (torch.full((tokens, heads * vdim), NAN, device=DEV) for _ in range(2))
    ops().attention_generic(q, keys, values, table, i32(pos), i32(np.repeat(np.arange(5), lengths)), want, **common)
    attention_on_tcgen05(q, keys, values, table, starts, lengths, got, **common)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    for row in range(5):                                  # a sequence at a time: their values are of very different sizes
        mine = slice(sum(lengths[:row]), sum(lengths[:row + 1]))
        fine = want[mine].isfinite()
        if fine.any():
            check(got[mine][fine], want[mine][fine], 330)


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 8, 64), (12, 2, 128)])
@pytest.mark.parametrize("spread", [1.0, 6.0])
def test_attention_on_tcgen05_is_as_near_to_64_bits_as_the_general_kernel(heads, kv_heads, dim, spread):
    """Against a softmax in 64 bits, with scores of a few units and of dozens: no further off than the tiles on mma.sync, or than the general
    kernel by a fifth."""
    starts, lengths = [0, 130, 1500], [300, 129, 100]
    keys, values, table, gen = paged(starts, lengths, kv_heads, kv_heads, dim, dim, 11)
    tokens = sum(lengths)
    q = torch.randn(tokens, heads * dim, device=DEV, generator=gen) * spread
    pos = np.concatenate([s + np.arange(n) for s, n in zip(starts, lengths)])
    slots, common = np.repeat(np.arange(3), lengths), dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, scale=dim ** -0.5, window=None)
    exact = torch.empty(tokens, heads, dim, dtype=torch.float64, device=DEV)
    for row in range(3):
        held, mine = starts[row] + lengths[row], slice(*(int(c) for c in np.searchsorted(slots, [row, row + 1])))
        pages = table[row, :(held + 63) // 64].long()
        k = keys[pages].double().permute(1, 0, 2, 3).reshape(kv_heads, -1, dim)[:, :held].repeat_interleave(heads // kv_heads, 0)
        v = values[pages].double().permute(1, 0, 3, 2).reshape(kv_heads, -1, dim)[:, :held].repeat_interleave(heads // kv_heads, 0)
        scores = q[mine].double().view(-1, heads, dim).transpose(0, 1) @ k.transpose(1, 2) * dim ** -0.5
        hidden = torch.arange(held, device=DEV)[None] > torch.as_tensor(pos[mine], device=DEV)[:, None]
        exact[mine] = (scores.masked_fill(hidden, -INF).softmax(-1) @ v).transpose(0, 1)
    exact = exact.view(tokens, heads * dim)
    general, tiles, got = (torch.full((tokens, heads * dim), NAN, device=DEV) for _ in range(3))
    ops().attention_generic(q, keys, values, table, i32(pos), i32(slots), general, **common)
    cut = [(b, q0) for b, n in enumerate(lengths) for q0 in range(0, n, 128)]
    ops().attention_f32_tiles(q, keys, values, table, i32([t[0] for t in cut]), i32([t[1] for t in cut]), i32(range(3)), i32(starts), i32(lengths),
                              i32(np.concatenate([[0], np.cumsum(lengths)])), tiles, **common)
    attention_on_tcgen05(q, keys, values, table, starts, lengths, got, **common)
    errors = [relative(t, exact) for t in (general, tiles, got)]
    print("errors: general %.2e, tiles on mma.sync %.2e, tcgen05 %.2e" % tuple(errors))
    assert errors[2] < max(errors[1], 1.2 * errors[0])


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps", TC_SHAPES[:3])
@pytest.mark.parametrize("number", [1e8, 1e12, 1e15, 1e20])
def test_large_finite_numbers_on_tcgen05_cost_no_other_token_its_digits(heads, kv_heads, dim, vdim, maps, form, number):
    """One large entry of a value or a key in the middle of a page, in a page of the first tokens, and in one that the windows leave out; an
    entry of the queries that meets only zeros; a large value seen with a weight of e^-40.  Every query's head by itself: its
    distance from the general kernel's, in units of the sum of its weights times its values' sizes, has the bounds of `check`."""
    starts, lengths = [0, 30, 0, 100, 0, 0], [100, 90, 200, 90, 70, 90]
    keys, values, table, gen = paged(starts, lengths, kv_heads, kv_heads // maps, dim, vdim, 13)
    tokens, cu = sum(lengths), [0, *(int(c) for c in np.cumsum(lengths))]
    q = torch.randn(tokens, heads * dim, device=DEV, generator=gen)
    plant(keys, values, table, 0, 40, value=number)
    plant(keys, values, table, 1, 40, key=number)
    plant(keys, values, table, 2, 2, value=number)
    plant(keys, values, table, 2, 150, key=-number, value=-number)
    plant(keys, values, table, 3, 60, value=number)
    plant(keys, values, table, 3, 61, key=number)
    for page in table[4, :2].tolist():
        keys[page, :, :, 0] = 0.0
    q.view(tokens, heads, dim)[cu[4]:cu[5], :, 0] = number
    one = torch.randn(dim, device=DEV, generator=gen)
    q.view(tokens, heads, dim)[cu[5]:] = one + 0.01 * torch.randn(90, heads, dim, device=DEV, generator=gen)
    keys[int(table[5, 0]), :, 20] = one * (-40.0 * dim ** 0.5 / (one * one).sum())
    plant(keys, values, table, 5, 20, value=1e17)
    common = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, v_dim=vdim, scale=dim ** -0.5, maps=maps,
                  **options(form, heads, tokens, gen))
    pos = i32(np.concatenate([s + np.arange(n) for s, n in zip(starts, lengths)]))
    slots = i32(np.repeat(np.arange(6), lengths))
    want, size, got = (torch.full((tokens, heads * vdim), NAN, device=DEV) for _ in range(3))
    ops().attention_generic(q, keys, values, table, pos, slots, want, **common)
    ops().attention_generic(q, keys, values.abs(), table, pos, slots, size, **common)
    attention_on_tcgen05(q, keys, values, table, starts, lengths, got, **common)
    assert got.isfinite().all()
    error = (got - want).abs().view(tokens, heads, vdim).amax(2) / size.view(tokens, heads, vdim).amax(2)
    print("largest error of each sequence:", [error[a:b].max().item() for a, b in zip(cu, cu[1:])])
    assert error.max() < (128 + 200 / 8) * 2.0 ** -24
