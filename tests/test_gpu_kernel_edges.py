"""Kernels and rules of a dispatch at the sizes where they can go wrong: edges of tiles and strips, remainders, the smallest
and largest of a range."""

import numpy as np
import pytest

import oracle_mixers as plain
from mixer_models import bf16_round
from test_gpu_mixers import close, download, empty, upload

pytestmark = pytest.mark.gpu


def _half(runtime, array):
    from llmopt_b200.cuda_native import Buffer

    return Buffer.of_array(runtime, np.ascontiguousarray(array, np.float16))


@pytest.mark.parametrize("tokens", [1, 2, 3, 7, 8, 9, 16, 17, 65])
@pytest.mark.parametrize("start", ["none", "apart", "in place"])
def test_short_conv_prompt_in_strips(runtime, oracle, tokens, start):
    """Every strip starts from the inputs ahead of it; a state updated in place is read before it is written.  The states are
    copies of halves or one rounding of a product: equal bits; an output rounds an fp32 sum once (oracle: double), so it may
    be one unit in the last place off."""
    from llmopt_b200 import dispatch
    from llmopt_b200.cuda_native import Buffer

    rng = np.random.default_rng(tokens)
    channels = 300
    rows = rng.standard_normal((tokens, 3 * channels)).astype(np.float16)
    weight = rng.standard_normal((channels, 1, 3)).astype(np.float16)
    initial = rng.standard_normal((channels, 3)).astype(np.float16)
    out = Buffer.create(runtime, tokens * channels * 2)
    before = _half(runtime, initial)
    after = before if start == "in place" else _half(runtime, np.full((channels, 3), np.nan))
    tensor = lambda buffer, shape: dispatch.Tensor(buffer, shape)
    dispatch.dispatch_short_conv_prefill(
        dispatch.Context(runtime), in_proj=tensor(_half(runtime, rows), (1, tokens, 3 * channels)),
        conv_weight=tensor(_half(runtime, weight), weight.shape), output=tensor(out, (1, tokens, channels)),
        conv_state_out=tensor(after, (1, channels, 3)),
        conv_state_in=None if start == "none" else tensor(before, (1, channels, 3)))
    want, state = oracle.short_conv_prefill(rows, weight.reshape(channels, 3), None if start == "none" else initial)
    got = out.to_numpy(np.float16, (tokens, channels))
    assert np.all(np.abs(got.astype(np.float64) - want) <= 2.0 ** -10 * np.abs(want) + 2.0 ** -12)
    assert np.array_equal(after.to_numpy(np.uint16), state.view(np.uint16).reshape(-1))


@pytest.mark.parametrize("tokens,channels", [(1, 64), (9, 300), (200, 1024), (65, 2051)])
@pytest.mark.parametrize("part", [0, 1, 2])
def test_short_conv_prompt_over_its_projections(runtime, tokens, channels, part):
    """Outputs may take the memory of the projected rows, from any of the first row's three parts on: a token's output then
    lies where an input of the same channel was that is read by then.  The same bits as in memory of their own."""
    from llmopt_b200 import parameters
    from llmopt_b200.cuda_native import Buffer

    rng = np.random.default_rng(tokens + part)
    rows = rng.standard_normal((tokens, 3 * channels)).astype(np.float16)
    weight = _half(runtime, rng.standard_normal((channels, 3)))

    def run(over):
        projected, apart = _half(runtime, rows), Buffer.create(runtime, tokens * channels * 2)
        out = projected.view(part * channels * 2, tokens * channels * 2) if over else apart
        state = Buffer.create(runtime, channels * 6)
        runtime.dispatch("llmopt_short_conv_prefill_f16", buffers=[projected, weight, out, state],
                         parameters=parameters.short_conv_prefill(tokens=tokens, channels=channels, has_initial_state=False))
        return out.contents(), state.contents()

    assert run(True) == run(False)


@pytest.mark.parametrize("apart,shared_state", [(0, False), (16, False), (0, True)])
def test_short_conv_steps_of_a_plan_as_one_launch(runtime, oracle, apart, shared_state):
    """Steps of sequences at equal distances run as one launch of a plan and leave the same bytes as one by one; steps on the
    same state follow each other."""
    from llmopt_b200 import parameters
    from llmopt_b200.cuda_native import Buffer, DispatchItem, Prebaked

    rng = np.random.default_rng(apart)
    count, channels = 3, 260
    weight = _half(runtime, rng.standard_normal((channels, 3)))
    step = 6 * channels + apart
    rows = Buffer.of_array(runtime, rng.standard_normal(count * step // 2).astype(np.float16))
    initial = rng.standard_normal(count * step // 2).astype(np.float16)

    def run(plan):
        states, out = Buffer.of_array(runtime, initial), Buffer.create(runtime, count * (2 * channels + apart))
        items = [DispatchItem("llmopt_short_conv_step_f16",
                              [rows.view(i * step, 6 * channels), states.view(0 if shared_state else i * step, 6 * channels), weight,
                               out.view(i * (2 * channels + apart), 2 * channels)], parameters.short_conv_step(channels=channels))
                 for i in range(count)]
        if plan:
            prebaked = Prebaked(runtime, items, None, None)
            assert prebaked.kernel_count() == (1 + count if shared_state else 2)  # the plan's prologue and the steps
            prebaked.execute(token=0, past_tokens=0)
        else:
            for item in items:
                runtime.dispatch(item.name, buffers=item.buffers, parameters=item.parameters)
        return states.contents(), out.contents()

    assert run(True) == run(False)


@pytest.mark.parametrize("m,n,k", [(1, 9, 4), (2, 8, 516), (4, 7, 128), (5, 33, 1028), (8, 16, 260), (9, 65, 36), (32, 64, 32),
                                   (33, 63, 2052), (64, 128, 1024), (65, 130, 96), (100, 256, 2048), (129, 20, 7168)])
def test_dense_fp32(runtime, m, n, k):
    """Streams of a few rows and tiles of every size.  fp32 sums of k products: an error of a few times
    2^-24 sqrt(k) of the terms' size, where the result has sqrt(k) of them; 3e-6 of the largest result."""
    from llmopt_b200 import parameters

    rng = np.random.default_rng(m * 1000 + n)
    x, w = rng.standard_normal((m, k)).astype(np.float32), (rng.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    y = x.astype(np.float64) @ w.T.astype(np.float64) + bias
    split = n // 2
    buffers = [upload(runtime, x), upload(runtime, w), upload(runtime, bias), empty(runtime, m * n), empty(runtime, m * n),
               upload(runtime, np.zeros(m, np.int64)), empty(runtime, 16)]
    runtime.dispatch("llmopt_dense_linear_f32", buffers=buffers, parameters=parameters.dense_linear(
        m=m, n=n, k=k, split=split, has_bias=True, epilogue=None))
    if split:
        close(download(buffers[3], (m, split)), y[:, :split], 3e-6)
    close(download(buffers[4], (m, n - split)), y[:, split:], 3e-6)
    if n % 2 == 0:
        runtime.dispatch("llmopt_dense_linear_f32", buffers=buffers, parameters=parameters.dense_linear(
            m=m, n=n, k=k, split=n, has_bias=True, epilogue="silu_pair"))
        close(download(buffers[3], (m, n // 2)), plain.silu(y[:, 0::2]) * y[:, 1::2], 6e-6)


@pytest.mark.parametrize("m,experts", [(32 * 65535, 0), (32 * 65535 + 1, 0), (64 * 65535, 0), (128 * 16383, 3), (128 * 16384 + 5, 3)])
def test_dense_fp32_of_millions_of_rows(runtime, m, experts):
    """More tiles of 32 rows than a grid holds, up to all that it holds of 64: plain, and rows sorted by expert.  Sums of four
    products of numbers of at most 4 bits: exact."""
    from llmopt_b200 import parameters

    rng = np.random.default_rng(m % 1000)
    n, k = 2, 4
    x = rng.integers(-8, 8, size=(m, k)).astype(np.float32)
    w = rng.integers(-8, 8, size=(max(experts, 1), n, k)).astype(np.float32)
    out = empty(runtime, m * n)
    if experts:
        bounds = [0, 100, m - 3, m]
        tiles = [(e, first, min(first + 128, bounds[e + 1])) for e in range(experts) for first in range(bounds[e], bounds[e + 1], 128)]
        most = m // 128 + experts
        assert len(tiles) <= most
        plan = np.zeros((1 + most, 4), np.uint32)
        plan[0, 0], plan[1:1 + len(tiles), :3] = len(tiles), tiles
        runtime.dispatch("llmopt_expert_rows_f32", buffers=[
            upload(runtime, x), upload(runtime, w), upload(runtime, plan), upload(runtime, np.ones(m, np.float32)), out],
            parameters=parameters.expert_rows(pairs=m, n=n, k=k, experts=experts, paired=False))
        want = np.concatenate([x[a:b] @ w[e].T for e, (a, b) in enumerate(zip(bounds, bounds[1:]))])
    else:
        spare = empty(runtime, 16)
        runtime.dispatch("llmopt_dense_linear_f32", buffers=[upload(runtime, x), upload(runtime, w), spare, out, spare, spare, spare],
                         parameters=parameters.dense_linear(m=m, n=n, k=k, split=n))
        want = x @ w[0].T
    assert np.array_equal(download(out, (m, n)), want)


@pytest.mark.parametrize("m,n,k", [(1, 18, 4), (3, 40, 1028), (8, 33, 516), (13, 65, 2052), (32, 64, 96), (33, 63, 36),
                                   (64, 130, 1024), (100, 2048, 260), (100, 7168, 64), (129, 20, 7168)])
def test_dense_fp32_equals_the_general_kernels(runtime, m, n, k):
    """Rows off 16-byte boundaries take the general kernels; the others add in the same order, to the last bit."""
    from llmopt_b200 import parameters

    rng = np.random.default_rng(m + n)
    x, w, bias = (rng.standard_normal(shape).astype(np.float32) for shape in ((m, k), (n, k), n))
    shifted = upload(runtime, np.concatenate((np.zeros(1, np.float32), x.reshape(-1)))).view(4, 4 * m * k)
    results = []
    for rows in (upload(runtime, x), shifted):
        out = [empty(runtime, m * n), empty(runtime, m * n)]
        runtime.dispatch("llmopt_dense_linear_f32", buffers=[
            rows, upload(runtime, w), upload(runtime, bias), *out, upload(runtime, np.zeros(m, np.int64)), empty(runtime, 16)],
            parameters=parameters.dense_linear(m=m, n=n, k=k, split=n // 3, has_bias=True, epilogue=None))
        results.append([download(one, (m, columns)) for one, columns in zip(out, (n // 3, n - n // 3))])
    for here, general in zip(*results):
        assert np.array_equal(here, general)


@pytest.mark.parametrize("m,k,columns", [(66, 192, (40,)), (257, 1024, (300,)), (300, 4608, (130,)), (700, 512, (1100,)),
                                         (2049, 64, (129,)), (40, 128, (130, 70, 64)), (72, 576, (576, 192, 192)),
                                         (300, 1024, (129, 512, 1)), (513, 320, (200, 60, 1000))])
def test_prompt_tiles_and_fused_projections(runtime, oracle, m, k, columns):
    """Every width of a prompt's tiles, with and without splits of k, with the residual read ahead; three matrices of unequal
    sizes as one launch.  The parity bound of the product, 2e-3 of the outputs' scale."""
    from conftest import assert_close_f16
    from helpers import random_w4
    from llmopt_b200 import dispatch
    from llmopt_b200.cuda_native import Buffer

    rng = np.random.default_rng(m)
    x = rng.standard_normal((m, k)).astype(np.float16)
    matrices = [random_w4(rng, n, k) for n in columns]
    upload_tensor = lambda array, kind="float16": dispatch.Tensor(Buffer.of_array(runtime, array), array.shape, kind)
    weights = [(upload_tensor(packed, "uint8"), upload_tensor(scale)) for packed, scale in matrices]
    outputs = [upload_tensor(np.full((m, n), np.nan, np.float16)) for n in columns]
    context = dispatch.Context(runtime)
    if len(columns) == 1:
        residual = rng.standard_normal((m, columns[0])).astype(np.float16)
        dispatch.dispatch_w4a16_linear(context, input=upload_tensor(x), weight=weights[0][0], scale=weights[0][1],
                                       output=outputs[0], bias=upload_tensor(residual), bias_row_stride=columns[0])
        wanted = [oracle.w4a16_linear(x, *matrices[0], residual, columns[0])]
    else:
        (q, k_, v) = weights
        dispatch.dispatch_w4a16_qkv_linear_command(
            context, input=upload_tensor(x), q_weight=q[0], q_scale=q[1], k_weight=k_[0], k_scale=k_[1], v_weight=v[0], v_scale=v[1],
            q_output=outputs[0], k_output=outputs[1], v_output=outputs[2])
        wanted = [oracle.w4a16_linear(x, *pair) for pair in matrices]
    for output, want in zip(outputs, wanted):
        assert_close_f16(output.buffer.to_numpy(np.float16, want.shape), want)


@pytest.mark.parametrize("rows,k,n", [(1, 64, 1), (1, 576, 200), (8, 576, 33), (3, 1984, 17), (2, 1088, 16), (5, 448, 50)])
def test_short_sums(runtime, oracle, monkeypatch, rows, k, n):
    """Few rows and a K that is no multiple of 512: a plain product with a residual, three matrices as one launch, and a plan
    that folds the RMS norm ahead of a product, whose rows equal the stand-alone norm's byte for byte."""
    from conftest import assert_close_f16
    from helpers import random_w4
    from llmopt_b200 import dispatch, parameters
    from llmopt_b200.cuda_native import Buffer, DispatchItem, Prebaked

    rng = np.random.default_rng(k + rows)
    x = rng.standard_normal((rows, k)).astype(np.float16)
    residual = rng.standard_normal((rows, n)).astype(np.float16)
    matrices = [random_w4(rng, columns, k) for columns in (n, 5, 40)]
    tensor = lambda array, kind="float16": dispatch.Tensor(Buffer.of_array(runtime, array), array.shape, kind)
    weights = [(tensor(packed, "uint8"), tensor(scale)) for packed, scale in matrices]
    outputs = [tensor(np.full((rows, len(packed)), np.nan, np.float16)) for packed, _ in matrices]
    context = dispatch.Context(runtime)
    in_place = tensor(residual)  # the residual's own buffer takes the sum
    dispatch.dispatch_w4a16_linear(context, input=tensor(x), weight=weights[0][0], scale=weights[0][1], output=in_place,
                                   bias=in_place, bias_row_stride=n)
    assert_close_f16(in_place.buffer.to_numpy(np.float16, (rows, n)), oracle.w4a16_linear(x, *matrices[0], residual, n))
    (q, k_, v) = weights
    dispatch.dispatch_w4a16_qkv_linear_command(
        context, input=tensor(x), q_weight=q[0], q_scale=q[1], k_weight=k_[0], k_scale=k_[1], v_weight=v[0], v_scale=v[1],
        q_output=outputs[0], k_output=outputs[1], v_output=outputs[2])
    for output, pair in zip(outputs, matrices):
        assert_close_f16(output.buffer.to_numpy(np.float16, output.shape), oracle.w4a16_linear(x, *pair))

    weight = rng.uniform(0.5, 1.5, size=k).astype(np.float16)
    results, counts = [], []
    for fold in ("1", "0"):
        monkeypatch.setenv("LLMOPT_CUDA_FOLD_NORMS", fold)
        normed = Buffer.of_array(runtime, np.full((rows, k), np.nan, np.float16))
        out = Buffer.of_array(runtime, np.full((rows, n), np.nan, np.float16))
        scales = weights[0][1].buffer
        plan = Prebaked(runtime, [
            DispatchItem("llmopt_rms_norm_f16_simd", [Buffer.of_array(runtime, x), Buffer.of_array(runtime, weight), normed],
                         parameters.rms_norm(rows=rows, width=k, epsilon=1e-5), (256, 1, 1), (256, 1, 1)),
            DispatchItem("llmopt_w4a16_linear_f16_g64_m4", [normed, weights[0][0].buffer, scales, scales, out],
                         parameters.u32s([rows, n, k, 0, 0]), (256, 1, 1), (256, 1, 1))], None, None)
        plan.execute(token=0, past_tokens=0)
        counts.append(plan.kernel_count())
        results.append((normed.to_numpy(np.float16, (rows, k)), out.to_numpy(np.float16, (rows, n))))
    assert counts[0] == counts[1] - 1
    assert np.array_equal(results[0][0].view(np.uint16), results[1][0].view(np.uint16))
    assert np.array_equal(results[0][1].view(np.uint16), results[1][1].view(np.uint16))
    assert_close_f16(results[0][1], oracle.w4a16_linear(results[0][0], *matrices[0]))


# ---- persistent streams (a tile of 16 columns for every SM and more) --------------------------------------

WIDE = [(1, 2370, 72), (8, 2370, 520), (9, 2370, 72), (16, 2370, 2048), (17, 2370, 520), (32, 2370, 2048),  # one or two tiles per block
        (8, 15010, 72), (16, 15010, 136), (32, 15010, 72)]                                                 # four and more, the ring crosses their ends


@pytest.mark.parametrize("m,n,k", WIDE)
def test_products_of_many_columns(runtime, m, n, k):
    """Plain (also an odd number of columns), pair and residual stores against fp64, with the bounds of the same checks at
    other sizes."""
    import test_gpu_dalorax as sublayers
    import test_gpu_mixers as mixers

    mixers.test_dense_linear(runtime, "bfloat16", m, n - 1, k, n // 3)
    sublayers.test_paired_columns_and_scale(runtime, "bfloat16", m, n, k)
    sublayers.test_product_that_ends_a_sublayer(runtime, "bfloat16", m, n, k)


@pytest.mark.parametrize("m,n,k", WIDE[:6] + [(32, 7300, 136)])
def test_cache_rows_of_many_columns(runtime, m, n, k):
    """Columns that go to the output, to a token's key and value row and to fp32 rows, borders off the tiles."""
    from llmopt_b200 import parameters
    from llmopt_b200.kv_cache import RowLayout

    rng = np.random.default_rng(m + k)
    heads, dim, vdim, extra = 3, 24, 40, 5
    keys, values = heads * dim, heads * vdim
    own = n - keys - values - extra
    x, w = bf16_round(rng.standard_normal((m, k))), bf16_round(rng.standard_normal((n, k)) / np.sqrt(k))
    bias = rng.standard_normal(n).astype(np.float32)
    layout = RowLayout([(1, 8, 16), (heads, dim, vdim)])
    region, stride, slots = layout.regions[1], 7, 7 * m + 3
    table = rng.permutation(slots)[:7 * m].reshape(m, stride).astype(np.uint32)
    past, which = rng.integers(0, stride, size=m).astype(np.uint32), rng.permutation(m).astype(np.uint32)
    before = bf16_round(rng.standard_normal((slots, layout.token_elements)))
    pool, out, out32 = upload(runtime, before, "bfloat16"), empty(runtime, m * own, "bfloat16"), empty(runtime, m * extra)
    runtime.dispatch("llmopt_dense_cached_bf16", buffers=[
        upload(runtime, x, "bfloat16"), upload(runtime, w, "bfloat16"), upload(runtime, bias), out, out32, pool, upload(runtime, table),
        upload(runtime, past), upload(runtime, which)], parameters=parameters.dense_cached(
            m=m, n=n, k=k, split=own, tokens=1, key_columns=keys, value_columns=values, has_bias=True,
            token_stride=layout.token_elements, key_offset=region.key_offset, value_offset=region.value_offset, table_stride=stride,
            table_rows=m, pool_rows=slots))
    y = x.astype(np.float64) @ w.T.astype(np.float64) + bias
    close(download(out, (m, own), "bfloat16"), y[:, :own], 6e-3, "rows")
    close(download(out32, (m, extra)), y[:, n - extra:], 1e-5, "fp32 rows")
    want = before.astype(np.float64)
    slot = table[which, past]
    want[slot, region.key_offset:region.key_offset + keys] = y[:, own:own + keys]
    want[slot, region.value_offset:region.value_offset + values] = y[:, own + keys:own + keys + values]
    got = download(pool, before.shape, "bfloat16")
    close(got, want, 6e-3, "cache")
    untouched = np.setdiff1d(np.arange(slots), slot)
    assert np.array_equal(got[untouched], before[untouched])


@pytest.mark.parametrize("rows,experts,top,n,k", [(1, 8, 4, 1218, 72), (8, 64, 8, 200, 520), (9, 40, 6, 122, 200), (16, 33, 2, 282, 136),
                                                  (17, 300, 3, 98, 72), (32, 60, 3, 90, 1000), (32, 16, 2, 1026, 2048),
                                                  (2, 4, 2, 58, 72), (40, 9, 2, 130, 104)])  # a tile per block
def test_expert_rows_of_many_tiles(runtime, rows, experts, top, n, k):
    """Gate and up rows of all chosen experts as one list of tiles, against fp64; a route of any words reads and writes nothing
    beyond its buffers."""
    from llmopt_b200 import parameters
    from llmopt_b200.cuda_native import Buffer
    from llmopt_b200.feed_forward import route_words

    rng = np.random.default_rng(rows + n)
    x, w = bf16_round(rng.standard_normal((rows, k))), bf16_round(rng.standard_normal((experts, n, k)) / np.sqrt(k))
    logits = (rng.standard_normal((rows, experts)) * 3).astype(np.float32)
    words, pairs = route_words(rows, experts, top), rows * top
    route = upload(runtime, np.zeros(words, np.uint32))
    runtime.dispatch("llmopt_route_step_f32", buffers=[upload(runtime, logits), route], parameters=parameters.route(rows=rows, experts=experts, top=top))
    guard = 64 * n
    out = Buffer.of_array(runtime, np.full(pairs * n // 2 + guard, 0x7FC0, np.uint16))
    operands = [upload(runtime, x, "bfloat16"), upload(runtime, w, "bfloat16")]
    block = parameters.expert_step(rows=rows, n=n, k=k, experts=experts, top=top)
    runtime.dispatch("llmopt_expert_step_bf16", buffers=[*operands, route, out.view(0, pairs * n)], parameters=block)
    choices = np.argsort(-logits, axis=1, kind="stable")[:, :top]
    order = np.argsort(choices.reshape(-1), kind="stable")
    want = np.empty((pairs, n // 2))
    for slot, pair in enumerate(order):
        row, expert = pair // top, choices.reshape(-1)[pair]
        y = w[expert].astype(np.float64) @ x[row] * plain.sigmoid(np.float64(logits[row, expert]))
        want[slot] = plain.silu(y[0::2]) * y[1::2]
    close(download(out, (pairs, n // 2), "bfloat16"), want, 6e-3)
    for seed in range(3):
        noise = np.random.default_rng(seed).integers(0, [2 ** 32, 2 * pairs + 2, pairs + 1][seed], size=words, dtype=np.uint32)
        noise[0] = [2 ** 32 - 1, experts, min(pairs, experts)][seed]
        runtime.dispatch("llmopt_expert_step_bf16", buffers=[*operands, upload(runtime, noise), out.view(0, pairs * n)], parameters=block)
    assert np.all(out.to_numpy(np.uint16)[pairs * n // 2:] == 0x7FC0)


# ---- rules that look at how much there is to do: the same bits alone and among many ----------------------

@pytest.mark.parametrize("dtype,heads,kv_heads,dim,vdim,tokens,many,splits", [
    ("float32", 16, 4, 20, 24, 9, 60, 1), ("float32", 16, 8, 128, 100, 3, 200, 1), ("float32", 8, 1, 256, 512, 2, 2000, 1),
    ("bfloat16", 16, 4, 18, 10, 7, 90, 1),                                                       # a block or a warp per row and head
    ("bfloat16", 16, 4, 128, 128, 1, 8, 13), ("bfloat16", 8, 8, 128, 128, 2, 40, 1), ("bfloat16", 8, 8, 128, 128, 1, 64, 1)])  # rings
def test_row_attention_alone_and_among_many(runtime, dtype, heads, kv_heads, dim, vdim, tokens, many, splits):
    """The first sequence alone and with others that make the dispatch choose another kernel or ring; a window and a cap on the way."""
    from llmopt_b200 import parameters
    from test_gpu_mixers import suffix

    rng = np.random.default_rng(dim + many)
    past = rng.integers(0, 400, size=many).astype(np.uint32)
    past[0] = 301
    stride, token_stride = 400 + tokens, kv_heads * (dim + vdim)
    pool_rows = 3000
    pool = upload(runtime, rng.standard_normal((pool_rows, token_stride)), dtype)
    table = upload(runtime, rng.integers(0, pool_rows, size=(many, stride)).astype(np.uint32))
    query = rng.standard_normal((many * tokens, heads * dim))
    for options in ({}, dict(window=70, keep_first=3, softcap=9.0)):
        results = []
        for sequences in (1, many):
            out = empty(runtime, sequences * tokens * heads * vdim, dtype)
            scratch = upload(runtime, np.zeros(4096 + sequences * kv_heads * splits * (32 + 16 * 256), np.float32))
            q = upload(runtime, query[:sequences * tokens], dtype)
            runtime.dispatch("llmopt_row_attention_" + suffix(dtype), buffers=[
                q, pool, table, upload(runtime, past), upload(runtime, np.arange(many, dtype=np.uint32)), out, scratch, q],
                parameters=parameters.row_attention(
                    sequences=sequences, tokens=tokens, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, token_stride=token_stride,
                    key_offset=0, value_offset=kv_heads * dim, table_stride=stride, table_rows=many, pool_rows=pool_rows, sink=bool(options),
                    splits=splits, scale=dim ** -0.5, **options))
            results.append(download(out, (sequences, tokens, heads, vdim), dtype)[0])
        assert np.all(np.isfinite(results[0])) and np.array_equal(*results)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("dim,vdim", [(40, 40), (128, 70), (160, 96), (256, 33)])
@pytest.mark.parametrize("tokens", [4, 70])
def test_matrix_memory_alone_and_among_many(runtime, dtype, dim, vdim, tokens):
    """One sequence (half slices) and forty alike (whole ones): the same read-outs and states."""
    from llmopt_b200 import parameters
    from llmopt_b200.kv_cache import matrix_state_elements
    from test_gpu_mixers import suffix

    rng = np.random.default_rng(dim + tokens)
    heads, results = 3, []
    width, stride = heads * (2 * dim + vdim), matrix_state_elements(heads, dim, vdim, normalized=True)
    slices = -(-vdim // 32)
    raw, gates = rng.standard_normal((tokens, width)) * 0.5, rng.standard_normal((tokens, 2 * heads)).astype(np.float32)
    state = (rng.standard_normal(stride) * 0.3).astype(np.float32)
    norms = heads * vdim * dim  # the copies of n and m of a head are alike
    state[norms:norms + heads * slices * dim] = np.repeat(rng.standard_normal((heads, 1, dim)), slices, 1).reshape(-1)
    state[norms + heads * slices * dim:][:heads * slices] = np.repeat(rng.standard_normal(heads), slices)
    for sequences in (1, 40):
        pool, out = upload(runtime, np.tile(state, (sequences, 1))), empty(runtime, sequences * tokens * heads * vdim)
        projected, scalars = upload(runtime, np.tile(raw, (sequences, 1)), dtype), upload(runtime, np.tile(gates, (sequences, 1)))
        runtime.dispatch("llmopt_memory_scan_" + suffix(dtype), buffers=[
            projected, projected, projected, scalars, scalars, pool, upload(runtime, np.full(sequences, 5, np.uint32)),
            upload(runtime, np.arange(sequences, dtype=np.uint32)), out], parameters=parameters.state_scan(
                sequences=sequences, tokens=tokens, heads=heads, kv_heads=heads, dim=dim, vdim=vdim, q_stride=width, q_column=0,
                k_stride=width, k_column=heads * dim, v_stride=width, v_column=2 * heads * dim, scalar_stride=2 * heads, first_column=0,
                second_column=heads, state_rows=sequences, state_stride=stride, gate_cap=6.0))
        results.append((download(out, (sequences, tokens, heads, vdim)), download(pool, (sequences, stride))))
    for alone, among in zip(*results):
        assert np.all(np.isfinite(alone)) and all(np.array_equal(alone[0], one) for one in among)


# ---- paged attention in its forms -----------------------------------------------------------------------

@pytest.mark.parametrize("batch,q_heads,k_heads,dim,group,past", [
    (1, 8, 2, 128, 64, 3100), (2, 16, 8, 64, 32, 3200),  # records and a merge
    (2, 16, 8, 128, 32, 900), (3, 8, 8, 64, 64, 1500),   # clusters of 8 blocks of 8 warps
    (5, 16, 8, 128, 64, 200), (8, 16, 8, 64, 64, 530), (5, 8, 8, 64, 32, 2100),  # 8 of 4
    (8, 20, 10, 128, 32, 200), (8, 20, 20, 64, 64, 150)])                        # 4 and 2 of 4
def test_attention_with_rotary_and_pack_in_every_form(runtime, monkeypatch, batch, q_heads, k_heads, dim, group, past):
    import test_gpu_cache_attention as attention

    attention.test_plan_hands_rotary_and_pack_to_the_attention_byte_for_byte(runtime, monkeypatch, batch, q_heads, k_heads, dim, group, past)


@pytest.mark.parametrize("batches,hkv,past", [(3, 8, 600), (3, 8, 1500), (5, 8, 520), (5, 8, 2100), (5, 8, 4500), (10, 8, 2100), (10, 8, 3300),
                                              (13, 8, 2100), (20, 8, 530), (32, 8, 140)])
def test_batches_behind_contexts(runtime, oracle, batches, hkv, past):
    """On both sides of the lines between clusters of 8 x 8, 8 x 4, 4 x 4 and 2 x 4 warps and records."""
    import test_gpu_cache_attention as attention
    from conftest import assert_close_f16

    got, want, names = attention._paged(runtime, oracle, batches=batches, hq=2 * hkv, hkv=hkv, dim=64, group=64, past=past, layers=1, layer=0,
                                        per_sequence=True, query_scale=3.0, seed=past)
    assert_close_f16(got, want, label=f"paged {names}")
