"""GPU parity of dense fp16 attention (prefill) against the float64 oracle, through the named dispatch."""

import numpy as np
import pytest

from conftest import assert_close_f16
from test_gpu_w4a16 import _ctx, _tensor

pytestmark = pytest.mark.gpu


def _attention(runtime, q, k, v, *, causal, scale, mask=None, token_first_output=False, mask_kind=None):
    from llmopt_b200 import dispatch

    b, h, ql, d = q.shape
    shape = (b, ql, h, d) if token_first_output else (b, h, ql, d)
    out = _tensor(runtime, np.full(shape, np.nan, np.float16))
    mask_tensor = None
    if mask is not None:
        mask_tensor = _tensor(runtime, mask, "bool" if mask_kind == "bool" else None)
    dispatch.dispatch_attention(_ctx(runtime), causal=causal, scale=scale, query=_tensor(runtime, q),
                                key=_tensor(runtime, k), value=_tensor(runtime, v), output=out, mask=mask_tensor)
    return out.buffer.to_numpy(np.float16, shape)


@pytest.mark.parametrize("b,h,kvh,ql,kl,d,causal,tfo,tfv", [
    (1, 3, 3, 8, 8, 64, True, True, False),        # the reference smoke's shape class (head-major in, token-first out)
    (2, 9, 3, 70, 70, 64, True, True, False),      # SmolLM2 head geometry, ragged query tile
    (1, 16, 8, 130, 130, 64, True, False, False),  # LFM attention geometry
    (1, 8, 2, 33, 97, 128, True, True, True),      # cached prefix (past = 64), token-first value
    (2, 4, 4, 40, 56, 128, False, False, False),   # no causal mask
    (1, 2, 1, 5, 5, 80, True, True, False),        # head size without a tensor-core specialisation
    (1, 2, 2, 3, 9, 40, False, False, True),
])
def test_dense_attention_matches_oracle(runtime, oracle, b, h, kvh, ql, kl, d, causal, tfo, tfv):
    rng = np.random.default_rng(20)
    q = rng.standard_normal((b, h, ql, d)).astype(np.float16)
    k = rng.standard_normal((b, kvh, kl, d)).astype(np.float16)
    v = rng.standard_normal((b, kl, kvh, d) if tfv else (b, kvh, kl, d)).astype(np.float16)
    scale = float(np.float32(1.0 / np.sqrt(d)))
    got = _attention(runtime, q, k, v, causal=causal, scale=scale, token_first_output=tfo)
    want = oracle.attention_dense(q, k, v, None, causal=int(causal), scale=scale, kv_heads=kvh,
                                  token_first_output=int(tfo), past_length=max(0, kl - ql), token_first_value=int(tfv))
    assert_close_f16(got, want, label=f"dense attention d={d} q={ql} k={kl}")


@pytest.mark.parametrize("b,h,kvh,ql,kl,d,causal,tfo,tfv,growth", [
    (1, 3, 1, 128, 128, 64, True, True, False, 0.0),    # one whole tile
    (1, 2, 2, 127, 129, 128, True, False, True, 0.0),   # one row less, one key more
    (1, 4, 2, 385, 385, 64, True, True, False, 0.02),   # maxima that grow, many times
    (2, 2, 1, 1, 300, 128, True, True, True, 0.05),     # a single query
    (1, 2, 1, 260, 130, 64, False, True, False, 0.3),   # fewer keys than queries
    (1, 1, 1, 200, 90, 128, True, True, False, 0.0),    # causal, keys that end before the queries
    (2, 48, 16, 520, 520, 64, True, True, False, 0.02),  # more tiles than SMs: two thread blocks share one
    (3, 40, 8, 390, 517, 128, True, True, True, 0.02),
])
def test_dense_attention_tiles_of_128(runtime, oracle, b, h, kvh, ql, kl, d, causal, tfo, tfv, growth):
    rng = np.random.default_rng(22)
    q = rng.standard_normal((b, h, ql, d)).astype(np.float16)
    places = 1.0 + growth * np.arange(kl)
    k = (rng.standard_normal((b, kvh, kl, d)) * np.minimum(places, 12.0)[:, None]).astype(np.float16)
    v = rng.standard_normal((b, kl, kvh, d) if tfv else (b, kvh, kl, d)).astype(np.float16)
    scale = float(np.float32(1.0 / np.sqrt(d)))
    got = _attention(runtime, q, k, v, causal=causal, scale=scale, token_first_output=tfo)
    want = oracle.attention_dense(q, k, v, None, causal=int(causal), scale=scale, kv_heads=kvh,
                                  token_first_output=int(tfo), past_length=max(0, kl - ql), token_first_value=int(tfv))
    assert_close_f16(got, want, label=f"dense attention d={d} q={ql} k={kl}")


@pytest.mark.parametrize("tokens,d,sharp", [(60, 64, 1.0), (333, 64, 3.0), (1000, 128, 3.0), (1000, 64, 1.0)])
def test_dense_attention_is_as_exact_on_both_kinds_of_tensor_cores(runtime, tokens, d, sharp):
    """The error against 64 bits without a mask (tensor memory) and with one that hides nothing (mma.sync): weights are rounded to half
    next to the running maximum in both, so the errors are alike.  Their mean over a hundred thousand results and more scatters by
    far less than the 1 % that the test puts up with."""
    rng = np.random.default_rng(26)
    q = (rng.standard_normal((1, 4, tokens, d)) * sharp).astype(np.float16)
    k, v = (rng.standard_normal((1, 4, tokens, d)).astype(np.float16) for _ in range(2))
    want = np.empty(q.shape)
    for head in range(4):
        score = (q[0, head].astype(np.float64) @ k[0, head].astype(np.float64).T) * d ** -0.5
        score[np.triu_indices(tokens, 1)] = -np.inf
        weight = np.exp(score - score.max(-1, keepdims=True))
        want[0, head] = weight / weight.sum(-1, keepdims=True) @ v[0, head].astype(np.float64)
    everything = np.ones((1, 1, tokens, tokens), np.uint8)
    error = [np.linalg.norm(_attention(runtime, q, k, v, causal=True, scale=d ** -0.5, mask=mask, mask_kind="bool") - want)
             for mask in (None, everything)]
    assert error[0] <= 1.01 * error[1]


@pytest.mark.parametrize("ql,kl,d,causal,growth", [(520, 520, 64, True, 0.02), (520, 600, 128, True, 0.3), (500, 333, 128, False, 0.02)])
def test_heads_alone_and_among_many(runtime, ql, kl, d, causal, growth):
    """Few heads have an SM for each tile of queries, two threads a row and two tiles of scores, many share: the same bits."""
    rng = np.random.default_rng(24)
    q = rng.standard_normal((1, 4, ql, d)).astype(np.float16)
    k = (rng.standard_normal((1, 2, kl, d)) * np.minimum(1.0 + growth * np.arange(kl), 12.0)[:, None]).astype(np.float16)
    v = rng.standard_normal((1, 2, kl, d)).astype(np.float16)
    few = _attention(runtime, q, k, v, causal=causal, scale=d ** -0.5)
    many = _attention(runtime, *(np.tile(x, (1, 30, 1, 1)) for x in (q, k, v)), causal=causal, scale=d ** -0.5)
    assert np.isfinite(few).all()
    for copy in range(30):
        assert np.array_equal(many[0, 4 * copy:4 * copy + 4].view(np.uint16), few[0].view(np.uint16))


@pytest.mark.parametrize("b,h,kvh,ql,kl,past,d,causal,tfo,tfv", [
    (1, 3, 1, 128, 128, 0, 64, 1, 1, 0),
    (1, 2, 2, 300, 363, 63, 128, 1, 1, 1),
    (2, 2, 1, 131, 400, 40, 64, 1, 0, 1),      # keys that no query sees yet: room of a cache
    (1, 1, 1, 1, 260, 100, 128, 1, 1, 0),
    (1, 2, 1, 70, 90, 0, 64, 0, 1, 0),         # every key is seen
    (1, 130, 26, 300, 330, 30, 128, 1, 0, 0),  # two thread blocks share an SM
    (1, 130, 26, 300, 400, 30, 64, 1, 1, 1),
])
def test_values_of_masked_keys_do_not_show(runtime, b, h, kvh, ql, kl, past, d, causal, tfo, tfv):
    """Infinities and NaN behind keys that a query does not see leave its results as they are, to the last bit, but for the queries of the
    same 64; results that do see them are no numbers in the same places; keys behind the last query's need not be initialised."""
    from llmopt_b200 import parameters

    rng = np.random.default_rng(23)
    q, k = rng.standard_normal((b, h, ql, d)).astype(np.float16), rng.standard_normal((b, kvh, kl, d)).astype(np.float16)
    v = rng.standard_normal((b, kl, kvh, d) if tfv else (b, kvh, kl, d)).astype(np.float16)
    poisoned_k, poisoned_v = k.copy(), v.copy()
    by_key = poisoned_v.swapaxes(1, 2) if tfv else poisoned_v  # [b, kvh, kl, d], a view
    by_key[..., kl // 2, 5], by_key[..., kl * 3 // 4, d - 1], by_key[..., kl - 1, :d // 4] = np.inf, np.nan, -np.inf
    if causal and kl > ql + past:
        poisoned_k[..., ql + past:, :], by_key[..., ql + past:, :] = np.nan, np.nan

    def run(keys, values):
        out = _tensor(runtime, np.full((b, h, ql, d), np.nan, np.float16))
        query = _tensor(runtime, q)
        runtime.dispatch(f"llmopt_attention_f16_simd_h{d}",
                         buffers=[query.buffer, _tensor(runtime, keys).buffer, _tensor(runtime, values).buffer, query.buffer, out.buffer],
                         parameters=parameters.attention(batches=b, heads=h, query_length=ql, key_length=kl, head_dimension=d,
                                                         mask_batches=0, mask_heads=0, causal=bool(causal), scale=d ** -0.5, kv_heads=kvh,
                                                         token_first_output=tfo, past_length=past, token_first_value=tfv, mask_dtype=0))
        got = out.buffer.to_numpy(np.float16, (b, ql, h, d) if tfo else (b, h, ql, d))
        return got.swapaxes(1, 2) if tfo else got

    clean, got = run(k, v), run(poisoned_k, poisoned_v)
    seen = np.minimum(np.arange(ql) + past + 1, kl) if causal else np.full(ql, kl)
    strange, near = np.zeros((b, kvh, ql, d), bool), np.zeros((b, kvh, ql, d), bool)  # dimensions of queries that see such a value
    for key, dimension in np.argwhere(~np.isfinite(by_key).all((0, 1))):
        strange[:, :, seen > key, dimension] = True
        near[:, :, np.arange(ql) // 64 == (key - past) // 64, dimension] = bool(causal)
    strange, near = np.repeat(strange, h // kvh, axis=1), np.repeat(near, h // kvh, axis=1)
    assert np.isfinite(clean).all() and not np.isfinite(got[strange]).any()
    assert np.array_equal(got[~strange & ~near].view(np.uint16), clean[~strange & ~near].view(np.uint16))


@pytest.mark.parametrize("why", ["mask", "scale", "address"])
@pytest.mark.parametrize("b,h,kvh,ql,kl,d,causal,tfo,tfv", [
    (1, 3, 1, 64, 64, 64, True, True, False),      # one whole tile
    (2, 4, 2, 65, 129, 128, True, False, True),    # one row more, cached keys, values token first
    (1, 8, 2, 333, 400, 64, True, True, True),     # several tiles of queries, by head
    (1, 6, 3, 260, 130, 128, True, True, False),   # keys that end before the queries
    (1, 2, 1, 200, 90, 64, False, False, False),
    (3, 40, 8, 250, 250, 128, True, True, True),   # more thread blocks than start at once: over all heads
    (2, 60, 20, 389, 420, 64, True, False, False),
])
def test_dense_attention_beside_the_tensor_memory_form(runtime, oracle, b, h, kvh, ql, kl, d, causal, tfo, tfv, why):
    """What a mask, a negative scale or an output that is aligned to four bytes only takes to the mma.sync kernel."""
    from llmopt_b200 import dispatch
    from llmopt_b200.cuda_native import Buffer

    rng = np.random.default_rng(25)
    q = rng.standard_normal((b, h, ql, d)).astype(np.float16)
    k = rng.standard_normal((b, kvh, kl, d)).astype(np.float16)
    v = rng.standard_normal((b, kl, kvh, d) if tfv else (b, kvh, kl, d)).astype(np.float16)
    scale = float(np.float32((-1.0 if why == "scale" else 1.0) / np.sqrt(d)))
    mask = (rng.random((1, 1, ql, kl)) > 0.2).astype(np.uint8) if why == "mask" else None
    shape, shift = (b, ql, h, d) if tfo else (b, h, ql, d), 4 if why == "address" else 0
    room = Buffer.of_array(runtime, np.full(2 * q.size + 16, 0xff, np.uint8))
    out = room.view(shift, 2 * q.size)
    dispatch.dispatch_attention(_ctx(runtime), causal=causal, scale=scale, query=_tensor(runtime, q), key=_tensor(runtime, k),
                                value=_tensor(runtime, v), output=dispatch.Tensor(out, shape, "float16"),
                                mask=None if mask is None else _tensor(runtime, mask, "bool"))
    want = oracle.attention_dense(q, k, v, mask, causal=int(causal), scale=scale, kv_heads=kvh, token_first_output=int(tfo),
                                  past_length=max(0, kl - ql), token_first_value=int(tfv), mask_dtype=1,
                                  mask_batches=0 if mask is None else 1, mask_heads=1)
    assert_close_f16(out.to_numpy(np.float16, shape), want, label=f"{why} d={d} q={ql} k={kl}")
    rest = room.to_numpy(np.uint8)
    assert (rest[:shift] == 0xff).all() and (rest[shift + 2 * q.size:] == 0xff).all()


@pytest.mark.parametrize("kind", ["bool", "float16"])
def test_dense_attention_masks(runtime, oracle, kind):
    rng = np.random.default_rng(21)
    b, h, ql, kl, d = 2, 4, 37, 37, 64
    q = rng.standard_normal((b, h, ql, d)).astype(np.float16)
    k = rng.standard_normal((b, h, kl, d)).astype(np.float16)
    v = rng.standard_normal((b, h, kl, d)).astype(np.float16)
    keep = rng.random((b, 1, ql, kl)) > 0.3
    keep[0, 0, 5, :] = False  # a query that sees nothing writes zeros
    if kind == "bool":
        mask, dtype = keep.astype(np.uint8), 1
    else:
        mask, dtype = np.where(keep, 0.0, -np.inf).astype(np.float16), 2
    scale = 0.125
    got = _attention(runtime, q, k, v, causal=False, scale=scale, mask=mask, mask_kind=kind)
    want = oracle.attention_dense(q, k, v, mask, causal=0, scale=scale, kv_heads=h, mask_dtype=dtype, mask_batches=b,
                                  mask_heads=1)
    assert np.all(got[0, :, 5, :] == 0)
    assert_close_f16(got, want, label=f"dense attention mask {kind}")
