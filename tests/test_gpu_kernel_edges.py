"""Kernels and rules of a dispatch at the sizes where they can go wrong: edges of tiles and strips, remainders, the smallest
and largest of a range."""

import numpy as np
import pytest

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
