"""AttentionStackRunner: two GPT-OSS-shaped layers (one with a 128-token window, one full), hidden
states through prefill in chunks, single-token forwards and a speculative verify + rewind, against
the attention blocks composed from the oracle's operators (ReferenceLayer.decode's order,
Sources/HydraReference/ReferenceLayer.swift:126-187).  The runner's invariant is the path's: the same
positions give the same bits whether they arrive in a prefill chunk, a verify pass or one by one."""
import numpy as np
import pytest

from oracle import hydra_oracle as ho
from tests import hydra_testlib as tl

pytestmark = pytest.mark.gpu


def oracle_stack(hidden, layers, qh, kvh, d, eps):
    """All positions at once: layer by layer, rounding to bf16 where the device's buffers are bf16."""
    total = hidden.shape[0]
    state = hidden.astype(np.float64)
    for w in layers:
        normed = ho.bf16_round(np.stack([ho.rms_norm(row, w.input_norm, eps, use_sqrt=True) for row in state]))
        q = ho.bf16_round(ho.linear(normed, w.wq, w.bq)).reshape(total, qh, d)
        k = ho.bf16_round(ho.linear(normed, w.wk, w.bk)).reshape(total, kvh, d)
        v = ho.bf16_round(ho.linear(normed, w.wv, w.bv)).reshape(total, kvh, d)
        attended = tl.oracle_path(q, k, v, np.arange(total), 1 / np.sqrt(d), window=w.window, sinks=w.sinks,
                                  inv_freq=np.asarray(w.inv_freq))
        attended = ho.bf16_round(attended).reshape(total, qh * d)
        # the device keeps the residual stream in fp32
        state = (state + ho.linear(attended, w.wo, w.bo)).astype(np.float32).astype(np.float64)
    return state


def test_runner_prefill_forward_verify_and_rewind():
    import hydra_b200 as hb
    from hydra_b200.runner import AttentionLayerWeights, AttentionStackRunner
    ctx = hb.Context(0)
    rng = np.random.default_rng(77)
    hidden_size, qh, kvh, d = 2880, 64, 8, 64
    inv = ho.inverse_frequencies(d, 150000.0)
    eps = 1e-5

    def layer(window):
        return AttentionLayerWeights(
            input_norm=ho.bf16_round(1.0 + 0.1 * rng.standard_normal(hidden_size)),
            wq=ho.bf16_round(rng.normal(0, 0.02, (qh * d, hidden_size))), bq=ho.bf16_round(rng.normal(0, 0.1, qh * d)),
            wk=ho.bf16_round(rng.normal(0, 0.02, (kvh * d, hidden_size))), bk=ho.bf16_round(rng.normal(0, 0.1, kvh * d)),
            wv=ho.bf16_round(rng.normal(0, 0.02, (kvh * d, hidden_size))), bv=ho.bf16_round(rng.normal(0, 0.1, kvh * d)),
            wo=ho.bf16_round(rng.normal(0, 0.02, (hidden_size, qh * d))), bo=ho.bf16_round(rng.normal(0, 0.1, hidden_size)),
            sinks=tl.normal_bf16(rng, (qh,)), window=window, inv_freq=inv)

    layers = [layer(128), layer(0)]
    prompt, single, draft = 300, 2, 5
    total = prompt + single + draft
    states = rng.standard_normal((total, hidden_size)).astype(np.float32)
    want = oracle_stack(states, layers, qh, kvh, d, eps)

    runner = AttentionStackRunner(ctx, layers, hidden_size, qh, kvh, d, context_length=1024, eps=eps,
                                  prefill_chunk_tokens=128)
    last = runner.prefill(states[:prompt])
    assert runner.position == prompt
    assert tl.within_tolerance(last, want[prompt - 1], bf16_output=False)
    got_single = np.stack([runner.forward(states[prompt + i]) for i in range(single)])
    assert tl.within_tolerance(got_single, want[prompt:prompt + single], bf16_output=False)
    # a draft of five tokens verified in one pass, three accepted: rewind, then the same three one by one
    base = runner.position
    verified = runner.verify(states[base:base + draft])
    assert tl.within_tolerance(verified, want[base:base + draft], bf16_output=False)
    assert runner.can_rewind(base + 3)
    runner.rewind(base + 3)
    assert runner.position == base + 3
    runner.rewind(base)
    again = np.stack([runner.forward(states[base + i]) for i in range(3)])
    assert np.array_equal(again, verified[:3])                     # verify pass == token by token, bit for bit
    tl.record_margin("two-layer attention stack: prefill 300, forward 2, verify 5", np.concatenate([got_single, verified]),
                     want[prompt:])
    runner.close()
    ctx.close()


@pytest.mark.parametrize("tokens, width", [(1, 2880), (5, 2880), (6, 2880), (40, 2880), (256, 64), (257, 64)])
def test_hidden_states_in_pinned_and_in_pageable_memory(tokens, width):
    """Up to 64 KB of pinned hidden states (five of 2880; 256 of 64 to the byte) are read and written where they are, by a
    launch each; the rest, pageable memory and buffers off a 16-byte boundary are copied."""
    import ctypes
    import torch
    import hydra_b200 as hb
    capi, qh, kvh, d = hb.capi, 8, 2, 64
    ctx = hb.Context(0)
    lib = capi.load()
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    shapes = dict(input_norm=(width,), wq=(qh * d, width), wk=(kvh * d, width), wv=(kvh * d, width), wo=(width, qh * d))
    weights = {name: (0.02 * torch.randn(shape, device="cuda", generator=gen)).to(torch.bfloat16) for name, shape in shapes.items()}
    block = (capi.BlockWeightsStruct * 1)()
    for name, tensor in weights.items():
        setattr(block[0], name, tensor.data_ptr())
    block[0].params = hb.AttnParams(q_heads=qh, kv_heads=kvh, head_dim=d, sm_scale=0.125, io_dtype=capi.HC_BF16).struct()
    workspace = torch.empty(lib.hc_attention_stack_bytes(block, 1, tokens, width), dtype=torch.uint8, device="cuda")
    states = torch.from_numpy(np.random.default_rng(tokens).standard_normal((tokens, width)).astype(np.float32))
    count, got, launches = tokens * width, [], []
    for pinned, offset in ((False, 0), (True, 0), (True, 1)):
        cache = hb.KVCache(ctx, [dict(q_heads=qh, kv_heads=kvh, head_dim=d, window=0)], 512, prefill_chunk=512)
        source, result = (torch.empty(count + offset, pin_memory=pinned)[offset:] for _ in range(2))
        source.copy_(states.reshape(-1))
        before = ctx.launch_count
        assert lib.hc_attention_stack_host(ctx.handle, cache.handle, block, 1, 0, source.data_ptr(), result.data_ptr(), tokens, width, 0,
                                           ctypes.c_float(1e-5), workspace.data_ptr(), None) == capi.HC_OK
        launches.append(ctx.launch_count - before)
        got.append(result.numpy().copy())
        cache.close()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    assert launches[1] - launches[0] == (2 if 4 * count <= 65536 else 0) and launches[2] == launches[0]
    ctx.close()
