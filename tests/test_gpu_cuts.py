"""Every way the kernels cut their work, at the sizes where a cut can go wrong: rows and keys on both sides of a tile,
a segment and a row tile, ragged batches, column widths of the projections, pieces of a host prompt.  The
reference is the oracle, plain PyTorch in fp32 for the projections, and the path's own invariant: a position's
result is the same bits whether it came in a prompt or as a decoded token."""
import ctypes
import dataclasses

import numpy as np
import pytest

from oracle import hydra_oracle as ho
from tests import hydra_testlib as tl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hb():
    import hydra_b200
    return hydra_b200


@pytest.fixture(scope="module")
def ctx(hb):
    c = hb.Context(0)
    yield c
    c.close()


def _filled(hb, ctx, d, qh, kvh, window, tokens, seqs=1, io="bf16", gated=False):
    rng = np.random.default_rng(d * 31 + qh + tokens)
    q = tl.normal_bf16(rng, (tokens, qh, d))
    k = tl.normal_bf16(rng, (tokens, kvh, d))
    v = tl.normal_bf16(rng, (tokens, kvh, d))
    sinks = tl.normal_bf16(rng, (qh,))
    gate = tl.normal_bf16(rng, (tokens, qh, d)) if gated else None
    layer = tl.Layer(hb, ctx, qh, kvh, d, 4608, window=window, sinks=sinks, io=io, max_seqs=seqs,
                     storage=hb.capi.HC_STORAGE_LINEAR)
    for seq in range(seqs):
        layer.append(k, v, 0, seq=seq)
    return layer, q, k, v, sinks, gate


@pytest.mark.parametrize("d, qh, kvh, window, tokens, io, gated", [
    (64, 64, 8, 0, 2203, "bf16", False),       # three segments of 1024, a last row tile of 11 tokens
    (64, 64, 8, 128, 1100, "f32", False),      # two tiles a row
    (64, 8, 8, 0, 1153, "bf16", True),         # one head a group: 128 tokens a row tile
    (64, 16, 2, 200, 1301, "f32", True),       # gated fp32 rows, several segments
    (128, 16, 2, 0, 1290, "bf16", False),
    (256, 16, 8, 1024, 2180, "bf16", False),   # pairs of SMs; the window crosses a segment of 2048
    (256, 16, 2, 0, 2305, "bf16", True),       # the gated epilogue
    (256, 4, 4, 0, 383, "f32", False),
    (512, 16, 1, 0, 1031, "bf16", False),      # two halves of O, segments of 2048 for decode and prefill alike
    (512, 8, 1, 0, 130, "bf16", False),
])
def test_prompt_rows_equal_decoded_tokens_and_the_oracle(hb, ctx, d, qh, kvh, window, tokens, io, gated):
    layer, q, k, v, sinks, gate = _filled(hb, ctx, d, qh, kvh, window, tokens, io=io, gated=gated)
    prompt = layer.prefill(q, 0, gate=gate)
    edges = [0, 1, 15, 16, 127, 128, 129, 255, 256, 1023, 1024, 1151, 1152, 2047, 2048, 2049, tokens - 2, tokens - 1]
    rows = sorted({r for r in edges if r < tokens})
    for r in rows:
        one = layer.decode(q[r:r + 1], [r], gate=None if gate is None else gate[r:r + 1])
        assert np.array_equal(one[0], prompt[r]), r
    want = ho.attention_rows(q[rows], np.asarray(rows), k, v, 1 / np.sqrt(d), window, sinks=sinks,
                             gate=None if gate is None else gate[rows])
    assert tl.within_tolerance(prompt[rows], want, bf16_output=io == "bf16")
    # the same rows as the end of a later chunk
    tail = min(tokens, 37)
    assert np.array_equal(layer.prefill(q[-tail:], tokens - tail, gate=None if gate is None else gate[-tail:]), prompt[-tail:])
    layer.close()


@pytest.mark.parametrize("d, qh, kvh, window", [(64, 64, 8, 0), (64, 64, 8, 128), (128, 16, 2, 0), (256, 16, 2, 0), (512, 16, 1, 0)])
@pytest.mark.parametrize("n_seq", [2, 13, 64])
def test_ragged_batches_equal_their_rows_alone(hb, ctx, d, qh, kvh, window, n_seq):
    tokens = 2305
    layer, q, k, v, sinks, _ = _filled(hb, ctx, d, qh, kvh, window, tokens, seqs=4)
    rng = np.random.default_rng(n_seq)
    positions = [0, 127, 128, 1023, 1024, 2047, 2048, tokens - 1] + [int(p) for p in rng.integers(0, tokens, 64)]
    positions = positions[-n_seq:] if n_seq < 8 else positions[:n_seq]
    ids = [b % 4 for b in range(n_seq)]
    got = layer.decode(q[positions], positions, seq_ids=ids)
    for b in range(0, n_seq, max(1, n_seq // 6)):
        alone = layer.decode(q[positions[b]:positions[b] + 1], positions[b:b + 1], seq_ids=ids[b:b + 1])
        assert np.array_equal(alone[0], got[b]), b
    want = ho.attention_rows(q[positions], np.asarray(positions), k, v, 1 / np.sqrt(d), window, sinks=sinks)
    assert tl.within_tolerance(got, want)
    layer.close()


@pytest.mark.parametrize("tokens", [1, 16, 17, 64, 65, 128, 129, 257, 900])
@pytest.mark.parametrize("n_in, widths", [(2880, (4096, 512, 512)), (2048, (9216,)), (64, (40,)), (192, (2880, 72)), (4096, (2888,))])
def test_projections_of_every_tile_shape(hb, ctx, tokens, n_in, widths):
    """Up to 128 tokens one column tile per SM (16 to 64 wide), above that pairs of SMs with 128 to 256 columns:
    token counts and widths around all of them, K steps that do not fill a stage."""
    import torch
    backend = hb.AttentionBackend(ctx)
    gen = torch.Generator(device="cuda").manual_seed(tokens + n_in)

    def bf16(*shape, scale=1.0):
        return (torch.randn(shape, generator=gen, device="cuda") * scale).to(torch.bfloat16)

    x = bf16(tokens, n_in)
    w = [bf16(n, n_in, scale=0.02) for n in widths]
    b = [bf16(n) for n in widths]
    want = [x.float() @ wi.float().T + bi.float() for wi, bi in zip(w, b)]
    out = [torch.empty((tokens, n), device="cuda") for n in widths]
    backend.linear_group(x, w, b, out, tokens, n_in, y_dtype=hb.capi.HC_F32)
    residual = torch.randn((tokens, widths[0]), generator=gen, device="cuda")
    updated = residual.clone()
    backend.linear(x, w[0], b[0], updated, tokens, n_in, widths[0], y_dtype=hb.capi.HC_F32, residual=updated)
    ctx.check()
    for got, ref in zip(out, want):
        assert float((got - ref).abs().max()) <= 1e-3 * max(1.0, float(ref.abs().max()))
    assert torch.equal(updated, out[0] + residual)


@pytest.mark.parametrize("d, qh, kvh, window, tokens, io", [
    (64, 64, 8, 0, 40, "bf16"), (64, 64, 8, 0, 2500, "bf16"), (64, 64, 8, 128, 1700, "bf16"),
    (64, 64, 8, 0, 700, "f32"), (256, 16, 8, 256, 3000, "bf16"), (128, 16, 2, 0, 4096, "bf16"),
])
def test_host_prompts_in_pieces_equal_device_prompts(hb, ctx, d, qh, kvh, window, tokens, io):
    import torch
    rng = np.random.default_rng(tokens)
    dtype = torch.bfloat16 if io == "bf16" else torch.float32
    host = [torch.from_numpy(tl.normal_bf16(rng, (tokens, h, d))).to(dtype).pin_memory() for h in (qh, kvh, kvh)]
    outs = []
    for on_host in (False, True):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 4608, window=window, io=io, prefill_chunk=256,
                         rope_inv_freq=ho.inverse_frequencies(d, 10000.0))
        q, k, v = host if on_host else [t.cuda() for t in host]
        out = torch.zeros((tokens, qh, d), dtype=dtype)
        out = out.pin_memory() if on_host else out.cuda()
        call = layer.backend.prefill_host if on_host else layer.backend.prefill_chunks
        call(layer.cache, 0, q, k, v, out, tokens, 0, 256, layer.params)
        ctx.check()
        outs.append(tl.to_host(out))
        layer.close()
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("tokens", [1, 5, 200])
def test_stack_call_equals_its_parts(hb, ctx, tokens):
    """hc_attention_stack_host over two gated layers of different windows against the same calls one by one."""
    import torch
    capi, width, qh, kvh, d = hb.capi, 320, 8, 2, 64
    backend = hb.AttentionBackend(ctx)
    gen = torch.Generator(device="cuda").manual_seed(tokens)

    def bf16(*shape, scale=0.05):
        return (torch.randn(shape, generator=gen, device="cuda") * scale).to(torch.bfloat16)

    windows = (128, 0)
    shapes = dict(input_norm=(width,), wq=(2 * qh * d, width), bq=(2 * qh * d,), wk=(kvh * d, width), bk=(kvh * d,),
                  wv=(kvh * d, width), bv=(kvh * d,), wo=(width, qh * d), bo=(width,))
    layers = [{name: bf16(*shape) for name, shape in shapes.items()} for _ in windows]
    params = [hb.AttnParams(q_heads=qh, kv_heads=kvh, head_dim=d, window=w, sm_scale=0.125, io_dtype=capi.HC_BF16,
                            gate_layout=capi.HC_GATE_INTERLEAVED) for w in windows]
    states = torch.randn((tokens, width), generator=gen, device="cuda")
    caches = [hb.KVCache(ctx, [dict(q_heads=qh, kv_heads=kvh, head_dim=d, window=w) for w in windows], 512) for _ in range(2)]
    want = states.clone()
    for i, (w, p) in enumerate(zip(layers, params)):
        normed = torch.empty((tokens, width), device="cuda", dtype=torch.bfloat16)
        q, k, v, attended = (torch.empty((tokens, n * d), device="cuda", dtype=torch.bfloat16) for n in (2 * qh, kvh, kvh, qh))
        backend.rms_norm(want, w["input_norm"], normed, tokens, width, 1e-5)
        backend.linear_group(normed, [w["wq"], w["wk"], w["wv"]], [w["bq"], w["bk"], w["bv"]], [q, k, v], tokens, width,
                             y_dtype=capi.HC_BF16)
        backend.layer_step(caches[0], i, q, k, v, attended, tokens, 0, p)
        backend.linear(attended, w["wo"], w["bo"], want, tokens, qh * d, width, y_dtype=capi.HC_F32, residual=want)
    blocks = (capi.BlockWeightsStruct * 2)()
    for block, w, p in zip(blocks, layers, params):
        for name, tensor in w.items():
            setattr(block, name, tensor.data_ptr())
        block.params = p.struct()
    lib = capi.load()
    workspace = torch.empty(lib.hc_attention_stack_bytes(blocks, 2, tokens, width), dtype=torch.uint8, device="cuda")
    host = states.cpu().numpy().copy()
    status = lib.hc_attention_stack_host(ctx.handle, caches[1].handle, blocks, 2, 0, host.ctypes.data, host.ctypes.data, tokens,
                                         width, 0, ctypes.c_float(1e-5), workspace.data_ptr(), None)
    assert status == 0
    assert np.array_equal(host, want.cpu().numpy())
    for cache in caches:
        cache.close()


@pytest.mark.parametrize("d, qh, kvh, window, first, tokens, io, gated", [
    (64, 16, 4, 128, 0, 256, "bf16", False),     # as many tokens as fit beside the ring's window
    (64, 16, 4, 128, 0, 257, "bf16", False),     # one more: the prompt attends outside the ring
    (64, 16, 4, 128, 131, 700, "f32", False),    # behind an odd history, which comes along
    (96, 8, 4, 130, 259, 600, "bf16", False),    # the CUDA-core kernels, the general prologue
    (128, 16, 2, 300, 640, 1290, "bf16", True),
    (256, 16, 8, 256, 77, 1500, "bf16", False),
    (256, 64, 4, 384, 515, 2300, "f32", False),  # more than the prepared queries have room for: two parts
    (256, 64, 4, 384, 515, 2300, "bf16", "separate"),     # a gate of its own, which the parts are given their rows of
    (64, 16, 4, 128, 131, 700, "f32", "separate"),
    (256, 16, 8, 256, 77, 1500, "bf16", "norms"),         # queries, keys and values normed
    (96, 8, 4, 130, 259, 600, "f32", "norms"),
])
def test_prompts_longer_than_a_ring_equal_linear_storage(hb, ctx, d, qh, kvh, window, first, tokens, io, gated):
    """Outputs, the ring's rows and a decoded token behind them: the same bits as with linear storage, twice in a row."""
    rng = np.random.default_rng(d + window + tokens)
    end, width = first + tokens, d * (2 if gated is True else 1)
    gate = tl.to_device(tl.normal_bf16(rng, (tokens + 1, qh, d)), io) if gated == "separate" else None
    norms = dict(q_norm=1 + 0.1 * tl.normal_bf16(rng, (d,)), k_norm=1 + 0.1 * tl.normal_bf16(rng, (d,)), norm_v=True) if gated == "norms" else {}
    k, v = tl.normal_bf16(rng, (end + 1, kvh, d)), tl.normal_bf16(rng, (end + 1, kvh, d))
    q = tl.normal_bf16(rng, (tokens + 1, qh, width))
    sinks = tl.normal_bf16(rng, (qh,))
    inv = ho.inverse_frequencies(d, 10000.0, d // 2)
    got = []
    for storage in (hb.capi.HC_STORAGE_RING, hb.capi.HC_STORAGE_LINEAR):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 4096, window=window, sinks=sinks, rope_inv_freq=inv, io=io, prefill_chunk=128,
                         storage=storage, gate_layout=hb.capi.HC_GATE_INTERLEAVED if gated is True else 0, max_seqs=2, **norms)
        prompt_params = decode_params = layer.params
        if gate is not None:
            prompt_params, decode_params = layer._with_gate(gate), layer._with_gate(gate[tokens:])
        dev = [tl.to_device(x, io) for x in (q, k, v)]
        out = tl.device_empty((tokens + 1, qh, d), io)
        for seq in (1, 1, 0):
            for at in range(0, first, 128):
                layer.append(k[at:min(at + 128, first)], v[at:min(at + 128, first)], at, seq=seq)
            out.fill_(7.0)
            layer.backend.prefill_chunks(layer.cache, 0, dev[0], dev[1][first:], dev[2][first:], out, tokens, first, 128,
                                         prompt_params, seq=seq)
            layer.backend.layer_step(layer.cache, 0, dev[0][tokens:], dev[1][end:], dev[2][end:], out[tokens:], 1, end, decode_params,
                                     seq=seq)
        ctx.check()
        held = min(end + 1, window + 128)
        rows = tl.read_cache(layer.cache, 0, held, kvh, d, seq=0, position=end + 1 - held)
        got.append([tl.to_host(out), *rows])
        layer.close()
    for ring, linear in zip(*got):
        assert np.array_equal(ring, linear)


@pytest.mark.parametrize("d, qh, kvh, window, first, tokens, blocks", [
    (64, 16, 4, 128, 0, 645, False),      # no history: nothing is copied out of the ring
    (64, 16, 4, 128, 259, 645, True),
    (96, 8, 4, 130, 77, 600, False),      # the CUDA-core kernels
    (96, 8, 4, 130, 0, 601, True),
    (128, 16, 2, 300, 131, 1001, False),
    (256, 16, 8, 256, 0, 1151, False),
    (256, 16, 8, 256, 77, 1027, True),
    (256, 64, 4, 384, 515, 2300, False),  # two parts, the first of which ends inside a key tile as well
    (512, 8, 1, 200, 3, 900, False),
])
def test_prompts_beside_a_ring_see_no_other_prompt(hb, ctx, d, qh, kvh, window, first, tokens, blocks):
    """Infinities and NaN in another sequence's prompt, of the same ring layer and of one of another geometry, right before
    it: the bits of linear storage, in which sequences and layers lie apart."""
    import torch
    geometry = [(qh, kvh, d, window), (6, 3, 64, 200)]
    rng = np.random.default_rng(d + first + tokens)
    bad = [torch.full((1100, k, dim), float("nan"), device="cuda") for _, k, dim, _ in geometry]
    for x in bad:
        x[::2] = float("inf")
    ends = np.zeros(tokens, np.int32)
    for at, n in ((3, 40), (90, 120), (tokens - 60, 60)):
        ends[at:at + n] = first + at + n
    ends = torch.from_numpy(ends).cuda() if blocks else None
    inputs = [[tl.to_device(tl.normal_bf16(rng, (n, heads, dim)), "f32") for n, heads in ((tokens, q), (first + tokens, k), (first + tokens, k))]
              for q, k, dim, _ in geometry]
    got = []
    for storage in (hb.capi.HC_STORAGE_RING, hb.capi.HC_STORAGE_LINEAR):
        cache = hb.KVCache(ctx, [dict(q_heads=q, kv_heads=k, head_dim=dim, window=w, storage=storage) for q, k, dim, w in geometry],
                           4096, prefill_chunk=128, max_seqs=2)
        be = hb.AttentionBackend(ctx)
        params = [hb.AttnParams(q_heads=q, kv_heads=k, head_dim=dim, window=w, sm_scale=dim ** -0.5, io_dtype=hb.capi.HC_F32)
                  for q, k, dim, w in geometry]
        outs = []
        for other in (0, 1):
            for layer, ((q, k, dim, _), (xq, xk, xv)) in enumerate(zip(geometry, inputs)):
                for at in range(0, first, 128):
                    n = min(128, first - at)
                    be.write_key_value(cache, layer, xk[at:], xv[at:], n, at, params[layer], seq=1)
                wide = torch.ones(1100, geometry[other][0], geometry[other][2], device="cuda")
                be.prefill_chunks(cache, other, wide, bad[other], bad[other], torch.empty_like(wide), 1100, 0, 128, params[other], seq=0)
                out = torch.full((tokens, q, dim), 7.0, device="cuda")
                be.prefill_chunks(cache, layer, xq, xk[first:], xv[first:], out, tokens, first, 128,
                                  dataclasses.replace(params[layer], block_ends=ends), seq=1)
                ctx.check()
                outs.append(out.cpu().numpy())
        got.append(outs)
        cache.close()
    for ring, linear in zip(*got):
        assert np.all(np.isfinite(linear)) and np.array_equal(ring, linear)


def test_a_ring_without_room_for_its_prompt_store(hb, ctx):
    """The ring takes more than half of the free memory, so that the store, as large, does not fit: prompts take the ring in
    pieces, with the bits of linear storage."""
    import torch
    torch.cuda.empty_cache()
    qh, kvh, d, tokens = 8, 8, 512, 700
    window = int(0.55 * torch.cuda.mem_get_info()[0]) // (4 * kvh * d) // 128 * 128
    rng = np.random.default_rng(7)
    q, k, v = (tl.normal_bf16(rng, (tokens, kvh, d)) for _ in range(3))
    got, launches = [], []
    for storage, w in ((hb.capi.HC_STORAGE_RING, window), (hb.capi.HC_STORAGE_RING, 1024), (hb.capi.HC_STORAGE_LINEAR, 1024)):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 4096, window=w, storage=storage, io="f32", prefill_chunk=128)
        out = tl.device_empty((tokens, qh, d), "f32")
        before = ctx.launch_count
        layer.backend.prefill_chunks(layer.cache, 0, tl.to_device(q, "f32"), tl.to_device(k, "f32"), tl.to_device(v, "f32"), out, tokens,
                                     0, 128, layer.params)
        ctx.check()
        launches.append(ctx.launch_count - before)
        got.append(tl.to_host(out))
        layer.close()
    assert np.array_equal(got[0], got[2]) and np.array_equal(got[1], got[2])
    assert launches[0] > launches[1]


@pytest.mark.parametrize("d, qh, kvh, tokens, window", [(64, 16, 2, 77, 0), (64, 64, 8, 300, 128), (256, 16, 8, 140, 0), (256, 8, 8, 515, 256),
                                                       (512, 8, 1, 65, 0)])
def test_outputs_on_16_byte_boundaries_that_are_no_32_byte_ones(hb, ctx, d, qh, kvh, tokens, window):
    import torch
    layer, q, k, v, sinks, _ = _filled(hb, ctx, d, qh, kvh, window, tokens)
    want = layer.prefill(q, 0)
    flat = torch.full((tokens * qh * d + 16,), 7.0, device="cuda", dtype=torch.bfloat16)
    layer.backend.attention_prefill(layer.cache, 0, tl.to_device(q), flat[8:-8].view(tokens, qh, d), tokens, 0, layer.params)
    ctx.check()
    assert np.array_equal(tl.to_host(flat[8:-8]).reshape(want.shape), want)
    assert bool((flat[:8] == 7).all()) and bool((flat[-8:] == 7).all())
    layer.close()


@pytest.mark.parametrize("d", [64, 128, 256, 512])
def test_fp32_rows_on_16_byte_boundaries_that_are_no_32_byte_ones(hb, ctx, d):
    """The prologue reads and writes fp32 vectors 32 bytes a lane where they lie so: appended rows and vectors normalised in
    place are the same bits where they do not."""
    import torch
    tokens, heads = 700, 5
    gen = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn(2, tokens, heads, d, device="cuda", generator=gen)
    weight = (1 + 0.1 * torch.randn(d, device="cuda", generator=gen)).to(torch.bfloat16)
    inv = ho.inverse_frequencies(d, 10000.0, d // 2)
    layer = tl.Layer(hb, ctx, heads, heads, d, 1024, rope_inv_freq=inv, io="f32")
    got = []
    for offset in (0, 4):
        flat = torch.full((2, tokens * heads * d + 8), 7.0, device="cuda")
        k, v = (flat[i, offset:offset + tokens * heads * d].view(tokens, heads, d) for i in range(2))
        k.copy_(x[0])
        v.copy_(x[1])
        layer.backend.write_key_value(layer.cache, 0, k, v, tokens, 0, layer.params)
        ctx.check()
        rows = tl.read_cache(layer.cache, 0, tokens, heads, d)
        layer.backend.rms_norm_heads(k, weight, tokens, heads, d, 1e-6)
        ctx.check()
        got.append([*rows, k.cpu().numpy()])
        assert float(flat[0, :offset].sub(7).abs().sum()) == 0.0 and bool((flat[0, offset + tokens * heads * d:] == 7).all())
    layer.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))
    want = x[0].double()
    want = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-6) * weight.double()
    assert np.max(np.abs(got[0][2] - want.cpu().numpy())) < 1e-5


@pytest.mark.parametrize("io", ["bf16", "f32"])
@pytest.mark.parametrize("d, heads", [(64, 5), (128, 6), (256, 16), (512, 3)])
def test_prologue_of_a_wave_and_of_more(hb, ctx, d, heads, io):
    """One token fewer and more than one wave of the kernel for few vectors holds: appended rows and vectors normed in place
    are the bits of a call for each half, which that kernel takes; normed vectors are float64's (relative error of the sum
    d 2^-24, of the root and two products 2^-22; bf16, which has 8 significant bits, half a step 2^-8 more)."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per_warp, blocks = max(256 // d, 1), 3 if d == 512 else 4
    gen = torch.Generator(device="cuda").manual_seed(d)
    weight = (1 + 0.1 * torch.randn(d, device="cuda", generator=gen)).to(torch.bfloat16)
    dtype, code = (torch.bfloat16, hb.capi.HC_BF16) if io == "bf16" else (torch.float32, hb.capi.HC_F32)
    most = sms * blocks * 8
    layer = tl.Layer(hb, ctx, heads, heads, d, most, rope_inv_freq=ho.inverse_frequencies(d, 10000.0, d // 2), io=io)
    be, bound = layer.backend, d * 2.0 ** -24 + 2.0 ** -22 + (2.0 ** -8 if io == "bf16" else 0)
    for tokens in [n + e for n in {most // -(-heads // per_warp), most // -(-2 * heads // per_warp)} for e in (0, 1)]:
        x = torch.randn(2, tokens, heads, d, device="cuda", generator=gen).to(dtype)
        got = []
        for cut in (tokens, tokens // 2):
            y = x[0].clone()
            for a, b in ((0, cut), (cut, tokens)):
                if a == b:
                    continue
                be.write_key_value(layer.cache, 0, x[0, a:], x[1, a:], b - a, a, layer.params)
                be.rms_norm_heads(y[a:], weight, b - a, heads, d, 1e-6, io_dtype=code)
            ctx.check()
            got.append([y.float().cpu().numpy(), *tl.read_cache(layer.cache, 0, tokens, heads, d)])
        assert all(np.array_equal(a, b) for a, b in zip(*got))
        want = x[0].double()
        want = (want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-6) * weight.double()).cpu().numpy()
        assert np.max(np.abs(got[0][0] - want) / np.maximum(np.abs(want), 1e-30)) < bound
    layer.close()


def test_fp32_rows_of_512_that_exceed_l2(hb, ctx):
    """More than 64 MB of them are appended by the kernel for few vectors, in a walk: the bits of a call for each third."""
    import torch
    tokens, heads, d = 2200, 8, 512                       # 72 MB of keys and values
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(2, tokens, heads, d, device="cuda", generator=gen)
    layer = tl.Layer(hb, ctx, heads, heads, d, tokens, rope_inv_freq=ho.inverse_frequencies(d, 10000.0, d // 2), io="f32")
    got = []
    for step in (tokens, 734):
        for a in range(0, tokens, step):
            layer.backend.write_key_value(layer.cache, 0, x[0, a:], x[1, a:], min(step, tokens - a), a, layer.params)
        ctx.check()
        got.append(tl.read_cache(layer.cache, 0, tokens, heads, d))
    layer.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))
