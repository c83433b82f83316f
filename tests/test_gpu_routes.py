"""Calls that take another way through the library than the one they are usually made in: each has to give what the
plain sequence of calls gives, bit for bit, or what the oracle gives."""
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


def _inputs(seed, tokens, qh, kvh, d):
    rng = np.random.default_rng(seed)
    return [tl.normal_bf16(rng, (tokens, h, d)) for h in (qh, kvh, kvh)]


@pytest.mark.parametrize("call", ["layer_step", "prefill_chunks"])
@pytest.mark.parametrize("d, rope", [(64, False), (256, True)])
def test_blocks_in_a_call_of_several_cache_chunks(hb, ctx, call, d, rope):
    """With bidirectional blocks a call is worked in chunks of the cache's prefill_chunk: the keys and values that are
    appended with a later chunk's queries are that chunk's own rows."""
    import torch
    qh, kvh, tokens, chunk = 8, 2, 300, 128
    q, k, v = _inputs(d, tokens, qh, kvh, d)
    ends = np.zeros(tokens, np.int32)
    ends[20:90], ends[140:200] = 90, 200
    outs, rows = [], []
    for fused in (False, True):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 1024, prefill_chunk=chunk,
                         rope_inv_freq=ho.inverse_frequencies(d, 10000.0) if rope else None)
        params = dataclasses.replace(layer.params, block_ends=torch.from_numpy(ends).cuda())
        qd, kd, vd, out = tl.to_device(q), tl.to_device(k), tl.to_device(v), tl.device_empty((tokens, qh, d))
        if not fused:
            layer.backend.write_key_value(layer.cache, 0, kd, vd, tokens, 0, layer.params)
            layer.backend.attention_prefill(layer.cache, 0, qd, out, tokens, 0, params)
        elif call == "layer_step":
            layer.backend.layer_step(layer.cache, 0, qd, kd, vd, out, tokens, 0, params)
        else:
            layer.backend.prefill_chunks(layer.cache, 0, qd, kd, vd, out, tokens, 0, tokens, params)
        ctx.check()
        outs.append(tl.to_host(out))
        rows.append(tl.read_cache(layer.cache, 0, tokens, kvh, d))
        layer.close()
    assert np.array_equal(rows[0][0], rows[1][0]) and np.array_equal(rows[0][1], rows[1][1])
    assert np.array_equal(outs[0], outs[1])


def test_runner_reads_its_weights_where_they_are_now(hb, ctx):
    """A program may put other tensors, sinks or parameters in a runner's lists between passes: what a pass reads is
    what they hold then."""
    from hydra_b200.runner import AttentionLayerWeights, AttentionStackRunner
    rng = np.random.default_rng(3)
    width, qh, kvh, d, tokens = 128, 4, 2, 64, 9
    shapes = dict(wq=(qh * d, width), bq=(qh * d,), wk=(kvh * d, width), bk=(kvh * d,), wv=(kvh * d, width),
                  bv=(kvh * d,), wo=(width, qh * d), bo=(width,))

    def layer():
        weights = {name: ho.bf16_round(rng.normal(0, 0.1, shape)) for name, shape in shapes.items()}
        return AttentionLayerWeights(input_norm=ho.bf16_round(1 + 0.1 * rng.standard_normal(width)), window=0,
                                     sinks=tl.normal_bf16(rng, (qh,)), **weights)

    def runner(layers):
        return AttentionStackRunner(ctx, layers, width, qh, kvh, d, context_length=256, prefill_chunk_tokens=128)

    states = rng.standard_normal((tokens, width)).astype(np.float32)
    first, second = [layer(), layer()], [layer(), layer()]
    changed, fresh = runner(first), runner(second)
    before = changed.verify(states)
    kept = list(changed.weights)                 # (the old tensors stay alive: nothing here reads freed memory)
    for index in range(2):
        changed.weights[index] = dict(fresh.weights[index])
        changed.params[index].sinks = fresh.weights[index]["sinks"]
    changed.reset()
    got, want = changed.verify(states), fresh.verify(states)
    assert not np.array_equal(before, want) and len(kept) == 2
    assert np.array_equal(got, want)
    changed.params[1].sm_scale = 0.5
    changed.reset()
    assert not np.array_equal(changed.verify(states), want)
    changed.params[1].sm_scale = fresh.params[1].sm_scale
    for weights in (changed.weights[0], fresh.weights[0]):
        weights["bk"] = None                     # a projection without a bias
    changed.reset()
    fresh.reset()
    without = changed.verify(states)
    assert np.array_equal(without, fresh.verify(states)) and not np.array_equal(without, want)
    changed.close()
    fresh.close()


@pytest.mark.parametrize("d, heads", [(64, 80000), (256, 20000), (512, 19000)])
def test_one_token_of_very_many_heads(hb, ctx, d, heads):
    """The element-wise entry points take the rows of a matrix as one token's heads: more of them than the launch has
    warps."""
    import torch
    be = hb.AttentionBackend(ctx)
    gen = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn((heads, d), device="cuda", generator=gen)
    weight = torch.randn(d, device="cuda", generator=gen).to(torch.bfloat16)
    table = hb.RopeTable(ctx, list(ho.inverse_frequencies(d, 10000.0)), 8)
    rows, one = x.clone(), x.clone()
    be.rms_norm_heads(rows, weight, heads, 1, d, 1e-6, hb.capi.HC_F32)
    be.rms_norm_heads(one, weight, 1, heads, d, 1e-6, hb.capi.HC_F32)
    ctx.check()
    assert torch.equal(rows, one) and not torch.equal(rows, x)
    parts, one = x.clone(), x.clone()
    for start in range(0, heads, 5000):
        count = min(5000, heads - start)
        be.apply_rope(parts[start:start + count], table, 1, count, d, 5, hb.capi.HC_F32)
    be.apply_rope(one, table, 1, heads, d, 5, hb.capi.HC_F32)
    ctx.check()
    assert torch.equal(parts, one) and not torch.equal(parts, x)
    table.close()


@pytest.mark.parametrize("context, chunk, tokens", [(200, 64, 2000), (4096, 64, 700)])
def test_host_prompt_on_a_ring(hb, ctx, context, chunk, tokens):
    """A ring takes prompts longer than the context the cache was made for; the pieces of a host prompt are as long as
    both the ring and the prepared-query buffer allow."""
    import torch
    qh, kvh, d, window = 8, 2, 64, 128
    q, k, v = _inputs(tokens, tokens, qh, kvh, d)
    outs = []
    for on_host in (False, True):
        layer = tl.Layer(hb, ctx, qh, kvh, d, context, window=window, storage=hb.capi.HC_STORAGE_RING, prefill_chunk=chunk)
        if on_host:
            host = [torch.from_numpy(a).to(torch.bfloat16).pin_memory() for a in (q, k, v)]
            out = torch.zeros((tokens, qh, d), dtype=torch.bfloat16).pin_memory()
            layer.backend.prefill_host(layer.cache, 0, *host, out, tokens, 0, chunk, layer.params)
        else:
            qd, kd, vd, out = tl.to_device(q), tl.to_device(k), tl.to_device(v), tl.device_empty((tokens, qh, d))
            for at in range(0, tokens, chunk):
                n = min(chunk, tokens - at)
                layer.backend.layer_step(layer.cache, 0, qd[at:], kd[at:], vd[at:], out[at:], n, at, layer.params)
        ctx.check()
        outs.append(tl.to_host(out))
        layer.close()
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("qh, d, io", [(1, 8, "bf16"), (1, 64, "f32"), (2, 64, "bf16")])
def test_host_step_of_the_smallest_caches(hb, ctx, qh, d, io):
    """The staging buffer holds a chunk of the cache's own size whatever that is."""
    import torch
    rng = np.random.default_rng(d)
    layer = tl.Layer(hb, ctx, qh, 1, d, 256, prefill_chunk=1, io=io)
    dtype = torch.bfloat16 if io == "bf16" else torch.float32
    k_rows, v_rows = [], []
    for position in range(3):
        q, k, v = (tl.normal_bf16(rng, (1, h, d)) for h in (qh, 1, 1))
        k_rows.append(k)
        v_rows.append(v)
        out = torch.zeros((1, qh, d), dtype=dtype)
        host = [torch.from_numpy(a).to(dtype) for a in (q, k, v)]
        layer.backend.layer_step_host(layer.cache, 0, *host, out, 1, position, layer.params)
        want = ho.attention_rows(q, np.asarray([position]), np.concatenate(k_rows), np.concatenate(v_rows), 1 / np.sqrt(d))
        assert tl.within_tolerance(tl.to_host(out), want, bf16_output=io == "bf16")
    layer.close()


@pytest.mark.parametrize("d, qh, kvh, window, rows", [(64, 64, 8, 0, 8), (64, 64, 8, 128, 16), (256, 16, 2, 0, 8),
                                                      (512, 16, 2, 0, 8), (64, 16, 16, 0, 40)])
def test_rows_of_one_sequence_in_one_launch(hb, ctx, d, qh, kvh, window, rows):
    """Several positions of one sequence decoded together: one launch as long as the workspace holds its partials."""
    tokens = 2100
    q, k, v = _inputs(d + rows, tokens, qh, kvh, d)
    layer = tl.Layer(hb, ctx, qh, kvh, d, 4608, window=window)
    layer.append(k, v, 0)
    positions = [0, 127, 128, 1023, 1024, 2047, 2048, tokens - 1] + list(range(100, 100 + 40 * (rows - 8), 40))
    before = ctx.launch_count
    got = layer.decode(q[positions], positions, seq_ids=[0] * rows)
    assert ctx.launch_count - before == 1
    for b in range(rows):
        alone = layer.decode(q[positions[b]:positions[b] + 1], positions[b:b + 1])
        assert np.array_equal(alone[0], got[b]), b
    layer.close()


@pytest.mark.parametrize("d, qh, kvh, window, paged", [(64, 64, 8, 0, False), (64, 64, 8, 128, True), (128, 16, 2, 0, True),
                                                       (256, 16, 2, 0, True), (512, 16, 1, 0, False), (64, 16, 16, 0, False)])
def test_a_full_batch_is_one_launch(hb, ctx, d, qh, kvh, window, paged):
    """64 ragged sequences in a cache made for them: one launch cut as one line, long lists of rows a block (1024 rows
    in the last case), the search over a full table of sequences, segments of 1024 keys."""
    tokens, n_seq = 2305, 64
    q, k, v = _inputs(d + kvh, tokens, qh, kvh, d)
    rng = np.random.default_rng(d)
    lengths = [1, 128, 129, 1024, 1025, 2048, 2049, tokens] + [int(n) for n in rng.integers(1, 700, n_seq - 8)]
    pages = sum((n + 127) // 128 for n in lengths) if paged else 0
    cache = hb.KVCache(ctx, [dict(q_heads=qh, kv_heads=kvh, head_dim=d, window=window)], 2432, max_seqs=n_seq, total_pages=pages)
    be = hb.AttentionBackend(ctx)
    params = hb.AttnParams(q_heads=qh, kv_heads=kvh, head_dim=d, window=window, sm_scale=1 / np.sqrt(d), io_dtype=hb.capi.HC_BF16)
    kd, vd = tl.to_device(k), tl.to_device(v)
    for seq, n in enumerate(lengths):
        if n > 1:
            be.write_key_value(cache, 0, kd, vd, n - 1, 0, params, seq=seq)
    positions, ids = [n - 1 for n in lengths], list(range(n_seq))
    be.write_key_value_batch(cache, 0, kd[positions], vd[positions], ids, positions, params)
    qd, out = tl.to_device(q[positions]), tl.device_empty((n_seq, qh, d))
    before = ctx.launch_count
    be.attention(cache, 0, qd, out, positions, params, seq_ids=ids)
    assert ctx.launch_count - before == 1
    ctx.check()
    got = tl.to_host(out)
    for b in list(range(10)) + [37, 63]:
        alone = tl.device_empty((1, qh, d))
        be.attention(cache, 0, qd[b:b + 1], alone, positions[b:b + 1], params, seq_ids=ids[b:b + 1])
        ctx.check()
        assert np.array_equal(tl.to_host(alone)[0], got[b]), b
    want = ho.attention_rows(q[positions], np.asarray(positions), k, v, 1 / np.sqrt(d), window)
    assert tl.within_tolerance(got, want)
    cache.close()


@pytest.mark.parametrize("d, qh, kvh, window", [(64, 8, 2, 128), (64, 64, 8, 1000), (256, 16, 8, 1024), (512, 8, 1, 300)])
def test_positions_beyond_eight_million(hb, ctx, d, qh, kvh, window):
    """A ring takes any position.  Without a rotation the results depend on where the keys lie in their tiles and
    segments only: far up the sequence they are what they are at its beginning, bit for bit."""
    rows, batch = window + 140, 12
    q, k, v = _inputs(d + window, rows, qh, kvh, d)
    got = []
    for base in (3 * 4096 + 77, (1 << 23) + 5 * 4096 + 77, (1 << 30) + 77):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 16384, window=window, storage=hb.capi.HC_STORAGE_RING, prefill_chunk=128)
        for at in range(0, rows, 128):
            layer.append(k[at:at + 128], v[at:at + 128], base + at)
        positions = [base + rows - 1 - 3 * b for b in range(batch)]
        take = [rows - 1 - 3 * b for b in range(batch)]
        together = layer.decode(q[take], positions, seq_ids=[0] * batch)
        alone = layer.decode(q[take[:1]], positions[:1])
        prompt = layer.prefill(q[-9:], base + rows - 9)
        assert np.array_equal(alone[0], together[0]) and np.array_equal(prompt[-1], alone[0])
        got.append((together, prompt))
        layer.close()
    for other in got[1:]:
        assert np.array_equal(got[0][0], other[0]) and np.array_equal(got[0][1], other[1])


@pytest.mark.parametrize("d, qh, kvh, n_seq, longest", [
    (64, 16, 16, 64, 12200),     # 1024 rows of some 90 key tiles: more rows than a launch lists
    (256, 16, 16, 64, 28600),    # the partials of its 2048-key segments take several launches
    (512, 2, 2, 64, 6100),
])
def test_static_decode_serves_what_its_limit_allows(hb, ctx, d, qh, kvh, n_seq, longest):
    """hc_attention_decode_static refuses by the general cut of the rows' keys, not by how the kernels cut them."""
    import torch
    rng = np.random.default_rng(d)
    layer = tl.Layer(hb, ctx, qh, kvh, d, longest + 60)
    gen = torch.Generator(device="cuda").manual_seed(d)
    k, v = (torch.randn((longest, kvh, d), device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2))
    layer.backend.write_key_value(layer.cache, 0, k, v, longest, 0, layer.params)
    positions = [int(p) for p in rng.integers(longest - longest // 10, longest, n_seq)]
    q = tl.normal_bf16(rng, (n_seq, qh, d))
    out = tl.device_empty((n_seq, qh, d))
    layer.backend.attention_static(layer.cache, 0, tl.to_device(q), out, positions, layer.params, seq_ids=[0] * n_seq)
    ctx.check()
    got = tl.to_host(out)
    assert np.array_equal(got, layer.decode(q, positions, seq_ids=[0] * n_seq))
    for b in (0, n_seq // 2, n_seq - 1):
        assert np.array_equal(layer.decode(q[b:b + 1], positions[b:b + 1])[0], got[b]), b
    layer.close()


def _off_by_one(array, io="bf16"):
    """The array on the device, one element behind a 16-byte boundary."""
    import torch
    flat = tl.to_device(array, io).reshape(-1)
    room = torch.empty(flat.numel() + 8, device="cuda", dtype=flat.dtype)
    room[1:1 + flat.numel()] = flat
    return room[1:1 + flat.numel()].view(array.shape)


@pytest.mark.parametrize("d, qh, kvh, window", [(64, 16, 2, 0), (64, 16, 2, 128), (128, 8, 2, 0), (256, 16, 2, 0), (512, 16, 2, 0)])
def test_queries_off_a_16_byte_boundary(hb, ctx, d, qh, kvh, window):
    """Queries that need no prologue, anywhere: the bits of the same queries on a boundary."""
    tokens, rows = 300, 5
    q, k, v = _inputs(d + window, tokens, qh, kvh, d)
    layer = tl.Layer(hb, ctx, qh, kvh, d, 512, window=window)
    kd, vd = _off_by_one(k), _off_by_one(v)
    layer.backend.write_key_value(layer.cache, 0, kd, vd, tokens, 0, layer.params)
    be, cache, params = layer.backend, layer.cache, layer.params
    positions, ids = [3, 127, 128, 256, tokens - 1], [0] * rows
    moved, out = _off_by_one(q), tl.device_empty((tokens, qh, d))
    assert moved.data_ptr() % 16 == 2
    be.attention_prefill(cache, 0, moved, out, tokens, 0, params)
    ctx.check()
    prompt = tl.to_host(out)
    assert np.array_equal(prompt, layer.prefill(q, 0))
    for call in (be.attention, be.attention_static):
        out = tl.device_empty((rows, qh, d))
        call(cache, 0, _off_by_one(q[positions]), out, positions, params, seq_ids=ids)
        ctx.check()
        assert np.array_equal(tl.to_host(out), prompt[positions])
    # a token's own rows, appended by its step
    out = tl.device_empty((1, qh, d))
    be.layer_step(cache, 0, _off_by_one(q[-1:]), _off_by_one(k[-1:]), _off_by_one(v[-1:]), out, 1, tokens - 1, params)
    ctx.check()
    assert np.array_equal(tl.to_host(out)[0], prompt[-1])
    layer.close()


@pytest.mark.parametrize("d, qh, kvh, window, io, gated, blocks", [
    (64, 16, 2, 0, "bf16", False, False), (64, 64, 8, 128, "f32", True, True), (128, 8, 2, 0, "bf16", True, True),
    (256, 16, 2, 0, "f32", True, False), (256, 16, 8, 300, "bf16", False, True), (512, 16, 2, 0, "bf16", False, False),
    (512, 8, 1, 0, "f32", True, True),
])
def test_outputs_off_a_16_byte_boundary(hb, ctx, d, qh, kvh, window, io, gated, blocks):
    """A prompt's rows stored element by element, in one pass or (the small workspace of a cache made for chunks of 16)
    several: the bits of the same call on a boundary, bidirectional blocks and gates included."""
    import torch
    tokens, first = 700, 1900
    rng = np.random.default_rng(d + tokens)
    q = tl.normal_bf16(rng, (tokens, qh, d))
    k, v = (tl.normal_bf16(rng, (first + tokens, kvh, d)) for _ in range(2))
    gate = tl.normal_bf16(rng, (tokens, qh, d))
    ends = np.zeros(tokens, np.int32)
    ends[100:230], ends[600:690] = first + 230, first + 690
    for chunk in (1024, 16):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 2816, window=window, io=io, prefill_chunk=chunk)
        layer.append(k, v, 0)
        more = dict(block_ends=torch.from_numpy(ends).cuda()) if blocks else {}
        if gated:
            more.update(gate_layout=hb.capi.HC_GATE_SEPARATE, gate=_off_by_one(gate, io))
        params = dataclasses.replace(layer.params, **more)
        qd = tl.to_device(q, io)
        outs = []
        for shift in (0, 1):
            room = torch.full((tokens * qh * d + 8,), 7.0, device="cuda", dtype=qd.dtype)
            out = room[shift:shift + tokens * qh * d].view(tokens, qh, d)
            layer.backend.attention_prefill(layer.cache, 0, qd, out, tokens, first, params)
            ctx.check()
            outs.append(tl.to_host(out))
            assert bool((room[:shift] == 7).all()) and bool((room[shift + tokens * qh * d:] == 7).all())
            one = room[shift:shift + qh * d].view(1, qh, d)
            layer.backend.attention(layer.cache, 0, qd[-1:], one, [first + tokens - 1],
                                    dataclasses.replace(params, gate=params.gate[-1:]) if gated else params)
            ctx.check()
            assert np.array_equal(tl.to_host(one)[0], outs[0][-1])
        assert np.array_equal(outs[0], outs[1])
        layer.close()


def test_partials_off_an_8_byte_boundary(hb, ctx):
    """The same for the row partials of a sequence shard."""
    import torch
    qh, kvh, d, tokens, first = 8, 2, 512, 300, 256
    q, k, v = _inputs(9, first + tokens, qh, kvh, d)
    q = q[first:]
    for rank in range(2):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 1024, shard=(hb.capi.HC_SHARD_SEQUENCE, rank, 2), prefill_chunk=1024)
        layer.append(k, v, 0)
        size = tokens * qh * (d + 2)
        outs = []
        for shift in (0, 1):
            room = torch.zeros(size + 4, device="cuda")
            partial = room[shift:shift + size]
            layer.backend.attention_prefill_partial(layer.cache, 0, tl.to_device(q), partial, tokens, first, layer.params)
            ctx.check()
            outs.append(partial.cpu().numpy())
        assert np.array_equal(outs[0], outs[1])
        layer.close()


@pytest.mark.parametrize("d, qh, kvh, window", [(64, 16, 2, 0), (256, 8, 2, 0), (512, 8, 1, 0), (64, 16, 2, 200), (128, 8, 2, 130)])
def test_prompt_partials_of_ranks_without_a_key(hb, ctx, d, qh, kvh, window):
    """The first tokens of a prompt (and on a window layer any) see no key tile of some ranks: those ranks' partials are
    the empty fold, whatever the buffer held."""
    import torch
    world, tokens = 4, 700
    q, k, v = _inputs(d + window, tokens, qh, kvh, d)
    sinks = tl.normal_bf16(np.random.default_rng(d), (qh,))
    gathered = None
    for rank in range(world):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 1024, window=window, sinks=sinks, prefill_chunk=1024,
                         shard=(hb.capi.HC_SHARD_SEQUENCE, rank, world), storage=hb.capi.HC_STORAGE_LINEAR)
        layer.append(k, v, 0)
        if gathered is None:
            gathered = torch.full((world, layer.backend.partial_bytes(layer.params, tokens) // 4), 1e30, device="cuda")
        layer.backend.attention_prefill_partial(layer.cache, 0, tl.to_device(q), gathered[rank], tokens, 0, layer.params)
        ctx.check()
        if rank + 1 < world:
            layer.close()
    out = tl.device_empty((tokens, qh, d))
    layer.backend.attention_combine(gathered, world, tokens, out, layer.params)
    ctx.check()
    want = ho.attention_rows(q, np.arange(tokens), k, v, 1 / np.sqrt(d), window, sinks=sinks)
    assert tl.within_tolerance(tl.to_host(out), want)
    layer.close()


def test_a_stack_call_that_cannot_run_queues_nothing(hb, ctx):
    """hc_attention_stack_host looks at every layer's positions before its first copy: a ring takes them, the full
    layer behind it does not."""
    import ctypes
    import torch
    capi, width, qh, kvh, d = hb.capi, 64, 2, 1, 64
    cache = hb.KVCache(ctx, [dict(q_heads=qh, kv_heads=kvh, head_dim=d, window=128, storage=capi.HC_STORAGE_RING),
                             dict(q_heads=qh, kv_heads=kvh, head_dim=d, window=0)], 256, prefill_chunk=128)
    shapes = dict(input_norm=(width,), wq=(qh * d, width), wk=(kvh * d, width), wv=(kvh * d, width), wo=(width, qh * d))
    weights = [{name: torch.ones(shape, device="cuda", dtype=torch.bfloat16) for name, shape in shapes.items()} for _ in range(2)]
    blocks = (capi.BlockWeightsStruct * 2)()
    for block, tensors, window in zip(blocks, weights, (128, 0)):
        for name, tensor in tensors.items():
            setattr(block, name, tensor.data_ptr())
        block.params = hb.AttnParams(q_heads=qh, kv_heads=kvh, head_dim=d, window=window, sm_scale=0.125,
                                     io_dtype=capi.HC_BF16).struct()
    lib = capi.load()
    tokens = 4
    workspace = torch.empty(lib.hc_attention_stack_bytes(blocks, 2, tokens, width), dtype=torch.uint8, device="cuda")
    host = np.ones((tokens, width), np.float32)

    def call(first_position, space=workspace.data_ptr(), wide=width):
        before = ctx.launch_count
        status = lib.hc_attention_stack_host(ctx.handle, cache.handle, blocks, 2, 0, host.ctypes.data, host.ctypes.data, tokens,
                                             wide, first_position, ctypes.c_float(1e-5), space, None)
        return status, ctx.launch_count - before

    assert call(254) == (capi.HC_KV_OVERFLOW, 0)
    assert call(-1) == (capi.HC_INVALID_ARGUMENT, 0)
    assert np.array_equal(host, np.ones_like(host))
    blocks[1].wo = None
    assert call(0) == (capi.HC_INVALID_ARGUMENT, 0)
    blocks[1].wo = weights[1]["wo"].data_ptr()
    status, launches = call(0)
    assert status == 0 and launches > 0
    cache.close()


@pytest.mark.parametrize("d, qh, kvh, window, chunk, cache_chunk, ring, io", [
    (64, 16, 2, 0, 128, 512, False, "bf16"), (64, 16, 2, 200, 96, 96, False, "f32"), (64, 8, 8, 128, 128, 64, True, "bf16"),
    (128, 8, 2, 0, 100, 512, False, "bf16"), (256, 16, 8, 300, 128, 128, True, "bf16"), (512, 8, 1, 0, 77, 200, False, "f32"),
    (256, 4, 4, 0, 300, 128, False, "bf16"), (96, 4, 2, 0, 60, 512, False, "bf16"),
    # (beside the ring, whose pieces bf16 queries as they come take)
    (64, 8, 8, 128, 128, 64, True, "f32"), (256, 16, 8, 300, 128, 128, True, "f32"), (96, 4, 2, 130, 64, 64, True, "f32"),
])
def test_blocks_of_a_prompt_end_with_their_chunks(hb, ctx, d, qh, kvh, window, chunk, cache_chunk, ring, io):
    """A prompt with bidirectional blocks in one call: the bits of the chunk-by-chunk calls, whichever chunk boundaries cut
    a block and however many chunks go in a launch (chunks that the cache's own do not divide included)."""
    import torch
    tokens, first = 1100, 0 if ring else 131
    rng = np.random.default_rng(d + chunk)
    q, k, v = (tl.normal_bf16(rng, (tokens, h, d)) for h in (qh, kvh, kvh))
    old = [tl.normal_bf16(rng, (max(first, 1), kvh, d)) for _ in range(2)]
    ends = np.zeros(tokens, np.int32)
    for at, n in ((3, 40), (90, 120), (250, 300), (600, 1), (700, 390)):
        ends[at:at + n] = first + at + n
    device_ends = torch.from_numpy(ends).cuda()
    storage = hb.capi.HC_STORAGE_RING if ring else hb.capi.HC_STORAGE_LINEAR
    outs, rows = [], []
    for at_once in (False, True):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 1536, window=window, io=io, prefill_chunk=cache_chunk, storage=storage)
        if first:
            layer.append(old[0], old[1], 0)
        qd, kd, vd, out = tl.to_device(q, io), tl.to_device(k, io), tl.to_device(v, io), tl.device_empty((tokens, qh, d), io)
        be, cache = layer.backend, layer.cache
        if at_once:
            be.prefill_chunks(cache, 0, qd, kd, vd, out, tokens, first, chunk, dataclasses.replace(layer.params, block_ends=device_ends))
        else:
            part = min(chunk, cache_chunk)
            edges = sorted({a for c in range(0, tokens, chunk) for a in range(c, min(c + chunk, tokens), part)})
            for a, b in zip(edges, edges[1:] + [tokens]):
                params = dataclasses.replace(layer.params, block_ends=device_ends[a:])
                be.write_key_value(cache, 0, kd[a:], vd[a:], b - a, first + a, params)
                be.attention_prefill(cache, 0, qd[a:], out[a:], b - a, first + a, params)
        ctx.check()
        outs.append(tl.to_host(out))
        layer.close()
    assert np.array_equal(outs[0], outs[1])
    edges = [a for c in range(0, tokens, chunk) for a in range(c, min(c + chunk, tokens), min(chunk, cache_chunk))] + [tokens]
    clamped = np.array([min(e, first + next(x for x in edges if x > t)) if e else 0 for t, e in enumerate(ends)])
    keys, values = (np.concatenate([o[:first], x]) for o, x in zip(old, (k, v)))
    some = np.arange(0, tokens, 7)
    want = ho.attention_rows(q[some], first + some, keys, values, 1 / np.sqrt(d), window, block_ends=clamped[some])
    assert tl.within_tolerance(outs[1][some], want, bf16_output=io == "bf16")


def test_pages_of_an_append_that_ran_out_are_not_lost(hb, ctx):
    """An append that finds too few free pages takes none: the pages it could have had serve the next one."""
    qh, kvh, d = 4, 2, 64
    q, k, v = _inputs(5, 400, qh, kvh, d)
    outs = []
    for pages in (0, 4):
        cache = hb.KVCache(ctx, [dict(q_heads=qh, kv_heads=kvh, head_dim=d, window=0)], 512, max_seqs=2, total_pages=pages)
        be = hb.AttentionBackend(ctx)
        params = hb.AttnParams(q_heads=qh, kv_heads=kvh, head_dim=d, sm_scale=0.125, io_dtype=hb.capi.HC_BF16)
        qd, kd, vd = tl.to_device(q), tl.to_device(k), tl.to_device(v)
        be.write_key_value(cache, 0, kd, vd, 200, 0, params, seq=0)              # two pages
        if pages:
            with pytest.raises(hb.HydraCudaError):
                be.write_key_value(cache, 0, kd, vd, 400, 0, params, seq=1)      # needs four
            assert cache.free_pages == 2
        out = tl.device_empty((256, qh, d))
        be.write_key_value(cache, 0, kd, vd, 256, 0, params, seq=1)
        be.attention_prefill(cache, 0, qd, out, 256, 0, params, seq=1)
        ctx.check()
        outs.append(tl.to_host(out))
        cache.close()
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("qh, kvh, tokens, first, io, gated", [
    (16, 2, 2300, 0, "bf16", False),      # Gemma's wide layer: the prompt crosses a segment of 2048 keys
    (16, 1, 500, 3900, "f32", True),      # three segments, 16 heads a group, the gated epilogue
    (4, 4, 300, 2000, "bf16", True),
    (8, 1, 40, 4200, "f32", False),       # few rows: segments as items, merged
])
def test_head_dim_512_beyond_a_segment(hb, ctx, qh, kvh, tokens, first, io, gated):
    """Whole rows that carry their second fold from segment to segment in two halves of 256 columns, and segments merged
    afterwards: against the oracle, against the rows decoded one by one, and cut at another place."""
    d, total = 512, first + tokens
    rng = np.random.default_rng(total)
    q = tl.normal_bf16(rng, (tokens, qh, d))
    k, v = (tl.normal_bf16(rng, (total, kvh, d)) for _ in range(2))
    gate = tl.normal_bf16(rng, (tokens, qh, d)) if gated else None
    sinks = tl.normal_bf16(rng, (qh,))
    layer = tl.Layer(hb, ctx, qh, kvh, d, 4608, sinks=sinks, io=io, prefill_chunk=512)
    layer.append(k, v, 0)
    prompt = layer.prefill(q, first, gate=gate)
    some = sorted({0, 1, 15, 16, 17, tokens // 2, tokens - 1} | {t for t in (2047 - first, 2048 - first, 2049 - first) if 0 <= t < tokens})
    for t in some:
        one = layer.decode(q[t:t + 1], [first + t], gate=None if gate is None else gate[t:t + 1])
        assert np.array_equal(one[0], prompt[t]), t
    cut = tokens // 3
    parts = [layer.prefill(q[a:b], first + a, gate=None if gate is None else gate[a:b]) for a, b in ((0, cut), (cut, tokens))]
    assert np.array_equal(np.concatenate(parts), prompt)
    want = ho.attention_rows(q[some], first + np.asarray(some), k, v, 1 / np.sqrt(d), 0, sinks=sinks,
                             gate=None if gate is None else gate[some])
    assert tl.within_tolerance(prompt[some], want, bf16_output=io == "bf16")
    layer.close()


@pytest.mark.parametrize("qh, kvh, d, tokens, chunk, io", [
    (64, 8, 64, 33, 512, "bf16"),       # at once, K and V behind the queries
    (64, 8, 64, 150, 128, "bf16"),      # at once, K and V ahead
    (64, 8, 64, 201, 128, "bf16"),      # two halves
    (64, 8, 64, 767, 256, "bf16"),
    (64, 8, 64, 769, 256, "bf16"),      # the schedule of six
    (64, 8, 64, 1100, 128, "f32"),      # chunk by chunk: the slots are too small for it
    (16, 2, 256, 257, 64, "f32"),
])
def test_host_prompt_schedules(hb, ctx, qh, kvh, d, tokens, chunk, io):
    """A host prompt on both sides of every line its pieces are drawn by."""
    import torch
    dtype = torch.bfloat16 if io == "bf16" else torch.float32
    host = [torch.from_numpy(a).to(dtype).pin_memory() for a in _inputs(tokens, tokens, qh, kvh, d)]
    outs, rows = [], []
    for on_host in (False, True):
        layer = tl.Layer(hb, ctx, qh, kvh, d, 1280, io=io, prefill_chunk=chunk, rope_inv_freq=ho.inverse_frequencies(d, 10000.0))
        q, k, v = host if on_host else [t.cuda() for t in host]
        out = torch.zeros((tokens, qh, d), dtype=dtype)
        out = out.pin_memory() if on_host else out.cuda()
        call = layer.backend.prefill_host if on_host else layer.backend.prefill_chunks
        call(layer.cache, 0, q, k, v, out, tokens, 0, chunk, layer.params)
        ctx.check()
        outs.append(tl.to_host(out))
        rows.append(tl.read_cache(layer.cache, 0, tokens, kvh, d))
        layer.close()
    assert np.array_equal(outs[0], outs[1])
    assert np.array_equal(rows[0][0], rows[1][0]) and np.array_equal(rows[0][1], rows[1][1])
