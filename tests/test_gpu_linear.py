"""hc_linear: the Q/K/V/O projections on the tensor cores against the oracle's double-precision
matVec, through the C ABI.  Shapes are the configurations' own (GPT-OSS hidden 2880 with its
64 x 64 query and 8 x 64 key/value widths, the output projection back to 2880, a Qwen-like
2x-tall query/gate projection) plus ragged edges: one token, a token count and an output width that
are not multiples of the tile."""
import numpy as np
import pytest

from oracle import hydra_oracle as ho
from tests import hydra_testlib as tl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens, n_in, n_out, with_bias, out_bf16", [
    (512, 2880, 4096, True, False),      # q_proj of a prefill chunk
    (1, 2880, 512, True, False),         # k_proj of one decode token
    (77, 4096, 2880, True, True),        # o_proj, ragged token count, 2880 = 11.25 column tiles
    (300, 2048, 8192, False, True),      # 2x-tall q_proj with the interleaved gate, no bias
    (130, 64, 40, False, False),         # one K step; output narrower than a tile
])
def test_linear_matches_the_oracle(tokens, n_in, n_out, with_bias, out_bf16):
    import hydra_b200 as hb
    ctx = hb.Context(0)
    backend = hb.AttentionBackend(ctx)
    rng = np.random.default_rng(tokens * 7 + n_out)
    x = tl.normal_bf16(rng, (tokens, n_in))
    w = ho.bf16_round(rng.normal(0.0, 0.02, (n_out, n_in)))
    bias = ho.bf16_round(rng.normal(0.0, 0.5, (n_out,))) if with_bias else None
    want = ho.linear(x, w, bias)
    xd, wd = tl.to_device(x), tl.to_device(w)
    bd = tl.to_device(bias) if with_bias else None
    out = tl.device_empty((tokens, n_out)) if out_bf16 else tl.device_empty((tokens, n_out), dtype="f32")
    dtype = hb.capi.HC_BF16 if out_bf16 else hb.capi.HC_F32
    for _ in range(2):                   # twice: the second call reuses the tensor-memory accumulators
        backend.linear(xd, wd, bd, out, tokens, n_in, n_out, y_dtype=dtype)
    ctx.check()
    got = tl.to_host(out)
    assert got.shape == want.shape
    # fp32 accumulation of bf16 products: far inside the parity bound; bf16 outputs add their rounding
    scale = max(1.0, float(np.abs(want).max()))
    bound = 1e-3 * scale + ((2.0 ** -8) * np.abs(want) if out_bf16 else 0.0)
    assert np.all(np.abs(got - want) <= bound), float(np.abs(got - want).max())
    tl.record_margin(f"linear {tokens}x{n_in}->{n_out}", got, want)
    ctx.close()


def test_linear_rows_do_not_depend_on_the_batch():
    """A token's projection is the same bits whether it is projected alone (the narrow, many-staged
    shape of the kernel, for decode), in a chunk of 100, or inside a prompt of 700 (the wide shape): the
    invariant the attention kernels keep between prefill and decode, kept by the projections too."""
    import hydra_b200 as hb
    ctx = hb.Context(0)
    backend = hb.AttentionBackend(ctx)
    rng = np.random.default_rng(3)
    tokens, n_in, n_out = 700, 2880, 1536
    x = tl.to_device(tl.normal_bf16(rng, (tokens, n_in)))
    w = tl.to_device(ho.bf16_round(rng.normal(0.0, 0.02, (n_out, n_in))))
    b = tl.to_device(ho.bf16_round(rng.normal(0.0, 0.5, (n_out,))))
    whole = tl.device_empty((tokens, n_out), dtype="f32")
    backend.linear(x, w, b, whole, tokens, n_in, n_out)
    chunk = tl.device_empty((100, n_out), dtype="f32")
    backend.linear(x[300:], w, b, chunk, 100, n_in, n_out)
    one = tl.device_empty((1, n_out), dtype="f32")
    backend.linear(x[333:], w, b, one, 1, n_in, n_out)
    ctx.check()
    whole, chunk, one = tl.to_host(whole), tl.to_host(chunk), tl.to_host(one)
    assert np.array_equal(whole[300:400], chunk)
    assert np.array_equal(whole[333], one[0])
    ctx.close()


@pytest.mark.parametrize("tokens", [1, 77, 700])
def test_linear_group_equals_the_separate_calls(tokens):
    """q_proj, k_proj and v_proj of the same x in one launch: the bits of three hc_linear calls, with
    widths that are not whole tiles and one projection without a bias."""
    import hydra_b200 as hb
    ctx = hb.Context(0)
    backend = hb.AttentionBackend(ctx)
    rng = np.random.default_rng(5)
    n_in, widths = 2880, (4096, 512, 520)
    x = tl.to_device(tl.normal_bf16(rng, (tokens, n_in)))
    weights = [tl.to_device(ho.bf16_round(rng.normal(0.0, 0.02, (n, n_in)))) for n in widths]
    biases = [tl.to_device(ho.bf16_round(rng.normal(0.0, 0.5, (n,)))) for n in widths]
    biases[1] = None
    for dtype, code in (("bf16", hb.capi.HC_BF16), ("f32", hb.capi.HC_F32)):
        separate = [tl.device_empty((tokens, n), dtype=dtype) for n in widths]
        grouped = [tl.device_empty((tokens, n), dtype=dtype) for n in widths]
        for w, b, y in zip(weights, biases, separate):
            backend.linear(x, w, b, y, tokens, n_in, w.shape[0], y_dtype=code)
        before = ctx.launch_count
        backend.linear_group(x, weights, biases, grouped, tokens, n_in, y_dtype=code)
        assert ctx.launch_count - before == 1
        ctx.check()
        for a, b in zip(separate, grouped):
            assert np.array_equal(tl.to_host(a), tl.to_host(b))
    with pytest.raises(hb.HydraCudaError):
        backend.linear_group(x, weights * 2, biases * 2, grouped * 2, tokens, n_in)
    ctx.close()


def test_linear_refuses_what_it_cannot_tile():
    import hydra_b200 as hb
    ctx = hb.Context(0)
    backend = hb.AttentionBackend(ctx)
    x = tl.device_empty((4, 72))
    w = tl.device_empty((16, 72))
    y = tl.device_empty((4, 16), dtype="f32")
    with pytest.raises(hb.DimensionMismatch):
        backend.linear(x, w, None, y, 4, 72, 16)
    ctx.close()


@pytest.mark.parametrize("tokens, width, outs", [
    (4096, 64, (2880,)),               # two rounds of wide tiles and one of halves, an odd half of 64 columns
    (3900, 128, (2880,)),              # a ragged last row tile
    (2048, 64, (4096, 512, 512)),      # three jobs; the cut lies in the first
    (4096, 64, (1000, 2880, 130)),     # last columns of one and two halves
    (4096, 64, (4096, 513)),           # a last half of one column
    (9000, 64, (100, 90)),             # no wide tile at all
    (4096, 64, (904,)),                # a last tile of 136 columns: wide, with zeros
    (4096, 64, (2200, 385, 511)),      # the same behind others, 152, 129 and 255 columns
    (4096, 64, (4680, 384)),           # a wide tile of 72 columns more than half among those cut in halves
])
def test_linear_tiles_of_two_widths(tokens, width, outs):
    """Sums of 64 or 128 products in fp32 against float64: 128 roundings of 2^-24 of sums below 40 stay under 4e-4.  With
    biases and residuals, which have a half tile's own columns: two roundings more of values below 50, 2^-24 each; in bf16
    half a step of 8 significant bits."""
    import torch
    import hydra_b200 as hb
    ctx = hb.Context(0)
    gen = torch.Generator(device="cuda").manual_seed(tokens + width)
    x = torch.randn(tokens, width, device="cuda", generator=gen).to(torch.bfloat16)
    w = [torch.randn(n, width, device="cuda", generator=gen).to(torch.bfloat16) for n in outs]
    y = [torch.full((tokens, n), 7.0, device="cuda") for n in outs]
    hb.AttentionBackend(ctx).linear_group(x, w, [None] * len(outs), y, tokens, width, y_dtype=hb.capi.HC_F32)
    ctx.check()
    for got, weight in zip(y, w):
        assert float((got.double() - x.double() @ weight.double().T).abs().max()) < 4e-4
    b = [torch.randn(n, device="cuda", generator=gen).to(torch.bfloat16) for n in outs]
    half = [torch.full((tokens, n), 7.0, device="cuda", dtype=torch.bfloat16) for n in outs]
    hb.AttentionBackend(ctx).linear_group(x, w, b, half, tokens, width, y_dtype=hb.capi.HC_BF16)
    ctx.check()
    for got, weight, bias in zip(half, w, b):
        want = x.double() @ weight.double().T + bias.double()
        assert bool(((got.double() - want).abs() <= 4.1e-4 + 2.0 ** -8 * want.abs()).all())
    for weight, bias in zip(w, b):
        residual = torch.randn(tokens, weight.shape[0], device="cuda", generator=gen)
        got = torch.full_like(residual, 7.0)
        hb.AttentionBackend(ctx).linear(x, weight, bias, got, tokens, width, weight.shape[0], residual=residual)
        ctx.check()
        assert float((got.double() - x.double() @ weight.double().T - bias.double() - residual.double()).abs().max()) < 4.1e-4
    ctx.close()


@pytest.mark.parametrize("outs", [(2000,), (2880,), (4600,), (4096, 512, 512), (6000,), (9600,), (41, 2, 130)])
@pytest.mark.parametrize("residual", [False, True])
def test_linear_of_few_tokens_at_the_edges_of_its_row_tiles(outs, residual):
    """64 and 128 rows an MMA and every width of column tile: the bits of the same rows in a call of 140 tokens, which
    the other kernel computes, and the fp32 sums of 192 products of float64's (192 roundings of 2^-24 of sums below 60)."""
    import torch
    import hydra_b200 as hb
    ctx = hb.Context(0)
    backend = hb.AttentionBackend(ctx)
    gen = torch.Generator(device="cuda").manual_seed(sum(outs))
    x = torch.randn(140, 192, device="cuda", generator=gen).to(torch.bfloat16)
    w = [torch.randn(n, 192, device="cuda", generator=gen).to(torch.bfloat16) for n in outs]
    b = [torch.randn(n, device="cuda", generator=gen).to(torch.bfloat16) for n in outs]
    res = [torch.randn(140, n, device="cuda", generator=gen) for n in outs]

    def call(tokens):
        y = [torch.full((tokens + 1, n), 7.0, device="cuda") for n in outs]
        if residual:
            for weight, bias, r, out in zip(w, b, res, y):
                backend.linear(x, weight, bias, out, tokens, 192, weight.shape[0], residual=r)
        else:
            backend.linear_group(x, w, b, y, tokens, 192, y_dtype=hb.capi.HC_F32)
        ctx.check()
        assert all(bool((out[tokens] == 7.0).all()) for out in y)
        return [out[:tokens] for out in y]

    whole = call(140)
    for got, weight, bias, r in zip(whole, w, b, res):
        want = x.double() @ weight.double().T + bias.double() + (r.double() if residual else 0.0)
        assert float((got.double() - want).abs().max()) < 1e-3
    for tokens in (1, 8, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 96, 127, 128, 129):
        for got, want in zip(call(tokens), whole):
            assert torch.equal(got, want[:tokens])
    ctx.close()
