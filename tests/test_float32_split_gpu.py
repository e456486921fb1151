"""The float32 product through three bfloat16 parts on the tensor cores: against 64 bits and the chain of FMA, whatever rows stand
beside a row, and with values that are not finite."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(x, w):
    from kv_cache_optimization_for_llm_b200 import ops
    out = torch.empty((x.shape[0], w.shape[0]), device="cuda")
    rc = ops.lib("gemm_f32").kvb_sgemm_nt(ops._p(x), x.stride(0), ops._p(w), w.stride(0), ops._p(out), w.shape[0], x.shape[0], w.shape[0],
                                          x.shape[1], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    return out


def _draw(M, N, K, seed, spread=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, w = (torch.randn(s, generator=g, device="cuda") for s in ((M, K), (N, K)))
    if spread:      # magnitudes over many binades, all of one sign: rounding errors that do not cancel would show
        x, w = (t.abs() * torch.exp2(torch.randint(-20, 20, t.shape, generator=g, device="cuda").float()) for t in (x, w))
    return x, w


# rows: 1, the edges of 16, of a block's 176 and of its halves; features: below, at and above 128; k: the tail of 64 and of 8, cut over
# 1, 2 and 4 blocks
@pytest.mark.parametrize("M,N,K", [(1, 128, 1024), (2, 1, 1028), (15, 130, 2048), (16, 2048, 2048), (17, 3072, 2048), (97, 127, 1028),
                                   (175, 256, 1024), (176, 129, 8192), (177, 2048, 8188), (353, 1000, 1088), (33, 19000, 1152)])
@pytest.mark.parametrize("spread", [False, True])
def test_split_product_is_as_close_as_a_chain_of_fma(M, N, K, spread):
    from kv_cache_optimization_for_llm_b200 import ops
    x, w = _draw(M, N, K, M + N + K, spread)
    assert ops.float32_split_ok(w)
    before = ops.choices["sgemm_nt_split"]
    out, ref = ops.linear(x, w), x.double() @ w.double().T
    assert ops.choices["sgemm_nt_split"] == before + 1
    scale = x.double().abs() @ w.double().abs().T
    err, chain = ((t.double() - ref).norm() / ref.norm() for t in (out, _chain(x, w)))
    assert err <= 1.05 * chain + 2.0 ** -25, (float(err), float(chain))
    # pieces of 64 k are cut to 24 bits at each of 24 products, then added with one rounding each
    bound = 24 * 2.0 ** -23 + (-(-K // 64) + 8) * 2.0 ** -24
    assert bool(((out.double() - ref).abs() <= bound * scale).all())


@pytest.mark.parametrize("M,N,K", [(200, 2048, 2048), (50, 300, 1024), (33, 16384 + 128, 1024)])
def test_a_row_is_the_same_alone_and_beside_others_and_at_any_alignment(M, N, K):
    from kv_cache_optimization_for_llm_b200 import ops
    x, w = _draw(M, N, K, 7)
    full = ops.linear(x, w)
    for rows in (slice(0, 1), slice(M - 1, M), slice(3, 20), slice(0, M // 2)):
        assert torch.equal(ops.linear(x[rows].contiguous(), w), full[rows])
    odd = torch.cat([x, x[:, :1]], 1)[:, :K]
    assert odd.stride(0) % 4 and torch.equal(ops.linear(odd, w), full)


def test_values_that_are_not_finite_come_out_as_from_the_chain():
    from kv_cache_optimization_for_llm_b200 import ops
    x, w = _draw(40, 384, 1024, 3)
    inf = float("inf")
    x[3, 5], x[4, 1000], x[5, 0], x[6, 17] = inf, -inf, float("nan"), 3.4e38      # the last rounds to infinity in bfloat16
    w[17, 900], w[200, 5], w[201, 5], w[300, 17] = inf, 0.0, -inf, 1e-3
    x[7, 900], x[8, 900] = 0.0, -1.0
    x[9], w[5] = 1e30, 1e30                                                       # the sum overflows
    out, ref = ops.linear(x, w), _chain(x, w)
    bad = ~torch.isfinite(ref)
    assert int(bad.sum()) > 1000 and torch.equal(torch.isfinite(out), ~bad)
    assert torch.equal(torch.nan_to_num(out[bad], nan=1.0), torch.nan_to_num(ref[bad], nan=1.0))
    # finite ones: a chain of K fmaf is off by at most K * 2^-24 of the sum of magnitudes, and the parts by less
    scale = torch.nan_to_num(x.double().abs() @ w.double().abs().T, nan=float("inf"))
    assert bool(((out.double() - ref.double()).abs() <= 2 * 1024 * 2.0 ** -24 * scale)[~bad].all())


@pytest.mark.parametrize("M,N,K", [(3, 256, 1024), (50, 200, 2048), (177, 2048, 1028)])
@pytest.mark.parametrize("binade", [-95, -108, -112, -118, -124])
@pytest.mark.parametrize("side", ["rows", "weights", "some rows"])
def test_operands_whose_last_parts_bfloat16_cannot_hold(M, N, K, binade, side):
    """Below 2^-110 the third part of an operand has fewer than eight bits: results that are made of such operands are as close as the
    chain's, and rows beside them are what they are without them."""
    from kv_cache_optimization_for_llm_b200 import ops
    x, w = _draw(M, N, K, M + N + K)
    plain = ops.linear(x, w)
    tiny = torch.zeros(M, dtype=torch.bool, device="cuda")
    tiny[::2 if side == "some rows" else 1] = True
    if side == "weights":
        w = w * 2.0 ** binade
    else:
        x = torch.where(tiny[:, None], x * 2.0 ** binade, x)
    out, ref, by_chain = ops.linear(x, w), x.double() @ w.double().T, _chain(x, w)
    err, chain = ((t.double() - ref)[tiny].norm() / ref[tiny].norm() for t in (out, by_chain))
    assert err <= 1.05 * chain + 2.0 ** -25, (float(err), float(chain))
    assert torch.equal(out[~tiny], plain[~tiny])


def test_products_that_the_parts_do_not_take_go_to_the_chain():
    from kv_cache_optimization_for_llm_b200 import ops
    x, w = _draw(20, 64, 1032, 1)
    for v in (w[:, :1020], w[:, 1:1029], w[:, :1030]):      # short, off 16 bytes, no multiple of four
        assert not ops.float32_split_ok(v)
        before = ops.choices["sgemm_nt_split"]
        assert torch.equal(ops.linear(x[:, :v.shape[1]], v), _chain(x[:, :v.shape[1]], v))
        assert ops.choices["sgemm_nt_split"] == before
