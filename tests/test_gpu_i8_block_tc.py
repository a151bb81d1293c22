"""The tcgen05 kernel of INT4 weights with INT8 compute (symmetric codes, K blocks of 128) at the edges of its
tiles: token counts around the three tile widths, odd numbers of K blocks, row tiles that do not fill, groups of
one, two and all blocks.  Block accumulators and codes bit-exact; outputs differ in the order of the fp32 sum
over K blocks only."""
import numpy as np
import pytest
import torch

from oracle import woq_oracle as O
from tests.helpers import bf16_numpy, bf16_tensor, make_acts

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ipex_b200 import _capi

    _capi.lib()
    return _capi


@pytest.mark.parametrize("m", [1, 16, 31, 33, 64, 65, 128, 129, 200, 290])
@pytest.mark.parametrize("n,k,g,mode", [(128, 128, 128, 7), (331, 640, 128, 7), (200, 1536, 256, 4), (1152, 2304, -1, 6)])
def test_tile_edges(capi, m, n, k, g, mode):
    rng = np.random.default_rng(n + k)
    w = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    if g > 0:
        qw, s, z = O.quantize_per_block(w, O.WOQ_DTYPE_INT4, g, False)
    else:
        qw, s, z = O.quantize_per_channel(w, O.WOQ_DTYPE_INT4, False)
        s, z = s[:, None], z[:, None]
    bias = np.linspace(-1, 1, n).astype(np.float32) if n % 2 else None
    t = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ctx = capi.WoqContext(t(qw), t(s), t(z), t(bias), n, k, O.WOQ_DTYPE_INT4, g, capi.LOWP_INT8, act_quant_mode=mode)
    assert ctx.route() == capi.ROUTE_INT8_BLOCK
    assert np.array_equal(ctx.unpack().cpu().numpy(), qw)
    x = O.rne_bf16(make_acts(m, k, seed=m))
    y_ref, blocks, qa_ref, sa_ref, _ = O.woq_linear_int8_blocks(x, qw, O.WOQ_DTYPE_INT4, s, z, bias, g, mode,
                                                                return_blocks=True)
    qa, sa, _, acc = ctx.int8_block_internals(bf16_tensor(x, "cuda"))
    np.testing.assert_array_equal(qa.cpu().numpy(), qa_ref.view(np.uint8))
    np.testing.assert_array_equal(sa.cpu().numpy(), sa_ref)
    np.testing.assert_array_equal(acc.cpu().numpy(), blocks)
    y = bf16_numpy(ctx.linear(bf16_tensor(x, "cuda")))
    ctx.workspace(m).status()
    mx, mr = O.parity_metrics(y, y_ref)
    assert mx <= O.MAX_ABS_TOL and mr < 2e-4, (mx, mr)


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("n,k,g,mode", [(331, 640, 128, 7), (331, 1152, 128, 7), (200, 4096, 256, 4), (137, 8320, -1, 7)])
def test_few_tokens(capi, m, n, k, g, mode):
    """Both sides of the line between the kernel of few tokens and the tcgen05 kernel, on one layout; numbers of K
    blocks that are no multiple of the eight its warps take at a time, rows that fill no tile."""
    test_tile_edges(capi, m, n, k, g, mode)


@pytest.mark.parametrize("m", [8, 9])
def test_few_tokens_on_large_weights(capi, m):
    """9 tokens on more than 64 MB of weights are the tcgen05 kernel's; the results of the same rows agree."""
    n, k = 28800, 4736
    gen = torch.Generator(device="cuda").manual_seed(0)
    qw = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    s = torch.rand((n, k // 128), device="cuda", generator=gen) * 0.004 + 0.001
    z = torch.randint(0, 128, (n, k // 128), device="cuda", generator=gen).float()
    make = lambda rows: capi.WoqContext(qw[rows].contiguous(), s[rows].contiguous(), z[rows].contiguous(), None,  # noqa: E731
                                        len(range(n)[rows]), k, O.WOQ_DTYPE_INT4, 128, capi.LOWP_INT8, act_quant_mode=7)
    whole, part = make(slice(0, n)), make(slice(n - 300, n))
    x = bf16_tensor(make_acts(m, k, seed=m), "cuda")
    assert torch.equal(whole.int8_block_internals(x)[3][:, :, n - 300:], part.int8_block_internals(x)[3])
    mx, mr = O.parity_metrics(bf16_numpy(whole.linear(x))[:, n - 300:], bf16_numpy(part.linear(x)))
    # the same block accumulators; another order of the fp32 sum over 37 blocks
    assert mx <= O.MAX_ABS_TOL and mr < 2e-4, (mx, mr)


@pytest.mark.parametrize("m", [20, 31, 33, 65, 129, 290])
@pytest.mark.parametrize("n,k,g", [(331, 640, 128), (200, 1536, 256), (1152, 2304, -1), (129, 4224, 128)])
def test_both_cuts(capi, m, n, k, g):
    """Whole tiles, and shares of the K blocks whose tiles are summed through the workspace: the same accumulators,
    outputs in another order of the fp32 sum; the counters are left at zero."""
    rng = np.random.default_rng(n + k + m)
    w = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    if g > 0:
        qw, s, z = O.quantize_per_block(w, O.WOQ_DTYPE_INT4, g, False)
    else:
        qw, s, z = O.quantize_per_channel(w, O.WOQ_DTYPE_INT4, False)
        s, z = s[:, None], z[:, None]
    bias = np.linspace(-1, 1, n).astype(np.float32) if n % 2 else None
    t = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    x = O.rne_bf16(make_acts(m, k, seed=m))
    resid = make_acts(m, n, seed=m + 1)
    xb, rb = bf16_tensor(x, "cuda"), bf16_tensor(resid, "cuda")
    y_ref, blocks, *_ = O.woq_linear_int8_blocks(x, qw, O.WOQ_DTYPE_INT4, s, z, bias, g, 7, return_blocks=True)
    y_ref = O.rne_bf16(y_ref + resid)
    for cut in (capi.PAIR_CUT_SHARES, capi.PAIR_CUT_WHOLE):
        ctx = capi.WoqContext(t(qw), t(s), t(z), t(bias), n, k, O.WOQ_DTYPE_INT4, g, capi.LOWP_INT8, act_quant_mode=7,
                              kernel_hint=capi.HINT_PAIR(0, cut))
        np.testing.assert_array_equal(ctx.int8_block_internals(xb)[3].cpu().numpy(), blocks)
        first = ctx.linear(xb, capi.FUSE_ADD, [rb])
        for _ in range(3):
            assert torch.equal(ctx.linear(xb, capi.FUSE_ADD, [rb]), first)
        ctx.workspace(m).status()
        mx, mr = O.parity_metrics(bf16_numpy(first), y_ref)
        # the operand's rounding after a sum that may round to the neighbouring bf16 value
        assert mx <= O.MAX_ABS_TOL and mr < 4e-4, (cut, mx, mr)


@pytest.mark.parametrize("m", [9, 70])
def test_zero_points_out_of_range_stay_on_the_other_kernels(capi, m):
    n, k = 96, 512
    w = (np.random.default_rng(1).standard_normal((n, k)) * 0.02).astype(np.float32)
    qw, s, z = O.quantize_per_block(w, O.WOQ_DTYPE_INT4, 128, False)
    z = z - np.float32(40)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ctx = capi.WoqContext(t(qw), t(s), t(z), None, n, k, O.WOQ_DTYPE_INT4, 128, capi.LOWP_INT8, act_quant_mode=7)
    x = O.rne_bf16(make_acts(m, k, seed=m))
    y = bf16_numpy(ctx.linear(bf16_tensor(x, "cuda")))
    mx, mr = O.parity_metrics(y, O.woq_linear_int8_blocks(x, qw, O.WOQ_DTYPE_INT4, s, z, None, 128, 7))
    assert mx <= O.MAX_ABS_TOL and mr <= O.MEAN_REL_TOL, (mx, mr)
