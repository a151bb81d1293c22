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
