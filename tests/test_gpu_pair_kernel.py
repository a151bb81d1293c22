"""The CTA-pair kernel (more than 16 tokens) at the edges of its tiles against the CPU oracle: token counts
around the widths of a token tile and of several tiles, odd numbers of 128-row tiles, K of one k-block and of
partial stages, outputs whose rows are not 16-byte aligned, every epilogue that reads or writes global
memory differently."""
import numpy as np
import pytest
import torch

from oracle import woq_oracle as O
from tests.helpers import bf16_numpy, bf16_tensor, make_acts, make_int4_layer, to_device_layer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ipex_b200 import _capi

    _capi.lib()
    return _capi


def make_ctx(capi, layer, flags=0):
    qw, s, z, b = to_device_layer(layer, "cuda")
    return capi.WoqContext(qw, s, z, b, layer["n"], layer["k"], capi.DTYPE_INT4, layer["g"], capi.LOWP_BF16,
                           layout_flags=flags)


def check(y, ref):
    mx, mr = O.parity_metrics(y, ref)
    # the oracle's bf16 weights and fp32 accumulation: only the order of the sum differs
    assert mx <= O.MAX_ABS_TOL and mr < 2e-4, (mx, mr)


@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 128, 129, 160, 161, 256, 257, 320, 513])
@pytest.mark.parametrize("n,k,g,bias", [(384, 64, 64, False), (1000, 1600, 64, True), (129, 832, -1, True),
                                        (2304, 2048, 256, False)])
def test_tile_edges(capi, m, n, k, g, bias):
    layer = make_int4_layer(n, k, g, seed=n + k + m, bias=bias)
    ctx = make_ctx(capi, layer)
    x = make_acts(m, k, seed=m)
    ws = capi.Workspace(ctx.workspace_bytes(m), "cuda")
    y = bf16_numpy(ctx.linear(bf16_tensor(x, "cuda"), workspace=ws))
    ws.status()
    check(y, O.woq_linear_bf16(x, layer["qw"], layer["s16"], layer["z"], layer["bias"], O.WOQ_DTYPE_INT4, g))


@pytest.mark.parametrize("m", [40, 300])
@pytest.mark.parametrize("fusion,n_others", [(O.FUSE_ADD, 1), (O.FUSE_ADD_ADD, 2), (O.FUSE_MUL, 1), (O.FUSE_GELU_ERF, 0)])
@pytest.mark.parametrize("n", [200, 331])
def test_epilogues(capi, m, fusion, n_others, n):
    layer = make_int4_layer(n, 512, 128, seed=n + fusion, std=0.05, bias=True)
    ctx = make_ctx(capi, layer)
    x = make_acts(m, 512, seed=m)
    others = [make_acts(m, n, seed=60 + i) for i in range(n_others)]
    y = bf16_numpy(ctx.linear(bf16_tensor(x, "cuda"), fusion, [bf16_tensor(o, "cuda") for o in others]))
    ref = O.woq_linear_bf16(x, layer["qw"], layer["s16"], layer["z"], layer["bias"], O.WOQ_DTYPE_INT4, 128, fusion, others)
    mx, mr = O.parity_metrics(y, ref)
    assert mx <= O.MAX_ABS_TOL and mr <= O.MEAN_REL_TOL, (mx, mr)


@pytest.mark.parametrize("m", [48, 290])
def test_large_zero_points_take_the_shifting_dequantiser(capi, m):
    """Zero points above 15 (or scales outside the in-place range) select the other dequantiser."""
    layer = make_int4_layer(320, 768, 128, seed=5)
    layer["z"] = layer["z"] + np.float32(40)
    ctx = make_ctx(capi, layer)
    x = make_acts(m, 768, seed=m)
    y = bf16_numpy(ctx.linear(bf16_tensor(x, "cuda")))
    check(y, O.woq_linear_bf16(x, layer["qw"], layer["s16"], layer["z"], None, O.WOQ_DTYPE_INT4, 128))
