"""INT8 and NF4 weights with bf16 activations and compute: the CTA-pair kernel on the row layout against the
oracle and against the general kernel on the same context, at the edges of its tiles and for every form of
scale and zero point that selects another dequantiser or keeps the layer on the plain layout."""
import numpy as np
import pytest
import torch

from oracle import woq_oracle as O
from tests.helpers import make_acts

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ipex_b200 import _capi

    _capi.lib()
    return _capi


def make_layer(form, n, k, g, seed):
    rng = np.random.default_rng(seed)
    dt = O.WOQ_DTYPE_NF4 if form == "nf4" else O.WOQ_DTYPE_INT8
    w = (rng.standard_normal((n, k)) * (20.0 if form == "int8_large" else 0.02) + (0.01 if dt == O.WOQ_DTYPE_INT8 else 0)).astype(np.float32)
    if g > 0:
        qw, s, z = O.quantize_per_block(w, dt, g, form == "nf4")
    else:
        qw, s, z = O.quantize_per_channel(w, dt, form == "nf4")
        s, z = s[:, None], None if z is None else z[:, None]
    if form == "int8_fraction":
        z = z + np.float32(0.5)
    return dict(dt=dt, qw=qw, s=s.astype(np.float32), z=z, n=n, k=k, g=g)


def make_ctx(capi, L, bias=None):
    t = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return capi.WoqContext(t(L["qw"]), t(L["s"]), t(L["z"]), t(bias), L["n"], L["k"], L["dt"], L["g"], capi.LOWP_NONE)


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).bfloat16().cuda()


def general(ctx, x, *args):
    """The same call with activation rows that no TMA copy can start at: the general kernel takes it."""
    wide = torch.zeros((x.shape[0], x.shape[1] + 1), dtype=x.dtype, device=x.device)
    wide[:, :-1] = x
    return ctx.linear_any(wide[:, :-1], *args)


@pytest.mark.parametrize("form", ["int8", "int8_large", "int8_fraction", "nf4"])
@pytest.mark.parametrize("n,k,g", [(128, 64, -1), (200, 832, 64), (331, 1600, -1), (2304, 1024, 256)])
@pytest.mark.parametrize("m", [1, 16, 33, 129, 257, 300])
def test_tile_edges(capi, form, n, k, g, m):
    L = make_layer(form, n, k, g, seed=n + k)
    bias = np.linspace(-1, 1, n).astype(np.float32) if n % 2 else None
    ctx = make_ctx(capi, L, bias)
    assert np.array_equal(ctx.unpack().cpu().numpy().view(np.uint8), np.ascontiguousarray(L["qw"]).view(np.uint8))
    xb = bf16(make_acts(m, k, seed=m))
    ws = ctx.workspace(m)
    y = ctx.linear_any(xb)
    ws.status()
    ref = O.woq_linear_any(xb.float().cpu().numpy(), L["qw"], L["s"], L["z"], bias, L["dt"], g, "bf16", "bf16")
    mx, mr = O.parity_metrics(y.float().cpu().numpy(), ref)
    # the same bf16 weights and fp32 accumulation: only the order of the sum differs
    assert mx <= O.MAX_ABS_TOL and mr < 2e-4, (mx, mr)
    mx, mr = O.parity_metrics(general(ctx, xb).float().cpu().numpy(), ref)
    assert mx <= O.MAX_ABS_TOL and mr < 2e-4, (mx, mr)


@pytest.mark.parametrize("m", [5, 70])
@pytest.mark.parametrize("fusion,n_others", [(O.FUSE_ADD, 1), (O.FUSE_ADD_ADD, 2), (O.FUSE_MUL, 1), (O.FUSE_SILU, 0),
                                             (O.FUSE_GELU_TANH, 0)])
def test_epilogues(capi, m, fusion, n_others):
    n, k = 331, 512
    L = make_layer("int8", n, k, 128, seed=fusion)
    ctx = make_ctx(capi, L)
    xb = bf16(make_acts(m, k, seed=m))
    others = [bf16(make_acts(m, n, seed=60 + i)) for i in range(n_others)]
    y, y_gen = ctx.linear_any(xb, fusion, others), general(ctx, xb, fusion, others)
    mx, mr = O.parity_metrics(y.float().cpu().numpy(), y_gen.float().cpu().numpy())
    # one bf16 rounding of the sum, then the same operations: neighbouring bf16 values at most
    assert mx <= O.MAX_ABS_TOL and mr <= O.MEAN_REL_TOL, (mx, mr)


def test_other_activation_types_and_small_workspace(capi):
    """fp16 / fp32 activations under lowp NONE read the row layout through the general kernel; so does a call
    whose workspace has only the header."""
    L = make_layer("int8", 192, 320, -1, seed=3)
    ctx = make_ctx(capi, L)
    x = make_acts(9, 320, seed=4)
    for io, dt in (("fp16", torch.float16), ("fp32", torch.float32)):
        xt = torch.from_numpy(x).to(dt).cuda()
        y = ctx.linear_any(xt).float().cpu().numpy()
        ref = O.woq_linear_any(xt.float().cpu().numpy(), L["qw"], L["s"], L["z"], None, L["dt"], -1, io, io)
        mx, mr = O.parity_metrics(y, ref)
        assert mx <= O.MAX_ABS_TOL and mr <= O.MEAN_REL_TOL, (mx, mr)
    xb = bf16(x)
    y = ctx.linear_any(xb)
    ctx._ws = capi.Workspace(capi.lib().woq_b200_workspace_header_bytes(), "cuda")
    out = torch.empty_like(y)
    capi._check(capi.lib().woq_b200_linear_any(ctx._h, xb.data_ptr(), 3, 9, xb.stride(0), 0, None, 0, out.data_ptr(),
                                               out.stride(0), ctx._ws.buf.data_ptr(), ctx._ws.nbytes, capi._stream()))
    assert torch.equal(out, general(ctx, xb))
