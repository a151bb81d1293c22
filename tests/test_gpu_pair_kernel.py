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


# ---- every way the launches are cut, at the edges ---------------------------------------------------------------
# Which one a call takes follows an estimate of its time; on small shapes that is never the one that shares tiles
# through the workspace.  Here each is asked for.
KINDS = {"int4": (O.WOQ_DTYPE_INT4, 128), "int4_shifting": (O.WOQ_DTYPE_INT4, 128), "int8": (O.WOQ_DTYPE_INT8, -1),
         "int8_large": (O.WOQ_DTYPE_INT8, 64), "nf4": (O.WOQ_DTYPE_NF4, 64)}
_layers = {}


def cut_case(kind, n, k, m):
    """One layer, its activations and extra operand, and the oracle's result (kept for the cuts of a shape)."""
    key = (kind, n, k, m)
    if key not in _layers:
        _layers.clear()
        dt, g = KINDS[kind]
        g = g if g > 0 and k % g == 0 else -1
        rng = np.random.default_rng(n + k + m)
        w = (rng.standard_normal((n, k)) * (20.0 if kind == "int8_large" else 0.02)).astype(np.float32)
        sym = dt == O.WOQ_DTYPE_NF4
        if g > 0:
            qw, s, z = O.quantize_per_block(w, dt, g, sym)
        else:
            qw, s, z = O.quantize_per_channel(w, dt, sym)
            s, z = s[:, None], None if z is None else z[:, None]
        if kind == "int4_shifting":
            z = z + np.float32(40)
        s = s.astype(np.float16) if dt == O.WOQ_DTYPE_INT4 else s.astype(np.float32)
        bias = (rng.standard_normal(n) * 0.1).astype(np.float32) if n % 2 else None
        x, other = make_acts(m, k, seed=m), make_acts(m, n, seed=m + 1)
        if dt == O.WOQ_DTYPE_INT4:
            ref = O.woq_linear_bf16(x, qw, s, z, bias, dt, g, O.FUSE_ADD, [other])
        else:
            ref = O.woq_linear_any(x, qw, s, z, bias, dt, g, "bf16", "bf16", O.FUSE_ADD, [other])
        _layers[key] = (dt, g, qw, s, z, bias, x, other, ref)
    return _layers[key]


def cut_ctx(capi, case, n, k, columns, cut):
    dt, g, qw, s, z, bias = case[:6]
    t = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return capi.WoqContext(t(qw), t(s), t(z), t(bias), n, k, dt, g, capi.LOWP_BF16,
                           kernel_hint=capi.HINT_PAIR(columns, cut))


# remainders of tokens, rows and k-blocks, outputs whose rows are not 16-byte aligned; tiles cut among many pairs;
# several tiles for each pair (153 of 256 rows x 32 tokens), alone and cut
CUT_SHAPES = [(331, 1600, 290, 32), (331, 1600, 161, 160), (129, 832, 33, 64), (1000, 1600, 65, 96),
              (2304, 2048, 513, 32), (2304, 2048, 513, 256), (520, 4096, 97, 128)]


@pytest.mark.parametrize("n,k,m,columns", CUT_SHAPES)
@pytest.mark.parametrize("kind", list(KINDS))
def test_every_cut(capi, kind, n, k, m, columns):
    case = cut_case(kind, n, k, m)
    x, other, ref = case[6:]
    xb, ob = bf16_tensor(x, "cuda"), bf16_tensor(other, "cuda")
    ws = capi.Workspace(cut_ctx(capi, case, n, k, 0, 0).workspace_bytes(m), "cuda")
    for cut in (capi.PAIR_CUT_SHARES, capi.PAIR_CUT_WHOLE, capi.PAIR_CUT_SPLIT2, capi.PAIR_CUT_SPLIT3, capi.PAIR_CUT_SPLIT4):
        if cut > 2 and k // 64 < 4 * (cut - 1):
            with pytest.raises(capi.WoqError, match="WOQ_B200_HINT_PAIR"):
                cut_ctx(capi, case, n, k, columns, cut).linear(xb, capi.FUSE_ADD, [ob], workspace=ws)
            continue
        ctx = cut_ctx(capi, case, n, k, columns, cut)
        out = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
        for _ in range(3):  # the counters of shared tiles are left at zero
            y = ctx.linear(xb, capi.FUSE_ADD, [ob], out=out[:m], workspace=ws)
            mx, mr = O.parity_metrics(bf16_numpy(y), ref)
            # weights of N(0, 20) make sums of which the extra operand is a rounding error: one more bf16 rounding
            assert mx <= O.MAX_ABS_TOL and mr < 4e-4, (cut, mx, mr)
        ws.status()
        assert bool((out[m] == 7.0).all())


@pytest.mark.parametrize("kind", ["int4", "int8", "nf4"])
@pytest.mark.parametrize("columns", [32, 128, 256])
def test_rings_wrap_over_many_segments(capi, kind, columns):
    """Every pair walks more than 120 k-blocks in several segments: each slot of the rings and the accumulators are
    used many times (mbarrier phases wrap), with whole tiles, shared tiles and splits."""
    n, k, m = 2304, 8192, 256 if columns == 32 else 600
    case = cut_case(kind, n, k, m)
    x, other, ref = case[6:]
    xb, ob = bf16_tensor(x, "cuda"), bf16_tensor(other, "cuda")
    for cut in (capi.PAIR_CUT_SHARES, capi.PAIR_CUT_WHOLE, capi.PAIR_CUT_SPLIT2):
        ctx = cut_ctx(capi, case, n, k, columns, cut)
        first = None
        for _ in range(4):
            y = ctx.linear(xb, capi.FUSE_ADD, [ob])
            first = y if first is None else first
            assert torch.equal(y, first)
        ctx.workspace(m).status()
        check(bf16_numpy(first), ref)
