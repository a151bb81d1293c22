"""Host threads that run linears of different token counts at the same time, each on its own stream and workspace:
every launch succeeds and gives what it gives alone."""
import threading

import pytest
import torch

from oracle import woq_oracle as O
from tests.helpers import bf16_tensor, make_acts, make_int4_layer, to_device_layer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ipex_b200 import _capi

    _capi.lib()
    return _capi


# token counts of one kernel whose launches ask for different amounts of shared memory
@pytest.mark.parametrize("route,tokens", [("int4", (17, 256)), ("int4", (1, 6)), ("int4_tc", (2, 16)), ("int8", (9, 256)),
                                          ("k_blocks", (20, 128))])
def test_two_threads(capi, route, tokens):
    n, k, g = 640, 1024, 128
    layer = make_int4_layer(n, k, g, seed=1)
    qw, s, z, _ = to_device_layer(layer, "cuda")
    if route == "int8":
        w8 = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda")
        ctx = capi.WoqContext(w8, torch.full((n, 1), 0.01, device="cuda"), None, None, n, k, O.WOQ_DTYPE_INT8, -1,
                              capi.LOWP_INT8, act_quant_mode=6)
    elif route == "k_blocks":
        ctx = capi.WoqContext(qw, s.float(), z, None, n, k, capi.DTYPE_INT4, g, capi.LOWP_INT8, act_quant_mode=7)
    else:
        ctx = capi.WoqContext(qw, s, z, None, n, k, capi.DTYPE_INT4, g, capi.LOWP_BF16,
                              kernel_hint=1 if route == "int4_tc" else 0)
    xs = [bf16_tensor(make_acts(m, k, seed=m), "cuda") for m in tokens]
    refs = [ctx.linear(x) for x in xs]
    torch.cuda.synchronize()
    start, errors, outs = threading.Barrier(2), [], [[], []]

    def work(i):
        try:
            torch.cuda.set_device(0)
            x, m = xs[i], tokens[i]
            ws = capi.Workspace(ctx.workspace_bytes(m), "cuda")
            out = [torch.empty_like(refs[i]) for _ in range(4)]
            torch.cuda.synchronize()
            stream = torch.cuda.Stream()
            # bare calls of the C ABI, so that the threads spend their time in the library, beside each other
            call = capi.lib().woq_b200_linear
            args = [(ctx.handle, x.data_ptr(), m, x.stride(0), 0, None, 0, y.data_ptr(), y.stride(0), ws.buf.data_ptr(),
                     ws.nbytes, stream.cuda_stream) for y in out]
            start.wait()
            codes = {call(*args[j % 4]) for j in range(20000)}
            stream.synchronize()
            assert codes == {0}, (codes, capi.lib().woq_b200_last_error())
            with torch.cuda.stream(stream):
                ws.status()
            outs[i] = out
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for out, ref in zip(outs, refs):
        assert len(out) == 4 and all(torch.equal(y, ref) for y in out)
