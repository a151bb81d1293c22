"""Host threads that run linears of different token counts at the same time, each on its own stream and workspace:
every launch succeeds and gives what it gives alone."""
import os
import subprocess
import sys
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


FIRST_CALLS = """
import threading, torch
from ipex_b200 import _capi as C
n, k, m = 256, 512, 32
ctxs = [C.WoqContext(torch.zeros((n, k // 2), dtype=torch.uint8, device="cuda"), torch.ones((n, 4), device="cuda"), None,
                     None, n, k, C.DTYPE_INT4, 128, C.LOWP_BF16) for _ in range(16)]
x, outs = torch.ones((m, k), device="cuda").bfloat16(), [torch.empty((m, n), device="cuda").bfloat16() for _ in ctxs]
ws = [C.Workspace(c.workspace_bytes(m), "cuda") for c in ctxs]
torch.cuda.synchronize()
start, codes, call = threading.Barrier(16), [], C.lib().woq_b200_linear
def work(i):
    args = (ctxs[i].handle, x.data_ptr(), m, k, 0, None, 0, outs[i].data_ptr(), n, ws[i].buf.data_ptr(), ws[i].nbytes,
            torch.cuda.Stream().cuda_stream)
    start.wait()
    codes.append(call(*args))
threads = [threading.Thread(target=work, args=(i,)) for i in range(16)]
[t.start() for t in threads]
[t.join() for t in threads]
torch.cuda.synchronize()
assert codes == [0] * 16, codes
assert all(bool((o == -8 * k).all()) for o in outs)
"""


def test_first_calls_of_a_process_from_many_threads():
    """What the library looks up once (driver entry points, capacities of the device) is there for every caller."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "intel-extension-for-pytorch_b200")]))
    for _ in range(3):
        out = subprocess.run([sys.executable, "-c", FIRST_CALLS], env=env, capture_output=True, text=True, timeout=300)
        assert out.returncode == 0, out.stderr[-2000:]
