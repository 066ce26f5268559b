"""A launch that the CUDA runtime refuses (an empty grid) is that call's error alone (GPU; nothing runs on the device)."""
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200.s14 import S14Context, S14Error, S14MatvecShape

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]


@pytest.mark.parametrize("operator", ["mxfp4_matvec", "fp8_matvec", "swiglu_limit", "route_mix", "moe_accumulate"])
def test_a_refused_launch_leaves_no_error_behind(operator):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    ctx = S14Context(0)
    p, n = ctx.pipelines, 128
    f, b = (lambda k: torch.ones(k, device="cuda")), (lambda k: torch.ones(k, dtype=torch.uint8, device="cuda"))
    x, y, w, s = f(n), f(n), b(n * n), b(64 * n)
    record = {"mxfp4_matvec": lambda: p.bind_mxfp4(S14MatvecShape(n, n), x, w, s, y),
              "fp8_matvec": lambda: p.bind_fp8(S14MatvecShape(n, n), x, w, s, y),
              "swiglu_limit": lambda: p.bind_swiglu_limit(n, x, x, y),
              "route_mix": lambda: p.bind_route_mix(n, 0.5, x, y),
              "moe_accumulate": lambda: p.bind_moe_accumulate(n, 0.5, x, y)}[operator]()
    if hasattr(record, "shape"):
        record.shape.n = 0   # the record is the caller's; binding would have refused this
    else:
        record.n = 0
    with pytest.raises(S14Error) as e:
        getattr(p, "cmd_" + operator)(record)
    assert e.value.code == L.ERR_CUDA
    # the next checks of the runtime's last error, torch's and the library's, are of calls that went well
    assert float(torch.full((4,), 2.0, device="cuda").sum()) == 8.0
    logits, token = torch.arange(12.0, device="cuda"), torch.empty(1, dtype=torch.int64, device="cuda")
    out = torch.empty(1, 3, device="cuda")
    ctx.cmd_head_logits(f(8), torch.ones(3, 8, dtype=torch.bfloat16, device="cuda").view(torch.int16), out)
    ctx.cmd_greedy_argmax(logits, token)
    assert int(token) == 11 and out.tolist() == [[8.0, 8.0, 8.0]]
    ctx.close()
