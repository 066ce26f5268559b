"""One token's FP8 projection where its launch changes form (GPU, against the product in float64): as many CTAs of eight rows as
SMs and one more, twice as many and one more, rows of 4096 and just below."""
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200.s14 import S14Context, S14MatvecShape

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]


@pytest.mark.parametrize("f32_scale", [False, True])
@pytest.mark.parametrize("n,k", [(1184, 4096), (1185, 4096), (1185, 4064), (2368, 4096), (2369, 4128), (4736, 4096)])
def test_one_token_of_all_forms(n, k, f32_scale):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    ctx = S14Context(0)
    g = torch.Generator(device="cuda").manual_seed(n + k)
    x = torch.randn(1, k, device="cuda", generator=g)
    w = torch.randint(0, 126, (n, k), dtype=torch.uint8, device="cuda", generator=g)
    w |= torch.randint(0, 2, (n, k), dtype=torch.uint8, device="cuda", generator=g) << 7
    nb, kb = (n + 127) // 128, (k + 127) // 128
    if f32_scale:
        s = torch.rand(nb, kb, device="cuda", generator=g) + 0.5
        scale, fmt, buf = s.double(), L.SCALE_F32, s
    else:
        codes = torch.randint(119, 123, (nb, kb), dtype=torch.uint8, device="cuda", generator=g)
        scale, fmt = torch.pow(2.0, codes.double() - 127), L.SCALE_UE8M0
        buf = torch.cat([codes.reshape(-1), torch.zeros(16, dtype=torch.uint8, device="cuda")])
    y = torch.full((1, n), 5.0, device="cuda")
    op = ctx.pipelines.bind_fp8(S14MatvecShape(n, k), x, w, buf, y, scale_format=fmt, n_tokens=1)
    ctx.pipelines.cmd_fp8_matvec(op)
    torch.cuda.synchronize()
    val = w.view(torch.float8_e4m3fn).double() * scale.repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
    ref, mag = val @ x[0].double(), val.abs() @ x[0].double().abs()
    # sixteen products of a piece in F32 (two chains of eight and one addition), then double, the result rounded once
    assert bool(((y[0].double() - ref).abs() <= 10 * 2.0 ** -24 * mag).all())
    ctx.close()
