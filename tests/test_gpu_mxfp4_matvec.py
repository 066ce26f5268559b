"""The MXFP4 row kernels where their form changes (GPU, against the double-accumulated product): fewer rows than
SMs, a last batch of pieces with a remainder, one and two rows per warp with a remainder of each, the longest row
held in shared memory and one beyond it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import synth
from colormlm_b200.s14 import S14Context, S14MatvecShape

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]
E2M1 = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64)


@pytest.mark.parametrize("n,k", [(1, 128), (147, 4224), (149, 12544), (2369, 384), (4735, 256), (4736, 1280), (7103, 4096),
                                 (3, 32768), (3, 32896)])
def test_rows_of_all_forms(n, k):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    ctx = S14Context(0)
    g = synth.rng(n + k)
    w, s = torch.from_numpy(synth.mxfp4_codes(g, n, k)).cuda(), torch.from_numpy(synth.mxfp4_scales(g, n, k)).cuda()
    x = torch.from_numpy(synth.activations(g, 1, k)[0]).cuda()
    y = torch.full((n + 1,), 5.0, device="cuda")
    sp = torch.cat([s.reshape(-1), torch.zeros(16, dtype=torch.uint8, device="cuda")])
    d = ctx.pipelines.bind_mxfp4(S14MatvecShape(n, k), x, w, sp, y[:n])
    ctx.pipelines.cmd_mxfp4_matvec(d)
    torch.cuda.synchronize()
    val = torch.stack([E2M1.cuda()[(w & 15).long()], E2M1.cuda()[(w >> 4).long()]], dim=2).reshape(n, k)
    val = val * torch.pow(2.0, s.double() - 127).repeat_interleave(32, dim=1)
    ref, mag = val @ x.double(), val.abs() @ x.double().abs()
    # 32 products of a piece are added in F32, two chains of sixteen and one addition: 17 roundings of 2^-24 of the
    # magnitudes at most, the result's own one
    assert bool(((y[:n].double() - ref).abs() <= 18 * 2.0 ** -24 * mag).all())
    assert float(y[n]) == 5.0
    ctx.close()
