"""The Sinkhorn rounds of hc_pre by themselves (csrc/s14_glue.cu, device_parts.cu): the oracle's bits, also where values on the way leave the range
of the rounds' own division and they are done over with the operator (GPU)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from .test_gpu_parts import part, ptr  # noqa: F401

pytestmark = pytest.mark.gpu


# (eps, spread of the logits, rounds, the smallest coefficient's magnitude is below 2^-60)
@pytest.mark.parametrize("eps,spread,iters,small", [
    (1e-6, 1.0, 20, False), (1e-6, 120.0, 20, False), (1e-6, 1.0, 1, False), (1e-30, 1.0, 20, False), (1e-30, 50.0, 3, True), (1e-30, 80.0, 20, True),
    (1e-38, 100.0, 2, True), (1e-19, 60.0, 20, True), (1e19, 1.0, 2, True), (3e-18, 60.0, 5, True)])
def test_the_rounds_have_the_oracles_bits(part, oracle, eps, spread, iters, small):  # noqa: F811
    g = np.random.default_rng(int(spread) + iters)
    n = 400
    mixes = g.uniform(-1, 1, (n, 24)).astype(np.float32)
    scale, base = np.asarray([0.5, 0.25, spread], np.float32), g.uniform(-1, 1, 24).astype(np.float32)
    dev = [torch.from_numpy(a).cuda() for a in (mixes, scale, base)]
    comb = torch.empty((n, 4, 4), device="cuda")
    assert part("SINKHORN").sinkhorn(n, *[ptr(t) for t in dev], iters, C.c_float(eps), ptr(comb)) == 0
    torch.cuda.synchronize()
    want = np.stack([oracle.hc_split_sinkhorn(m, scale, base, iters=iters, eps=eps)[2] for m in mixes])
    assert (bool((np.abs(want[want != 0]) < 2.0 ** -60).any())) == small
    assert np.array_equal(comb.cpu().numpy().view(np.uint32), want.view(np.uint32))
