"""The selection of the routes where scores are equal: the lowest ids, whatever lane and word of a lane holds them (GPU,
against the CPU oracle)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import synth
from colormlm_b200.s14 import S14Context

from .test_gpu_parity import dev

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    c = S14Context(0)
    yield c
    c.close()


# as many experts as picks, a warp's and one more, the most; picks up to the operator's eight
@pytest.mark.parametrize("n_experts,top_k", [(1, 1), (6, 6), (8, 8), (32, 6), (33, 8), (255, 6), (256, 8)])
@pytest.mark.parametrize("levels", [1, 2, 5])   # different values of the bias
def test_lowest_ids_of_equal_scores(ctx, oracle, n_experts, top_k, levels):
    g = synth.rng(17 + n_experts + levels)
    hidden, tokens = 512, 3
    x = synth.activations(g, tokens, hidden)
    wr = np.zeros((n_experts, hidden), np.uint16)
    bias = (g.integers(0, levels, n_experts) * 0.25 - 1.0).astype(np.float32)   # score 1/2: keys of either sign and zero
    ids = torch.empty((tokens, top_k), dtype=torch.int32, device="cuda")
    wts = torch.empty((tokens, top_k), dtype=torch.float32, device="cuda")
    ctx.cmd_router(dev(x), dev(wr.view(np.int16)), dev(bias), ids, wts, score_fn=L.SCORE_SIGMOID, top_k=top_k, route_scale=1.5)
    torch.cuda.synchronize()
    want = np.argsort(-bias, kind="stable")[:top_k]
    for t in range(tokens):
        rid, rw, _, _ = oracle.router(x[t], wr, bias, score_fn=L.SCORE_SIGMOID, top_k=top_k, route_scale=1.5)
        assert np.array_equal(rid, want) and np.array_equal(ids[t].cpu().numpy(), want)
        assert np.array_equal(wts[t].cpu().numpy().view(np.uint32), rw.view(np.uint32))
