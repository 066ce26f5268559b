"""The router of blocks of more than 64 tokens (csrc/s14_router.cu) takes a score in double only where an error bound says that the expert
can be among the picked ones.  Ids and weights have the bits of the CPU oracle's router, which takes all of them (GPU)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import synth
from colormlm_b200.pages import ExpertPageLayout
from colormlm_b200.s14 import MoeBlock, S14Context

from .test_gpu_parity import dev

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    c = S14Context(0)
    yield c
    c.close()


def bf16(a):
    return synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(np.ascontiguousarray(a, np.float32)))


def rows(g, kind, n_tokens, n_experts, hidden):
    """Tokens, router weights (BF16 values as F32) and biases of one kind."""
    x = g.standard_normal((n_tokens, hidden)).astype(np.float32)
    w = bf16(g.standard_normal((n_experts, hidden)) * 0.02)
    b = (g.random(n_experts) * 0.2 - 0.1).astype(np.float32)
    if kind == "ties":            # every expert twice: equal scores, the lower id first
        w[1::2], b[1::2] = w[:-1:2][:len(w[1::2])], b[:-1:2][:len(b[1::2])]
    elif kind == "near":          # experts a last bit of one weight apart: more candidates than a pass takes
        w[:] = w[0]
        w[:, 0] = bf16(0.5 + np.arange(n_experts) * 2.0 ** -9)
        b[:] = 0
    elif kind == "small":         # squares of the tokens underflow
        x *= np.float32(1e-30)
    elif kind == "large":         # ... overflow: every expert is a candidate
        x *= np.float32(1e25)
        w = bf16(w * 1e-22)
    elif kind == "zero":          # all scores equal but for the bias, of which some are equal
        x[:] = 0
        b = np.round(b * 20).astype(np.float32) / 16
    elif kind == "outlier":       # one element carries the dot product
        x[:, 3] *= 3000
    return x, w, b


# one token above the boundary, tiles of 16 tokens with a rest, the largest tile and one more; experts of one tile and of two, of a pass and
# fewer than a group of maxima; every number of K steps from 1 to 8 at the ends
@pytest.mark.parametrize("kind,n_tokens,n_experts,hidden,top_k", [
    ("plain", 65, 256, 512, 6), ("plain", 144, 129, 2560, 6), ("plain", 145, 7, 1024, 6), ("plain", 300, 128, 4096, 3), ("plain", 1024, 250, 512, 6),
    ("ties", 80, 256, 1024, 6), ("near", 80, 256, 1024, 6), ("near", 80, 40, 512, 1), ("small", 70, 200, 1024, 6), ("large", 70, 200, 1024, 6),
    ("zero", 66, 256, 512, 6), ("outlier", 90, 256, 4096, 6)])
@pytest.mark.parametrize("score_fn", [L.SCORE_SIGMOID, L.SCORE_SQRT_SOFTPLUS])
def test_routes_have_the_oracles_bits(ctx, oracle, kind, n_tokens, n_experts, hidden, top_k, score_fn):
    g = synth.rng(40 + n_tokens + n_experts + hidden)
    x, w, b = rows(g, kind, n_tokens, n_experts, hidden)
    bits = synth.f32_to_bf16_bits(w)
    page = torch.zeros(ExpertPageLayout(hidden, 512, L.PAGE_MXFP4).page_bytes, dtype=torch.uint8, device="cuda")
    table = torch.full((n_experts,), page.data_ptr(), dtype=torch.int64, device="cuda")
    ids = torch.full((n_tokens, top_k), -1, dtype=torch.int32, device="cuda")
    wts = torch.full((n_tokens, top_k), float("nan"), device="cuda")
    blk = MoeBlock(ctx, hidden, 512, n_tokens)
    try:
        blk.cmd_routed_moe_block(dev(x), dev(bits.view(np.int16)), dev(b), table, page.data_ptr(), torch.empty((n_tokens, hidden), device="cuda"),
                                 ids, wts, score_fn=score_fn, top_k=top_k, route_scale=1.5)
        torch.cuda.synchronize()
        assert ctx.device_status() == 0
        ids_np, w_np = ids.cpu().numpy(), wts.cpu().numpy()
        for t in range(0, n_tokens, max(1, n_tokens // 50)):
            rid, rw, _, _ = oracle.router(x[t], bits, b, score_fn=score_fn, top_k=top_k, route_scale=1.5)
            assert np.array_equal(ids_np[t], rid), t
            assert np.array_equal(w_np[t].view(np.uint32), rw.view(np.uint32)), t
    finally:
        blk.close()
