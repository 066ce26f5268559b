"""Official blocks whose CTA pairs have more items than a batch of records (56), in the forms for 16 and for 32 tokens to a chunk: the same bits as
the same tokens in blocks of twelve, which take the form for four and one batch (GPU)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import synth
from colormlm_b200.s14 import MoeBlock, S14Context, TokenRoute

from .test_gpu_parity import dev, dev_page, make_layer

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]
BATCH, N_PAGES = 56, 8


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    c = S14Context(0)
    yield c
    c.close()


# sixteen tokens: up items (252 pairs over 252 experts, fewer than the 256 a large chunk needs), down items (510 pairs of short pages); 32: both
@pytest.mark.parametrize("hidden,inter,n_tokens,more", [(512, 4096, 42, "up"), (4096, 512, 85, "down"), (4096, 4096, 300, "both")])
def test_items_beyond_a_batch(ctx, hidden, inter, n_tokens, more):
    g, pages, shared = make_layer(2300 + n_tokens, hidden, inter, N_PAGES, L.PAGE_MXFP4)
    shared_dev = dev_page(shared, hidden, inter)
    keep = [dev_page(p, hidden, inter) for p in pages]
    pages_dev = [p.data_ptr() for p in keep]
    x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(synth.activations(g, n_tokens, hidden)))
    dx = dev(x)
    routes = []
    for t in range(n_tokens):
        ids = [(6 * t + j) % 256 for j in range(6)]
        routes.append(TokenRoute(ids, g.uniform(0.05, 0.4, 6).astype(np.float32), [pages_dev[e % N_PAGES] for e in ids]))

    def run(first, count):
        y = torch.full((count, hidden), float("nan"), device="cuda")
        blk = MoeBlock(ctx, hidden, inter, count)
        try:
            blk.set_semantics(True)
            blk.cmd_moe_block(dx[first:first + count], y, routes[first:first + count], shared_dev.data_ptr())
            torch.cuda.synchronize()
            assert ctx.device_status() == 0
            return y, blk.last_counts()
        finally:
            blk.close()

    y, (chunks, n_up, n_down, bad) = run(0, n_tokens)
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert bad == 0
    if more in ("up", "both"):
        assert n_up > BATCH * pairs
    if more in ("down", "both"):
        assert n_down > BATCH * pairs
    # (32 tokens to a chunk: 16 would cut the shared expert's into twice as many)
    assert chunks == min(6 * n_tokens, 256) + -(-n_tokens // (32 if more == "both" else 16))
    for first in range(0, n_tokens, 12):
        count = min(12, n_tokens - first)
        assert torch.equal(y[first:first + count].view(torch.int32), run(first, count)[0].view(torch.int32)), first
