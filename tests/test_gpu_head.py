"""The LM head's kernels at the edges of their tiles (GPU): logits against a float64 product, the greedy token
against numpy, the fused steps before the logits against the operators they are made of."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import synth
from colormlm_b200.s14 import S14Context, TokenRoute

from .test_gpu_parity import dev, dev_page, make_layer

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    c = S14Context(0)
    yield c
    c.close()


# rows: less than a tile, tiles with a remainder, few and many tiles, more tiles than the CTAs hold at a time (8 tokens of 4096 walk K in phases); hidden: one group of
# steps, several phases, sizes the tensor-core kernel leaves to the other one (264; 1048: more than its four pieces per lane)
@pytest.mark.parametrize("tokens,rows,hidden", [(1, 1, 256), (8, 15, 256), (7, 17, 1280), (3, 2385, 4096), (5, 33, 264), (3, 300, 1048),
                                                (8, 300, 1048), (7, 1000, 7168), (8, 2369, 4096), (8, 132700, 1024), (8, 132700, 4096),
                                                (1, 4096, 512), (1, 4097, 768), (2, 2048, 256), (4, 1025, 1024), (6, 683, 256)])
def test_logits_at_the_edges_of_the_tiles(ctx, tokens, rows, hidden):
    g = torch.Generator(device="cuda").manual_seed(tokens * rows + hidden)
    x = torch.randn(tokens, hidden, device="cuda", generator=g)
    w = torch.empty(rows, hidden, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=g)
    out = torch.full((tokens, rows + 3), 7.0, device="cuda")
    ctx.cmd_head_logits(x, w.view(torch.int16), out, n_rows=rows)
    for r0 in range(0, rows, 16384):
        wd = w[r0:r0 + 16384].double()
        ref, mag = x.double() @ wd.T, x.double().abs() @ wd.T.abs()
        # exact products; a sum of sixteen loses at most three units of 2^-23 of its terms' magnitudes on its way into
        # double, the result one of 2^-24
        assert bool(((out[:, r0:min(r0 + 16384, rows)].double() - ref).abs() <= 4 * 2.0 ** -23 * mag).all())
    assert bool((out[:, rows:] == 7.0).all())


@pytest.mark.parametrize("rows", [40, 2100])
def test_logits_of_infinite_and_largest_values(ctx, rows):
    x = torch.zeros(2, 512, device="cuda")
    x[0, 5], x[1, 300] = float("inf"), 3.4028e38
    w = torch.ones(rows, 512, dtype=torch.bfloat16, device="cuda") * 0.5
    out = torch.empty(2, rows, device="cuda")
    ctx.cmd_head_logits(x, w.view(torch.int16), out)
    assert bool((out[0] == float("inf")).all())
    assert bool((out[1] == x[1, 300] * 0.5).all())


@pytest.mark.parametrize("bf16", [False, True])
def test_logits_are_as_close_as_sums_of_eight_products(ctx, bf16):
    """What the sums add to the error of rounding the result, root mean square over that of the results: no more than sums of
    eight products in F32 do, measured with the register kernel at N(0,1) x N(0,0.02) over 4096 (4.02e-8 for F32 x; 7.5e-9 for
    BF16 values, whose products are exact)."""
    g = torch.Generator(device="cuda").manual_seed(17)
    x = torch.randn(8, 4096, device="cuda", generator=g)
    x = x.to(torch.bfloat16).float() if bf16 else x
    w = torch.empty(20000, 4096, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=g)
    for tokens in (1, 8):
        out = torch.empty(tokens, 20000, device="cuda")
        ctx.cmd_head_logits(x[:tokens], w.view(torch.int16), out)
        ref = x[:tokens].double() @ w.double().T
        added = (out.double() - ref).pow(2).mean() - (ref.float().double() - ref).pow(2).mean()
        assert float((added.clamp(min=0) / ref.pow(2).mean()).sqrt()) <= (7.5e-9 if bf16 else 4.02e-8)


# 264: the register kernel; 4096 with eight tokens: several phases of K
@pytest.mark.parametrize("tokens,hidden,rows", [(1, 256, 4100), (1, 264, 70), (1, 512, 70), (3, 512, 1400), (8, 4096, 70)])
def test_logits_of_infinite_weights_and_overflowing_products(ctx, tokens, hidden, rows):
    """One infinite weight gives an infinite logit of its sign (x is finite and nowhere 0), both signs or a NaN give NaN,
    and a product or sum beyond the largest float is infinite; the rows beside them are the ordinary ones."""
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    inf = float("inf")
    x = (torch.rand(tokens, hidden, device="cuda", generator=g) + 0.5).to(torch.bfloat16).float()  # the last part is 0
    x[-1] *= 1.0 + 2.0 ** -20                                                                       # ... or is not
    w = torch.empty(rows, hidden, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=g)
    out, plain = torch.empty(tokens, rows, device="cuda"), torch.empty(tokens, rows, device="cuda")
    ctx.cmd_head_logits(x, w.view(torch.int16), plain)
    w[3, 7], w[20, hidden - 1], w[33, 0], w[33, hidden // 2], w[41, 9], w[69, 8] = inf, -inf, inf, -inf, float("nan"), 3.3e38
    w[50, ::2] = -2.0 ** 127
    x[0, 8] = 3.0
    ctx.cmd_head_logits(x, w.view(torch.int16), out)
    assert bool((out[:, 3] == inf).all()) and bool((out[:, 20] == -inf).all()) and bool((out[:, 50] == -inf).all())
    assert bool(out[:, [33, 41]].isnan().all()) and float(out[0, 69]) == inf
    others = [r for r in range(rows) if r not in (3, 20, 33, 41, 50, 69)]
    assert torch.equal(out[1:, others], plain[1:, others]) and bool(out[:, others].isfinite().all())
    # the greedy token is the row with the positive infinity (without the NaN rows)
    out[:, [33, 41]] = 0.0
    token = torch.empty(1, dtype=torch.int64, device="cuda")
    ctx.cmd_greedy_argmax(out[0].contiguous(), token)
    assert int(token) == 3


# the kernel of few row tiles and the other one, in phases (8 tokens of 4096) and not, one block of K per half and many; above a
# tile per SM CTAs of one tile (up to 2048 tokens x hidden), of two, rounds of one (3 of 7168), parts in registers (8 tokens)
@pytest.mark.parametrize("tokens,hidden", [(1, 256), (3, 768), (1, 2048), (1, 4096), (5, 1024), (4, 4096), (8, 4096), (2, 6144), (3, 7168), (8, 7168)])
def test_logits_of_a_vocabulary_shard_have_the_bits_of_the_whole(ctx, tokens, hidden):
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    x = torch.randn(tokens, hidden, device="cuda", generator=g)
    w = torch.empty(9000, hidden, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=g).view(torch.int16)
    whole = torch.empty(tokens, 9000, device="cuda")
    ctx.cmd_head_logits(x, w, whole)
    for r0, r1 in ((0, 1), (5, 22), (100, 2468), (100, 2470), (100, 4836), (100, 4837), (8985, 9000)):
        part = torch.empty(tokens, r1 - r0, device="cuda")
        ctx.cmd_head_logits(x, w[r0:r1], part)
        assert torch.equal(part, whole[:, r0:r1]), (r0, r1)


@pytest.mark.parametrize("rows", [4000, 40000])
def test_logits_behind_a_kernel_that_fills_shared_memory(ctx, rows):
    """The step of a decode loop: the layer kernel, then the logits as its dependent launch.  The 40000 rows' step took 1.36 times
    as long as with a kernel in between, because the SMs kept the layer kernel's division and left the loads no L1."""
    hidden, inter = 4096, 2048
    g, pages, shared = make_layer(77, hidden, inter, 2, L.PAGE_MXFP4)
    pages_dev, shared_dev = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter)
    route = TokenRoute([0, 1], np.asarray([0.6, 0.4], np.float32), [p.data_ptr() for p in pages_dev])
    ctx.set_accumulation(L.ACCUM_PAIRWISE)
    x, y = dev(synth.activations(g, 1, hidden)), torch.empty(1, hidden, device="cuda")
    ws = [torch.empty(rows, hidden, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02).view(torch.int16) for _ in range(max(1, 80000 // rows))]
    out, between = torch.empty(1, rows, device="cuda"), torch.zeros(1, device="cuda")

    def run(apart):
        times = []
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for w in ws * (80 // len(ws)):
                ctx.cmd_moe_layer(x, y, [route], shared_dev.data_ptr(), L.PAGE_MXFP4, hidden, inter)
                if apart:
                    between.add_(1.0)
                ctx.cmd_head_logits(y, w, out)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)

    run(True)
    assert ctx.last_layer_path & 0xFF == L.LAYER_PATH_TENSOR
    assert run(False) < 1.15 * run(True)


@pytest.mark.parametrize("vocab,offset", [(1, 0), (3, 0), (2047, 1), (4096, 0), (16385, 0), (129280, 0), (129281, 3)])
def test_greedy_token(ctx, vocab, offset):
    g = np.random.default_rng(vocab)
    full = torch.empty(vocab + offset, device="cuda")
    res = torch.empty(1, dtype=torch.int64, device="cuda")

    def token(v):
        full[offset:] = torch.from_numpy(v).cuda()
        ctx.cmd_greedy_argmax(full[offset:], res)
        return int(res.item())

    v = g.standard_normal(vocab).astype(np.float32)
    assert token(v) == int(v.argmax())
    hits = np.unique(g.integers(0, vocab, 3))  # the lowest id of the largest value, wherever the others lie
    v[hits] = 9.0
    assert token(v) == int(hits[0])
    v = -np.abs(v) * 0.0
    v[vocab - 1] = 0.0  # -0 and +0 are equal
    assert token(v) == 0
    assert token(np.full(vocab, -np.inf, np.float32)) == 0
    v[vocab // 2] = np.nan
    assert token(v) == -1


@pytest.mark.parametrize("hidden", [256, 1024, 2304, 4096])
def test_full_logits_equal_their_operators(ctx, hidden):
    g = torch.Generator(device="cuda").manual_seed(hidden)
    state = torch.randn(1, 4, hidden, device="cuda", generator=g).to(torch.bfloat16)
    fn, base = torch.randn(4, 4 * hidden, device="cuda", generator=g) * 0.02, torch.rand(4, device="cuda", generator=g) - 0.5
    scale, norm = torch.rand(1, device="cuda", generator=g), torch.rand(hidden, device="cuda", generator=g) + 0.5
    w = (torch.randn(100, hidden, device="cuda", generator=g) * 0.02).to(torch.bfloat16).view(torch.int16)
    out, want = torch.empty(100, device="cuda"), torch.empty(100, device="cuda")
    red, pre = torch.empty(1, hidden, dtype=torch.bfloat16, device="cuda"), torch.empty(1, 4, device="cuda")
    normed = torch.empty_like(red)
    ctx.exec_hc_head_norm_full_logits(state, fn, scale, base, norm, w, out)
    ctx.cmd_hc_head_reduce(state, fn, scale, base, red, pre)
    ctx.cmd_rms_norm(red, norm, normed)
    ctx.cmd_head_logits(normed.float(), w, want)
    # the double sums run in another order: a coefficient may round the other way, which moves an element of the
    # reduced vector by at most one BF16 unit (2^-8 relative) and so a logit by 2^-8 |x| |w|
    mag = normed.float().abs()[0] @ w.view(torch.bfloat16).float().abs().T
    assert bool(((out - want).abs() <= 2.0 ** -8 * mag).all())


# one value; fewer than a warp's; a thread's loads of a round and one more; a whole round of the cluster and its neighbours
@pytest.mark.parametrize("vocab", [1, 5, 2047, 2049, 32767, 131072, 131077])
@pytest.mark.parametrize("offset", [0, 1])   # 16-byte loads, and not
def test_greedy_token_at_the_edges_of_a_round(ctx, vocab, offset):
    torch.manual_seed(vocab)
    base = torch.randn(vocab + offset, device="cuda")
    res = torch.empty(1, dtype=torch.int64, device="cuda")

    def token(v):
        full = base.clone()
        full[offset:] = v
        ctx.cmd_greedy_argmax(full[offset:], res)
        return int(res.item())

    v = base[offset:]
    assert token(v) == int(v.cpu().argmax())
    places = sorted({0, vocab // 3, vocab // 2, vocab - 1})
    for p in places:
        w = v.clone()
        w[p] = 50.0
        assert token(w) == p
        w[places[-1]] = 50.0                      # the lowest of equal ones
        assert token(w) == p
        w[p] = float("inf")
        assert token(w) == p
        w[places[0]] = float("nan")
        assert token(w) == -1
    assert token(torch.full_like(v, -float("inf"))) == 0
    w = torch.full_like(v, -1.0)
    w[places[-1]] = 0.0
    w[places[len(places) // 2]] = -0.0            # equal to +0
    assert token(w) == places[len(places) // 2]
