"""The layer-glue operators where their kernels change form: the cluster kernels' last token counts and the first of
the matrix kernel (on 148 SMs), a group of sixteen tokens with a remainder, the smallest and the largest hidden size, buffers
that are not aligned to 16 bytes (GPU, against the CPU oracle)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import synth
from colormlm_b200.s14 import S14Context, S14Error

from .test_gpu_glue import bits16, close_coeff, close_streams, dev, f32_of_bits

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    c = S14Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n_tokens,hidden", [(1, 256), (7, 512), (8, 1280), (9, 256), (9, 8192), (13, 512), (14, 2048), (27, 256),
                                              (28, 768), (55, 256), (56, 1280), (111, 256), (112, 256), (150, 1024), (15, 512),
                                              (149, 1024), (593, 256), (889, 512), (300, 512), (300, 768), (300, 1024),
                                              (600, 1024), (300, 5120), (889, 2048)])
def test_sites_of_all_forms(ctx, oracle, bf16, n_tokens, hidden):
    g = synth.rng(77 + n_tokens + hidden)
    fn, scale, base = synth.hc_params(g, hidden)
    nw = g.uniform(0.5, 1.5, size=hidden).astype(np.float32)
    x = dev(synth.hc_streams(g, n_tokens, hidden), bf16)
    host = (lambda t: bits16(t)) if bf16 else (lambda t: t.cpu().numpy())
    as_f32 = (lambda a: f32_of_bits(a)) if bf16 else (lambda a: a)
    red, merged = torch.empty((n_tokens, hidden), dtype=x.dtype, device="cuda"), torch.empty_like(x)
    post, comb = torch.empty((n_tokens, 4), device="cuda"), torch.empty((n_tokens, 4, 4), device="cuda")
    normed = torch.empty_like(red)
    ctx.cmd_hc_pre(x, dev(fn), dev(scale), dev(base), red, post, comb)
    ctx.cmd_rms_norm(red, dev(nw), normed)
    ctx.cmd_hc_post(normed, x, post, comb, merged)
    torch.cuda.synchronize()
    r_ref, p_ref, c_ref = oracle.hc_pre(host(x), fn, scale, base, dtype=int(bf16))
    close_coeff(post.cpu().numpy(), p_ref)
    close_coeff(comb.cpu().numpy(), c_ref)
    close_streams(as_f32(host(red)), as_f32(r_ref), bf16)
    close_streams(as_f32(host(normed)), as_f32(oracle.rms_norm(host(red), nw, dtype=int(bf16))), bf16)
    m_ref = oracle.hc_post(host(normed), host(x), post.cpu().numpy(), comb.cpu().numpy(), dtype=int(bf16))
    assert np.array_equal(as_f32(host(merged)), as_f32(m_ref))
    # hc_pre's clusters: sixteen CTAs up to 7 tokens, then two launches whose slices of K go by the tokens; F32 norms change form at 149,
    # 593 and 889 tokens; the head's reduce: clusters of sixteen CTAs per token (up to 13 tokens), eight (27), four (55), two
    # (short rows, up to 111 or 74), two launches
    hfn, hscale, hbase = synth.hc_params(g, hidden, head=True)
    pre = torch.empty((n_tokens, 4), device="cuda")
    ctx.cmd_hc_head_reduce(x, dev(hfn), dev(hscale), dev(hbase), red, pre)
    h_ref, pre_ref = oracle.hc_head_reduce(host(x), hfn, hscale, hbase, dtype=int(bf16))
    close_coeff(pre.cpu().numpy(), pre_ref)
    close_streams(as_f32(host(red)), as_f32(h_ref), bf16)


@pytest.mark.parametrize("bf16", [False, True])
def test_buffers_that_are_not_16_byte_aligned(ctx, bf16):
    g = torch.Generator(device="cuda").manual_seed(3)
    t, h, dt = 3, 512, torch.bfloat16 if bf16 else torch.float32
    make = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dt)
    branch, res, nw = make(t, h), make(t, 4, h), torch.rand(h, device="cuda", generator=g)
    post, comb = torch.rand(t, 4, device="cuda", generator=g), torch.rand(t, 4, 4, device="cuda", generator=g)

    def moved(a):
        big = torch.empty(a.numel() + 1, dtype=a.dtype, device="cuda")
        big[1:] = a.reshape(-1)
        return big[1:].view(a.shape)

    want_m, want_n = torch.empty_like(res), torch.empty_like(branch)
    ctx.cmd_hc_post(branch, res, post, comb, want_m)
    ctx.cmd_rms_norm(branch, nw, want_n)
    got_m, got_n = moved(want_m), moved(want_n)
    got_m.zero_(), got_n.zero_()
    ctx.cmd_hc_post(moved(branch), moved(res), post, comb, got_m)
    ctx.cmd_rms_norm(moved(branch), moved(nw), got_n)
    assert torch.equal(got_m, want_m) and torch.equal(got_n, want_n)


def _offset(a, elements):
    """A copy of a that lies `elements` past a 16-byte boundary."""
    big = torch.empty(a.numel() + elements, dtype=a.dtype, device="cuda")
    big[elements:] = a.reshape(-1)
    return big[elements:].view(a.shape)


@pytest.mark.parametrize("tokens", [1, 11])
def test_reduce_of_streams_on_the_boundaries_it_takes(ctx, tokens):
    """BF16 streams on an 8-byte boundary and results on any are taken; what the dot products cannot read is refused before
    anything is launched."""
    g = torch.Generator(device="cuda").manual_seed(8)
    h = 512
    x = torch.randn(tokens, 4, h, device="cuda", generator=g)
    fn = torch.randn(24, 4 * h, device="cuda", generator=g) * 0.02
    scale, base = torch.rand(3, device="cuda", generator=g), torch.rand(24, device="cuda", generator=g)
    post, comb, pre = torch.empty(tokens, 4, device="cuda"), torch.empty(tokens, 4, 4, device="cuda"), torch.empty(tokens, 4, device="cuda")
    b = x.to(torch.bfloat16)
    red, moved = torch.empty(tokens, h, dtype=b.dtype, device="cuda"), _offset(torch.zeros(tokens, h, dtype=b.dtype, device="cuda"), 1)
    ctx.cmd_hc_pre(b, fn, scale, base, red, post, comb)
    ctx.cmd_hc_pre(_offset(b, 4), fn, _offset(scale, 1), _offset(base, 3), moved, _offset(post, 1), _offset(comb, 1))
    assert torch.equal(red, moved)
    launched = ctx.launch_count
    for streams, matrix in ((_offset(b, 1), fn), (_offset(b, 2), fn), (_offset(x, 1), fn), (_offset(x, 2), fn), (x, _offset(fn, 1)),
                            (b, _offset(fn, 2))):
        out = torch.empty(tokens, h, dtype=streams.dtype, device="cuda")
        for call in (lambda: ctx.cmd_hc_pre(streams, matrix, scale, base, out, post, comb),
                     lambda: ctx.cmd_hc_head_reduce(streams, matrix, scale, base, out, pre)):
            with pytest.raises(S14Error) as e:
                call()
            assert e.value.code == L.ERR_CONTRACT
    w, norm, logits = torch.ones(20, h, dtype=torch.bfloat16, device="cuda").view(torch.int16), torch.ones(h, device="cuda"), torch.empty(20, device="cuda")
    for state, matrix, head in ((_offset(b[:1], 1), fn, w), (b[:1], _offset(fn, 1), w), (b[:1], fn, _offset(w, 4))):
        with pytest.raises(S14Error):
            ctx.exec_hc_head_norm_full_logits(state, matrix, scale, base, norm, head, logits)
    assert ctx.launch_count == launched
    torch.cuda.synchronize()


# slices of K that are no whole number of steps each (37 of 128 steps at 190 x 512, 24 of 192 at 60 x 768), a step per warp (64 x 256),
# one group of tokens and 64 slices (16 x 2048), one more token; the last token count whose streams are read in front of the wait on
# 148 SMs and the one behind it (BF16 592, F32 740)
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n_tokens,hidden", [(190, 512), (60, 768), (64, 256), (16, 2048), (17, 2304), (592, 512), (594, 512), (740, 512), (741, 256)])
def test_sites_at_the_edges_of_slices(ctx, oracle, bf16, n_tokens, hidden):
    test_sites_of_all_forms(ctx, oracle, bf16, n_tokens, hidden)


@pytest.mark.parametrize("bf16", [False, True])
def test_reduce_of_many_tokens_into_an_unaligned_result(ctx, bf16):
    g = torch.Generator(device="cuda").manual_seed(9)
    t, h, dt = 40, 768, torch.bfloat16 if bf16 else torch.float32
    x = torch.randn(t, 4, h, device="cuda", generator=g).to(dt)
    fn = torch.randn(24, 4 * h, device="cuda", generator=g) * 0.02
    scale, base = torch.rand(3, device="cuda", generator=g), torch.rand(24, device="cuda", generator=g)
    post, comb = torch.empty(t, 4, device="cuda"), torch.empty(t, 4, 4, device="cuda")
    red, moved = torch.empty(t, h, dtype=dt, device="cuda"), _offset(torch.zeros(t, h, dtype=dt, device="cuda"), 1)
    ctx.cmd_hc_pre(x, fn, scale, base, red, post, comb)
    ctx.cmd_hc_pre(_offset(x, 4), fn, scale, base, moved, post, comb)
    torch.cuda.synchronize()
    assert torch.equal(red, moved)


# the head's clusters of two of short rows (on 148 SMs up to 111 tokens of 1024, 74 of 1792) and the two launches behind them; five
# slices of K to an SM (F32, 592 tokens of 2048); hc_post's division of the SMs (32 tokens), its values a thread (186 of 2048) and its registers
# (148 of 4096)
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n_tokens,hidden", [(111, 1024), (112, 1024), (74, 1792), (75, 1792), (74, 2048), (592, 2048), (32, 512), (33, 512),
                                             (185, 2048), (186, 2048), (148, 4096), (149, 4096)])
def test_sites_where_forms_change(ctx, oracle, bf16, n_tokens, hidden):
    test_sites_of_all_forms(ctx, oracle, bf16, n_tokens, hidden)


# what goes by the number of tokens on other boundaries too: hc_post's values a thread and registers, the norm's forms
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("t,h", [(148, 1024), (149, 1024), (185, 2048), (186, 2048), (149, 4096), (296, 1024), (297, 1024), (444, 1024),
                                 (445, 1024)])
def test_many_tokens_on_any_boundary(ctx, bf16, t, h):
    g = torch.Generator(device="cuda").manual_seed(t + h)
    dt = torch.bfloat16 if bf16 else torch.float32
    make = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dt)
    branch, res, nw = make(t, h), make(t, 4, h), torch.rand(h, device="cuda", generator=g)
    post, comb = torch.rand(t, 4, device="cuda", generator=g), torch.rand(t, 4, 4, device="cuda", generator=g)
    want_m, want_n = torch.empty_like(res), torch.empty_like(branch)
    ctx.cmd_hc_post(branch, res, post, comb, want_m)
    ctx.cmd_rms_norm(branch, nw, want_n)
    b, r = branch.float(), res.float()
    ref = nw * (b * torch.rsqrt(b.double().pow(2).mean(1, keepdim=True) + 1e-6).float())
    # an F32 sum in another order and three roundings: some 1e-6 of the result; a BF16 value is rounded by 2^-9 of it
    assert (want_n.float() - ref).abs().max() <= (2.0 ** -8 if bf16 else 2e-6) * ref.abs().max()
    ref = post[:, :, None] * b[:, None, :] + torch.einsum("tio,tid->tod", comb, r)
    assert (want_m.float() - ref).abs().max() <= (2.0 ** -8 if bf16 else 2e-6) * ref.abs().max()
    for offset in (1, 2, 4):
        got_m, got_n = _offset(torch.zeros_like(want_m), offset), _offset(torch.zeros_like(want_n), offset)
        ctx.cmd_hc_post(_offset(branch, offset), _offset(res, offset), post, comb, got_m)
        ctx.cmd_rms_norm(_offset(branch, offset), _offset(nw, offset), got_n)
        assert torch.equal(got_m, want_m) and torch.equal(got_n, want_n)


@pytest.mark.parametrize("n_tokens", [1, 20])
@pytest.mark.parametrize("eps,spread,iters", [(1e-6, 120.0, 20), (1e-30, 1.0, 20), (1e-30, 50.0, 3), (1e-6, 1.0, 1)])
def test_sinkhorn_rounds_of_any_values(ctx, oracle, n_tokens, eps, spread, iters):
    """Logits whose softmax underflows, an epsilon out of the range of the rounds' own division (which then are done over with the operator), few
    rounds: the oracle's coefficients."""
    hidden = 512
    g = synth.rng(91)
    fn, scale, base = synth.hc_params(g, hidden)
    base = (g.uniform(-1, 1, size=base.shape) * spread).astype(np.float32)
    x = dev(synth.hc_streams(g, n_tokens, hidden))
    red = torch.empty((n_tokens, hidden), device="cuda")
    post, comb = torch.empty((n_tokens, 4), device="cuda"), torch.empty((n_tokens, 4, 4), device="cuda")
    ctx.cmd_hc_pre(x, dev(fn), dev(scale), dev(base), red, post, comb, iters=iters, hc_eps=eps)
    torch.cuda.synchronize()
    r_ref, p_ref, c_ref = oracle.hc_pre(x.cpu().numpy(), fn, scale, base, iters=iters, hc_eps=eps)
    close_coeff(post.cpu().numpy(), p_ref)
    close_coeff(comb.cpu().numpy(), c_ref)
    close_streams(red.cpu().numpy(), r_ref, False)
