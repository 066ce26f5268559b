"""Layers with the checkpoint's page kinds - routed MXFP4 experts, FP8 shared expert - on the path that runs the
shared expert by kernels of its own behind the tensor-core layer kernel (GPU), against the CPU oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import synth
from colormlm_b200.s14 import DecodeStack, S14Context, TokenRoute

from .test_gpu_parity import assert_pairwise_close, dev, dev_page, make_layer

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]
PATH = L.LAYER_PATH_TENSOR | L.LAYER_PATH_FP8_SHARED_KERNEL


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    c = S14Context(0)
    yield c
    c.close()


# every width of a lane's share of a row; one route and six
@pytest.mark.parametrize("hidden,inter,routed", [(1024, 4096, 6), (2048, 2048, 1), (4096, 1024, 6)])
def test_layer_and_executor_step_with_an_fp8_shared_expert(ctx, oracle, hidden, inter, routed):
    g, pages, shared = make_layer(71 + hidden + routed, hidden, inter, routed, L.PAGE_FP8)
    pages_dev, shared_dev = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter, L.PAGE_FP8)
    w = np.asarray([0.4, 0.3, 0.25, 0.2, 0.2, 0.15][:routed], np.float32)
    route = TokenRoute(list(range(routed)), w, [p.data_ptr() for p in pages_dev])
    x16 = dev(synth.activations(g, 1, hidden)[0]).to(torch.bfloat16)
    x = x16.float()
    want = oracle.moe_layer_acc64(x.cpu().numpy(), pages, w, shared, L.PAGE_FP8, hidden, inter)
    y = torch.empty(1, hidden, device="cuda")
    for _ in range(2):
        ctx.cmd_moe_layer(x[None], y, [route], shared_dev.data_ptr(), L.PAGE_FP8, hidden, inter)
        torch.cuda.synchronize()
        assert ctx.device_status() == 0 and ctx.last_layer_path == PATH
        assert_pairwise_close(oracle, y.cpu().numpy()[0], want)
    residual = dev(synth.hc_streams(g, 1, hidden)[0]).to(torch.bfloat16)
    post, comb = dev(g.uniform(0.2, 1.8, 4).astype(np.float32)), dev(g.uniform(0.05, 0.6, (4, 4)).astype(np.float32))
    state, branch = torch.empty_like(residual), torch.empty_like(x16)
    ctx.exec_routed_and_shared_moe_then_hc_post(x16, residual, post, comb, route, shared_dev.data_ptr(), L.PAGE_FP8, inter, state, branch)
    assert ctx.last_layer_path == PATH
    merged = torch.empty_like(residual)
    ctx.cmd_hc_post(branch[None], residual[None], post[None], comb[None], merged[None])
    torch.cuda.synchronize()
    assert torch.equal(branch, y[0].to(torch.bfloat16)) and torch.equal(state, merged)


def routed_layer(seed, hidden, inter, n_experts):
    """A routed layer with an FP8 shared page: host pages and router, and what the calls take."""
    g, pages, shared = make_layer(seed, hidden, inter, n_experts, L.PAGE_FP8)
    wr, bias = synth.router_weight_bf16(g, n_experts, hidden), synth.router_bias(g, n_experts)
    pd, sd = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter, L.PAGE_FP8)
    table = torch.tensor([p.data_ptr() for p in pd], dtype=torch.int64, device="cuda")
    x = synth.activations(g, 1, hidden)
    return pages, shared, wr, bias, x, (pd, sd), (dev(wr.view(np.int16)), dev(bias), table, sd.data_ptr(), L.PAGE_FP8, inter)


# the router inside the layer kernel: fewer experts than SMs, and two experts' rows for some CTAs
@pytest.mark.parametrize("hidden,inter,n_experts", [(1024, 2048, 7), (2048, 1024, 200), (4096, 2048, 24)])
def test_routed_layer_with_an_fp8_shared_expert(ctx, oracle, hidden, inter, n_experts):
    """The device call with and without outputs for the route, the call on host buffers and the bound one: the
    oracle's route, its layer, and the same bits from each."""
    pages, shared, wr, bias, x, keep, args = routed_layer(40 + n_experts, hidden, inter, n_experts)
    ids, wts = torch.empty(6, dtype=torch.int32, device="cuda"), torch.empty(6, device="cuda")
    y, again = torch.empty(1, hidden, device="cuda"), torch.empty(1, hidden, device="cuda")
    for out, outs in ((y, (ids, wts)), (again, ())):
        ctx.cmd_routed_moe_layer(dev(x)[0], *args, out, *outs)
        torch.cuda.synchronize()
        assert ctx.device_status() == 0 and ctx.last_layer_path == PATH
    rid, rw, _, _ = oracle.router(x[0], wr, bias, 0, 6, 1.0)
    assert np.array_equal(ids.cpu().numpy(), rid) and np.array_equal(wts.cpu().numpy().view(np.uint32), rw.view(np.uint32))
    want = oracle.moe_layer_acc64(x[0], [pages[i] for i in rid], rw, shared, L.PAGE_FP8, hidden, inter)
    assert_pairwise_close(oracle, y.cpu().numpy()[0], want)
    assert torch.equal(y, again)
    bound = ctx.bind_routed_moe_layer_host(*args)
    for call in (lambda *a: bound(x[0], *a), lambda out, i, w: ctx.routed_moe_layer_host(x[0], out, *args, i, w)):
        host, host_ids, host_w = np.full(hidden, np.nan, np.float32), np.full(6, -1, np.int32), np.zeros(6, np.float32)
        call(host, host_ids, host_w)
        assert np.array_equal(host.view(np.uint32), y.cpu().numpy()[0].view(np.uint32))
        assert np.array_equal(host_ids, rid) and np.array_equal(host_w.view(np.uint32), rw.view(np.uint32))


def test_kernel_timing_leaves_the_layer_on_its_path(ctx):
    hidden, inter = 1024, 2048
    _, _, _, _, x, keep, args = routed_layer(12, hidden, inter, 16)
    dx, plain, timed = dev(x), torch.empty(1, hidden, device="cuda"), torch.empty(1, hidden, device="cuda")
    ctx.cmd_routed_moe_layer(dx[0], *args, plain)
    path = ctx.last_layer_path
    ctx.set_kernel_timing(True)
    try:
        ctx.cmd_routed_moe_layer(dx[0], *args, timed)
        times, calls = ctx.kernel_times()
    finally:
        ctx.set_kernel_timing(False)
    assert path == PATH and ctx.last_layer_path == path and torch.equal(plain, timed)
    assert calls == 1 and times["up"] > 0.0  # (one mark after all of the layer's kernels)


# elements past a 16-byte boundary: 2-, 4- and 8-byte ones; the state and the branch lie there too
@pytest.mark.parametrize("offset", [1, 2, 4])
@pytest.mark.parametrize("kind", [L.PAGE_FP8, L.PAGE_MXFP4])
def test_executor_step_of_buffers_on_any_boundary(ctx, kind, offset):
    hidden, inter, routed = 2048, 1024, 2
    g, pages, shared = make_layer(5, hidden, inter, routed, kind)
    pages_dev, shared_dev = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter, kind)
    route = TokenRoute(list(range(routed)), np.asarray([0.7, 0.4], np.float32), [p.data_ptr() for p in pages_dev])
    x, residual = (dev(a).to(torch.bfloat16) for a in (synth.activations(g, 1, hidden)[0], synth.hc_streams(g, 1, hidden)[0]))
    post, comb = dev(g.uniform(0.2, 1.8, 4).astype(np.float32)), dev(g.uniform(0.05, 0.6, (4, 4)).astype(np.float32))

    def moved(a):
        big = torch.empty(a.numel() + offset, dtype=a.dtype, device="cuda")
        big[offset:] = a.reshape(-1)
        return big[offset:].view(a.shape)

    outs = []
    for place in (lambda a: a, moved):
        state, branch = place(torch.zeros_like(residual)), place(torch.zeros_like(x))
        ctx.exec_routed_and_shared_moe_then_hc_post(place(x), place(residual), post, comb, route, shared_dev.data_ptr(), kind, inter,
                                                    state, branch)
        outs.append((state, branch))
    torch.cuda.synchronize()
    assert ctx.device_status() == 0 and torch.count_nonzero(outs[0][1]) > 0
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("residual", [True, False])
def test_stack_with_fp8_shared_experts(ctx, oracle, residual):
    """A chain of layers stays on the F32 register kernels, whose sums it is to reproduce: a layer's difference of
    4e-7 grows along the chain."""
    hidden, inter, n_experts, n_layers = 1024, 1024, 24, 3
    host, layers, keep = [], [], []
    for l in range(n_layers):
        g, pages, shared = make_layer(900 + l, hidden, inter, n_experts, L.PAGE_FP8)
        wr, bias = synth.router_weight_bf16(g, n_experts, hidden), synth.router_bias(g, n_experts)
        host.append((pages, shared, wr, bias))
        pd, sd = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter, L.PAGE_FP8)
        keep.append((pd, sd))
        layers.append({"wr": dev(wr.view(np.int16)), "bias": dev(bias), "shared": sd.data_ptr(),
                       "table": torch.tensor([p.data_ptr() for p in pd], dtype=torch.int64, device="cuda"),
                       "ids": torch.empty(6, dtype=torch.int32, device="cuda"),
                       "weights": torch.empty(6, device="cuda"), "y": torch.empty(hidden, device="cuda")})
    stack = DecodeStack(ctx, layers, inter=inter, shared_kind=L.PAGE_FP8, residual=residual)
    x = synth.activations(synth.rng(5), 1, hidden)[0] * np.float32(0.25)
    h = dev(x)
    try:
        stack.cmd_decode(h, h)  # in place
        torch.cuda.synchronize()
        assert ctx.device_status() == 0 and ctx.last_layer_path == L.LAYER_PATH_F32 | L.LAYER_PATH_ROUTER_KERNEL
        cur = x
        for (pages, shared, wr, bias), ly in zip(host, layers):
            rid, rw, _, _ = oracle.router(cur, wr, bias, 0, 6, 1.0)
            assert np.array_equal(ly["ids"].cpu().numpy(), rid)
            want = oracle.moe_layer_acc64(cur, [pages[i] for i in rid], rw, shared, L.PAGE_FP8, hidden, inter)
            assert_pairwise_close(oracle, ly["y"].cpu().numpy(), want)
            got = ly["y"].cpu().numpy()
            cur = (cur + got).astype(np.float32) if residual else got
        assert np.array_equal(h.cpu().numpy(), cur)
    finally:
        stack.close()


@pytest.mark.parametrize("kind", [L.PAGE_FP8, L.PAGE_MXFP4])
def test_calls_in_place_and_one_after_another(ctx, kind):
    """The layer's y in place of x; the executor's state in place of the residual and its branch in place of the token; steps in a
    row, each of which reads what the one before left."""
    hidden, inter, routed = 2048, 2048, 3
    g, pages, shared = make_layer(55, hidden, inter, routed, kind)
    pages_dev, shared_dev = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter, kind)
    route = TokenRoute(list(range(routed)), np.asarray([0.3, 0.2, 0.1], np.float32), [p.data_ptr() for p in pages_dev])
    x = dev(synth.activations(g, 1, hidden))
    want, got = x.clone(), x.clone()
    for _ in range(3):
        y = torch.empty_like(want)
        ctx.cmd_moe_layer(want * 0.01, y, [route], shared_dev.data_ptr(), kind, hidden, inter)
        want = y
        got *= 0.01
        ctx.cmd_moe_layer(got, got, [route], shared_dev.data_ptr(), kind, hidden, inter)
    assert torch.equal(got, want)
    residual = dev(synth.hc_streams(g, 1, hidden)[0]).to(torch.bfloat16)
    post, comb = dev(g.uniform(0.2, 1.8, 4).astype(np.float32)), dev(g.uniform(0.05, 0.6, (4, 4)).astype(np.float32))
    t, s, t2, s2 = x[0].to(torch.bfloat16), residual, x[0].to(torch.bfloat16), residual.clone()
    for _ in range(3):
        branch, state = torch.empty_like(t), torch.empty_like(s)
        ctx.exec_routed_and_shared_moe_then_hc_post(t, s, post, comb, route, shared_dev.data_ptr(), kind, inter, state, branch)
        ctx.exec_routed_and_shared_moe_then_hc_post(t2, s2, post, comb, route, shared_dev.data_ptr(), kind, inter, s2, t2)
        t, s = branch * 0.01, state
        t2 *= 0.01
    torch.cuda.synchronize()
    assert ctx.device_status() == 0 and torch.equal(t, t2) and torch.equal(s, s2) and torch.isfinite(s.float()).all()
