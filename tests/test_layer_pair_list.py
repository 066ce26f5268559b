"""The deal of a layer's work where CTAs run in pairs: up items that do not go round evenly are shared by a pair along K.
The lists on the CPU, the layer's results where items are shared against the double-accumulated oracle (GPU)."""
import ctypes as C

import numpy as np
import pytest

from colormlm_b200 import _lib as L
from colormlm_b200 import synth

DOWN, HALF, SECOND = 1 << 31, 1 << 30, 1 << 29


def pair_list(block, n_ctas, n_jobs, n_early, hidden, inter, cap=1024):
    items = (C.c_uint32 * cap)()
    count = C.c_uint32(0)
    L.check(L.lib().s14_layer_pair_list(block, n_ctas, n_jobs, n_early, hidden, inter, items, cap, C.byref(count)))
    return [int(v) for v in items[:count.value]]


@pytest.mark.parametrize("n_early", [0, 1])
@pytest.mark.parametrize("n_ctas", [148, 132, 64, 2])
@pytest.mark.parametrize("n_jobs", [1, 2, 5, 6, 7])
@pytest.mark.parametrize("hidden,inter", [(4096, 2048), (2048, 1024), (1024, 1024), (1024, 4096), (512, 512), (1536, 2048)])
def test_every_item_once_or_as_two_halves_of_a_pair(cuda_lib, n_ctas, n_jobs, hidden, inter, n_early):
    S, RT = inter // 64, hidden // 128
    lists = [pair_list(b, n_ctas, n_jobs, n_early, hidden, inter) for b in range(n_ctas)]
    seen = {}
    for b, items in enumerate(lists):
        kinds = [(it & DOWN) != 0 for it in items]
        assert kinds == sorted(kinds)                       # up items first
        downs = [(it >> 8 & 0xFF) * RT + (it & 0xFF) for it in items if it & DOWN]
        assert downs == sorted(downs)                       # in the order of the jobs
        early = [(it >> 8 & 0xFF) < n_early for it in items if not it & DOWN]
        assert early == sorted(early, reverse=True)
        halves = [it for it in items if it & HALF]
        assert len(halves) <= 1
        for it in halves:                                   # its other half is the partner's
            assert it ^ SECOND in lists[b ^ 1] and (it >> 8 & 0xFF) >= n_early and hidden // 256 % 4 == 0
        for it in items:
            assert it not in seen
            seen[it] = b
    whole = {it & ~(HALF | SECOND) for it in seen}
    assert whole == {j << 8 | i for j in range(n_jobs) for i in range(S)} | {DOWN | j << 8 | i for j in range(n_jobs) for i in range(RT)}
    assert len(seen) == len(whole) + sum(1 for it in seen if it & SECOND)


def test_the_benchmark_layer_shares_what_does_not_go_round(cuda_lib):
    """192 routed up items of 16 units on 148 CTAs: 44 are shared, no CTA has more than 24 units of the up projection."""
    lists = [pair_list(b, 148, 7, 1, 4096, 2048) for b in range(148)]
    assert sum(1 for items in lists for it in items if it & SECOND) == 44
    units = [sum(8 if it & HALF else 16 for it in items if not it & DOWN and it >> 8 & 0xFF) for items in lists]
    assert max(units) == 24 and min(units) == 16
    assert max(u + sum(8 for it in items if it & DOWN) for u, items in zip(units, lists)) <= 40


def test_long_down_items_go_to_the_pairs_that_share(cuda_lib):
    """Three given jobs of 4096 x 4096 on 148 CTAs: a down item is as long as a whole up item, and after one of them a CTA without
    a half has 32 units where the others have 24, so the others come first when the rest goes round."""
    lists = [pair_list(b, 148, 3, 0, 4096, 4096) for b in range(148)]
    assert any(it & HALF for items in lists for it in items)
    assert max(sum(8 if it & HALF else 16 for it in items) for items in lists) == 40


def test_rejects_bad_arguments(cuda_lib):
    count = C.c_uint32(0)
    for args in ((148, 148, 7, 0, 4096, 2048), (0, 0, 7, 0, 4096, 2048), (0, 147, 7, 0, 4096, 2048), (0, 148, 7, 0, 4000, 2048)):
        with pytest.raises(L.S14Error):
            L.check(L.lib().s14_layer_pair_list(*args, None, 0, C.byref(count)))


@pytest.fixture(scope="module")
def ctx():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from colormlm_b200.s14 import S14Context

    c = S14Context(0)
    yield c
    c.close()


# (with 148 CTAs; a launch is in pairs where hidden is 4096) every up item shared; 4 of 448; 44 of 192, no shared expert; 12 of 160
@pytest.mark.gpu
@pytest.mark.parametrize("hidden,inter,routed,shared", [(4096, 1024, 2, True), (4096, 4096, 6, True), (4096, 2048, 6, False),
                                                        (4096, 2048, 4, True)])
def test_layer_with_shared_items(cuda_lib, ctx, oracle, hidden, inter, routed, shared):
    from .test_gpu_parity import assert_pairwise_close, dev_page, make_layer, run_layer

    g, pages, sh = make_layer(91 + hidden + inter, hidden, inter, routed, L.PAGE_MXFP4)
    x = synth.activations(g, 1, hidden)
    w = np.asarray([0.4, 0.3, 0.25, 0.2, 0.2, 0.15][:routed], np.float32)
    want = oracle.moe_layer_acc64(x[0], pages, w, sh if shared else None, 0 if shared else 2, hidden, inter)
    pages_dev, shared_dev = [dev_page(p, hidden, inter) for p in pages], dev_page(sh, hidden, inter) if shared else None
    for _ in range(2):
        y = run_layer(ctx, x, pages_dev, shared_dev, [(list(range(routed)), w)], L.PAGE_MXFP4, hidden, inter)[0]
        assert_pairwise_close(oracle, y, want)


# long down items: the rest of them goes round the pairs that share first
@pytest.mark.gpu
@pytest.mark.parametrize("routed,shared", [(2, True), (3, False)])
def test_layer_with_shared_items_and_long_down_items(cuda_lib, ctx, oracle, routed, shared):
    test_layer_with_shared_items(cuda_lib, ctx, oracle, 4096, 4096, routed, shared)


@pytest.mark.gpu
def test_stack_with_shared_items_and_early_ones(cuda_lib, ctx, oracle):
    """Three chained layers of 4096 x 2048: the shared expert's items run early, 44 of the 192 routed ones are shared, in
    every layer (the barriers' phases)."""
    torch = pytest.importorskip("torch")
    from colormlm_b200.s14 import DecodeStack

    from .test_gpu_parity import assert_chain_close, dev, dev_page, make_layer, oracle_stack

    hidden, inter, n_experts = 4096, 2048, 7
    host, layers, keep = [], [], []
    for l in range(3):
        g, pages, shared = make_layer(9300 + l, hidden, inter, n_experts, L.PAGE_MXFP4)
        wr, bias = synth.router_weight_bf16(g, n_experts, hidden), synth.router_bias(g, n_experts)
        host.append({"wr": wr, "bias": bias, "shared": shared, "page": (lambda e, p=pages: p[e])})
        pd, sd = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter)
        keep.append((pd, sd))
        layers.append({"wr": dev(wr.view(np.int16)), "bias": dev(bias), "shared": sd.data_ptr(),
                       "table": torch.tensor([p.data_ptr() for p in pd], dtype=torch.int64, device="cuda"),
                       "ids": torch.empty(6, dtype=torch.int32, device="cuda"), "weights": torch.empty(6, device="cuda"),
                       "y": torch.empty(hidden, device="cuda")})
    stack = DecodeStack(ctx, layers, inter=inter, residual=True)
    try:
        for seed in (9401, 9402):
            x = synth.activations(synth.rng(seed), 1, hidden)[0] * np.float32(0.25)
            want_h, want_y, routes = oracle_stack(oracle, x, host, hidden, inter, True, True)
            h = torch.full((hidden,), float("nan"), device="cuda")
            stack.cmd_decode(dev(x), h)
            torch.cuda.synchronize()
            assert ctx.device_status() == 0
            for l in range(3):
                assert np.array_equal(layers[l]["ids"].cpu().numpy(), routes[l][0])
                assert_chain_close(oracle, layers[l]["y"].cpu().numpy(), want_y[l], ("layer", l))
            assert_chain_close(oracle, h.cpu().numpy(), want_h, "final token")
    finally:
        stack.close()


@pytest.mark.gpu
@pytest.mark.parametrize("call,hidden,inter,routed,paired", [("layer", 4096, 1024, 2, True), ("layer", 4096, 4096, 2, True), ("layer", 4096, 2048, 6, False),
                                                             ("layer", 2048, 2048, 6, False), ("routed", 4096, 2048, 6, False),
                                                             ("stack", 4096, 2048, 6, True), ("stack", 2048, 2048, 6, False)])
def test_which_launches_run_in_pairs(cuda_lib, ctx, call, hidden, inter, routed, paired):
    """By the mark of a traced launch (on 148 SMs): without it the tests above would pass on the kernel without pairs."""
    torch = pytest.importorskip("torch")
    from colormlm_b200.s14 import DecodeStack

    from .test_gpu_parity import dev, dev_page, make_layer, run_layer

    if ctx.sm_count != 148:
        pytest.skip("the deals are those of 148 SMs")
    g, pages, shared = make_layer(55, hidden, inter, 7, L.PAGE_MXFP4)
    x, w = synth.activations(g, 1, hidden), np.full(routed, 0.25, np.float32)
    pd, sd = [dev_page(p, hidden, inter) for p in pages], dev_page(shared, hidden, inter)
    wr, table = dev(synth.router_weight_bf16(g, 7, hidden).view(np.int16)), torch.tensor([p.data_ptr() for p in pd], dtype=torch.int64, device="cuda")
    ctx.set_layer_trace(True)
    try:
        if call == "layer":
            run_layer(ctx, x, pd, sd, [(list(range(routed)), w)], L.PAGE_MXFP4, hidden, inter)
        elif call == "routed":
            ctx.cmd_routed_moe_layer(dev(x)[0], wr, None, table, sd.data_ptr(), L.PAGE_MXFP4, inter, torch.empty(1, hidden, device="cuda"))
        else:
            layer = {"wr": wr, "bias": None, "shared": sd.data_ptr(), "table": table, "ids": None, "weights": None, "y": None}
            stack = DecodeStack(ctx, [layer, layer], inter=inter, residual=True)
            h = dev(x)[0]
            stack.cmd_decode(h * 0.25, h)
            torch.cuda.synchronize()
            stack.close()
        torch.cuda.synchronize()
        mark = ctx.read_layer_trace()[:, 15]
    finally:
        ctx.set_layer_trace(False)
    assert ctx.device_status() == 0 and len(mark) == 148
    assert set(int(m) >> 24 for m in mark if m) == {int(paired)} and (mark != 0).sum() > 100
