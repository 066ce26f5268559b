"""Operators behind a kernel of the caller that lets its dependents start early and writes their operands late, weights
and pages included: the operator reads what that kernel leaves (GPU)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import synth
from colormlm_b200.s14 import MoeBlock, S14Context, S14MatvecShape, TokenRoute

from .test_gpu_parity import dev, dev_page, make_layer

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_lib")]

# Copies the *n 4-byte words of src to dst about 100 us after its dependents may start (150 naps of at most 2 x 700 ns:
# it waits for nothing).
SOURCE = """
extern "C" __global__ void write_late(const unsigned int *src, unsigned int *dst, const unsigned long long *n) {
    asm volatile("griddepcontrol.launch_dependents;");
    for (int i = 0; i < 150; ++i) __nanosleep(700);
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < *n; i += gridDim.x * (unsigned long long)blockDim.x)
        dst[i] = src[i];
}
"""


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    c = S14Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def write_late(ctx):
    kernel = torch.cuda._compile_kernel(SOURCE, "write_late")

    def run(src, dst):
        assert src.nbytes == dst.nbytes and src.nbytes % 4 == 0 and src.is_contiguous() and dst.is_contiguous()
        kernel((64, 1, 1), (256, 1, 1), (src, dst, torch.tensor([src.nbytes // 4], dtype=torch.int64, device="cuda")))

    return run


def _codes(*shape, high=256):
    return torch.randint(0, high, shape, dtype=torch.uint8, device="cuda")


def _mxfp4(ctx):
    n, k = 300, 1024
    w, s, x, y = _codes(n * k // 2), _codes(n * k // 32, high=4) + 119, torch.randn(k, device="cuda"), torch.empty(n, device="cuda")
    op = ctx.pipelines.bind_mxfp4(S14MatvecShape(n, k), x, w, s, y)
    return [w, s], (lambda keep=x: ctx.pipelines.cmd_mxfp4_matvec(op)), y  # (a bound operator holds addresses alone)


def _fp8(ctx):
    n, k = 256, 1024
    w, s, x, y = _codes(n * k, high=127), _codes(n // 128 * k // 128, high=4) + 119, torch.randn(k, device="cuda"), torch.empty(n, device="cuda")
    op = ctx.pipelines.bind_fp8(S14MatvecShape(n, k), x, w, s, y)
    return [w, s], (lambda keep=x: ctx.pipelines.cmd_fp8_matvec(op)), y


def _head(ctx):
    w, x, y = torch.randn(700, 1024, device="cuda").to(torch.bfloat16), torch.randn(2, 1024, device="cuda"), torch.empty(2, 700, device="cuda")
    return [w], (lambda: ctx.cmd_head_logits(x, w.view(torch.int16), y)), y


def _site(tokens):
    def make(ctx):
        h = 1024
        x = torch.randn(tokens, 4, h, device="cuda")
        fn, scale, base = torch.randn(24, 4 * h, device="cuda") * 0.02, torch.rand(3, device="cuda"), torch.rand(24, device="cuda")
        red, post, comb = torch.empty(tokens, h, device="cuda"), torch.empty(tokens, 4, device="cuda"), torch.empty(tokens, 4, 4, device="cuda")
        return [fn, scale, base], (lambda: ctx.cmd_hc_pre(x, fn, scale, base, red, post, comb)), red

    return make


def _layer(ctx):
    h, i, routed = 1024, 1024, 2
    g, pages, shared = make_layer(3, h, i, routed, L.PAGE_FP8)
    pages_dev, shared_dev = [dev_page(p, h, i) for p in pages], dev_page(shared, h, i, L.PAGE_FP8)
    route = TokenRoute(list(range(routed)), np.asarray([0.7, 0.4], np.float32), [p.data_ptr() for p in pages_dev])
    x, y = dev(synth.activations(g, 1, h)), torch.empty(1, h, device="cuda")
    return pages_dev + [shared_dev], (lambda: ctx.cmd_moe_layer(x, y, [route], shared_dev.data_ptr(), L.PAGE_FP8, h, i)), y


def _exec(ctx):
    # (the shared expert's first launch reads the token and its page without a wait of its own)
    h, i, routed = 1024, 2048, 2
    g, pages, shared = make_layer(6, h, i, routed, L.PAGE_FP8)
    pages_dev, shared_dev = [dev_page(p, h, i) for p in pages], dev_page(shared, h, i, L.PAGE_FP8)
    route = TokenRoute(list(range(routed)), np.asarray([0.7, 0.4], np.float32), [p.data_ptr() for p in pages_dev])
    x, residual = (dev(a).to(torch.bfloat16) for a in (synth.activations(g, 1, h)[0], synth.hc_streams(g, 1, h)[0]))
    post, comb = torch.rand(4, device="cuda") + 0.2, torch.rand(4, 4, device="cuda")
    state = torch.empty_like(residual)
    return [x, residual, shared_dev, pages_dev[0], post, comb], (lambda keep=pages_dev: ctx.exec_routed_and_shared_moe_then_hc_post(
        x, residual, post, comb, route, shared_dev.data_ptr(), L.PAGE_FP8, i, state, None)), state


def _routed_layer(ctx):
    h, i, experts = 1024, 1024, 9
    g, pages, shared = make_layer(8, h, i, experts, L.PAGE_FP8)
    pages_dev, shared_dev = [dev_page(p, h, i) for p in pages], dev_page(shared, h, i, L.PAGE_FP8)
    table = torch.tensor([p.data_ptr() for p in pages_dev], dtype=torch.int64, device="cuda")
    wr, bias = dev(synth.router_weight_bf16(g, experts, h).view(np.int16)), dev(synth.router_bias(g, experts))
    x, y = dev(synth.activations(g, 1, h))[0], torch.empty(1, h, device="cuda")
    return [x, wr, bias, shared_dev] + pages_dev, (lambda: ctx.cmd_routed_moe_layer(x, wr, bias, table, shared_dev.data_ptr(), L.PAGE_FP8, i, y)), y


def _block(tokens, official, routed):
    """The block calls: their first digits launch reads x in front of its wait, behind the router's launches (or the copies of
    the host's routes), which have waited."""
    def make(ctx):
        h, i, experts = 1024, 512, 8
        g, pages, shared = make_layer(4, h, i, experts, L.PAGE_MXFP4)
        pages_dev, shared_dev = [dev_page(p, h, i) for p in pages], dev_page(shared, h, i)
        table = torch.tensor([p.data_ptr() for p in pages_dev], dtype=torch.int64, device="cuda")
        x, y = dev(synth.activations(g, tokens, h)), torch.empty(tokens, h, device="cuda")
        wr, bias = dev(synth.router_weight_bf16(g, experts, h).view(np.int16)), dev(synth.router_bias(g, experts))
        blk = MoeBlock(ctx, h, i, tokens)
        blk.set_semantics(official)
        if routed:
            return [x, wr, bias, pages_dev[0], shared_dev], (lambda keep=pages_dev: blk.cmd_routed_moe_block(x, wr, bias, table, shared_dev.data_ptr(), y)), y
        routes = [TokenRoute([e, e + 2], np.asarray([0.7, 0.4], np.float32), [pages_dev[e].data_ptr(), pages_dev[e + 2].data_ptr()])
                  for e in (t % 6 for t in range(tokens))]
        return [x, pages_dev[0], shared_dev], (lambda keep=pages_dev: blk.cmd_moe_block(x, y, routes, shared_dev.data_ptr())), y

    return make


@pytest.mark.parametrize("make", [_mxfp4, _fp8, _head, _site(1), _site(20), _layer, _exec, _routed_layer, _block(3, False, True), _block(20, False, True),
                                  _block(3, True, True), _block(70, True, True), _block(5, False, False)],
                         ids=["mxfp4", "fp8", "head", "site", "site20", "fp8_shared_layer", "executor_step", "fp8_shared_routed_layer", "block", "block20", "block_official",
                              "block70_official", "block_host_routes"])
def test_operands_written_late_by_a_kernel_that_lets_dependents_start(ctx, write_late, make):
    torch.manual_seed(1)
    operands, call, y = make(ctx)
    call()
    torch.cuda.synchronize()
    want, new = y.clone(), [o.clone() for o in operands]
    assert torch.count_nonzero(want) > 0
    with torch.cuda.stream(torch.cuda.Stream()):
        for o, n in zip(operands, new):   # each operand on its own, wrong until the late kernel has run
            o.zero_()
            y.zero_()
            torch.cuda.synchronize()
            write_late(n, o)
            call()
            torch.cuda.synchronize()
            assert torch.equal(y, want)
    assert ctx.device_status() == 0


def test_streams_named_in_every_form(ctx):
    x, w, want = torch.randn(3, 512, device="cuda"), torch.rand(512, device="cuda"), torch.empty(3, 512, device="cuda")
    ctx.cmd_rms_norm(x, w, want)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for stream in (side, side.cuda_stream, ctypes.c_void_p(side.cuda_stream), None):
        out = torch.zeros_like(want)
        torch.cuda.synchronize()
        ctx.cmd_rms_norm(x, w, out, stream=stream)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
