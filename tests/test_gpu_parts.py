"""Device code of the library by itself, built here with its source (GPU)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from colormlm_b200 import _lib as L
from colormlm_b200 import build, synth

from .test_gpu_parity import dev, dev_page, make_layer

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
NO_SUM = 0xFFFFFFFF   # kNoSum of s14_internal.h


@pytest.fixture(scope="module")
def part(tmp_path_factory):
    """part(name): device_parts.cu built with that part of it."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    built = {}

    def get(name):
        if name not in built:
            out = str(tmp_path_factory.mktemp("parts") / (name + ".so"))
            subprocess.run([build._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                            "-I" + build.CSRC, "-DPART_" + name, "-o", out, os.path.join(HERE, "device_parts.cu")], check=True)
            built[name] = C.CDLL(out)
        return built[name]

    return get


class BranchPost(C.Structure):
    _fields_ = [("branch_out", C.c_void_p), ("residual", C.c_void_p), ("post", C.c_void_p), ("comb", C.c_void_p), ("merged", C.c_void_p),
                ("done", C.c_bool)]


def ptr(t):
    return C.c_void_p(t.data_ptr())


def handed_sums(hidden):
    """A layer kernel's sums, and what it left of them: in two runs of 100 rows it gave up."""
    sums = torch.randn(hidden, device="cuda")
    left = torch.ones(hidden, dtype=torch.bool, device="cuda")
    left[300:400] = left[hidden - 100:] = False
    return sums, left


def given(sums, left):
    return torch.where(left, sums.view(torch.int32), torch.full_like(sums, 0).view(torch.int32) - 1).view(torch.float32)


def outputs(hidden, fill):
    g = synth.rng(4)
    keep = [torch.full((hidden,), fill, dtype=torch.bfloat16, device="cuda"), dev(synth.hc_streams(g, 1, hidden)[0]).to(torch.bfloat16),
            dev(g.uniform(0.2, 1.8, 4).astype(np.float32)), dev(g.uniform(0.05, 0.6, (4, 4)).astype(np.float32)),
            torch.full((4, hidden), fill, dtype=torch.bfloat16, device="cuda")]
    return BranchPost(*[t.data_ptr() for t in keep], False), keep


@pytest.mark.parametrize("with_post", [False, True])
def test_fp8_expert_behind_a_layer_kernel_that_gave_up(part, with_post):
    """Rows without a sum get no result, whatever lay there before; the sums that were taken are marked as taken."""
    lib, hidden, inter = part("HANDED"), 2048, 1024
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert lib.no_sum() & 0xFFFFFFFF == NO_SUM
    page = dev_page(make_layer(7, hidden, inter, 1, L.PAGE_FP8)[2], hidden, inter, L.PAGE_FP8)
    x, h = torch.randn(hidden, device="cuda"), torch.empty(inter, device="cuda")
    sums, left = handed_sums(hidden)

    def run(routed):
        y = torch.full((hidden,), 7.0, device="cuda")
        post, keep = outputs(hidden, 7.0)
        assert lib.fp8_expert(sms, ptr(x), ptr(page), ptr(h), ptr(routed), ptr(y), hidden, inter, C.byref(post) if with_post else None) == 0
        torch.cuda.synchronize()
        assert (routed.view(torch.int32) == -1).all()
        return [keep[0], keep[4]] if with_post else [y]

    for got, want in zip(run(given(sums, left)), run(sums.clone())):
        assert torch.equal(got[..., left], want[..., left]) and (got[..., ~left] == 7.0).all() and (want[..., ~left] != 7.0).any()


def test_end_of_the_executors_step_behind_a_layer_that_gave_up(part):
    lib, hidden = part("BRANCH"), 2048
    sums, left = handed_sums(hidden)

    def run(y):
        post, keep = outputs(hidden, 7.0)
        assert lib.branch_post(hidden, ptr(y), C.byref(post)) == 0
        torch.cuda.synchronize()
        assert (y.view(torch.int32) == -1).all()
        return [keep[0], keep[4]]

    for got, want in zip(run(given(sums, left)), run(sums.clone())):
        assert torch.equal(got[..., left], want[..., left]) and (got[..., ~left] == 7.0).all() and (want[..., ~left] != 7.0).any()


def test_greedy_token_of_either_cluster(part):
    """Clusters of sixteen, and the eight that every device takes where sixteen are refused: the same token."""
    lib = part("GREEDY")
    assert [lib.cluster_of(n) for n in (16, 15, 8, 0)] == [16, 8, 8, 8]
    for vocab in (1, 5, 4095, 129280):
        logits = torch.randint(-50, 50, (vocab + 1,), device="cuda").float()   # (many ties)
        for x in (logits[:vocab], logits[1:]):
            want, got = int((x == x.max()).nonzero()[0]), torch.empty(2, dtype=torch.int64, device="cuda")
            for k, cluster in enumerate((8, 16)):
                assert lib.greedy(cluster, ptr(x), vocab, ptr(got[k:])) == 0
            torch.cuda.synchronize()
            assert got.tolist() == [want, want]


def test_what_the_fast_forms_settle_is_exact(part):
    """The official blocks' SwiGLU over every BF16 gate, and their sums of six digit shares, many of them at BF16 ties: where the fast
    form says that it settles the value, it is the exact form's."""
    lib = part("QUICK")
    g = torch.Generator().manual_seed(1)
    ups = torch.cat([torch.tensor([0.0, -0.0, 1.0, 9.9375, 10.0, 10.0625, -10.0, -12.0, 2.0 ** -120, -2.0 ** -60, 3e38]),
                     torch.randn(40, generator=g) * 4.0]).to(torch.bfloat16).float().cuda()
    weights = torch.cat([torch.tensor([1.0, 0.0, 1.5, 2.0 ** -100, 1e30]), torch.rand(11, generator=g)]).cuda()
    counts = torch.zeros(4, dtype=torch.int64, device="cuda")
    assert lib.swiglu(ptr(ups), len(ups), ptr(weights), len(weights), ptr(counts)) == 0
    assert lib.sums(64, ptr(counts[2:])) == 0
    torch.cuda.synchronize()
    swiglu, swiglu_wrong, sums, sums_wrong = counts.tolist()
    assert swiglu_wrong == 0 and sums_wrong == 0
    assert swiglu > 0.2 * 65536 * len(ups) * len(weights) and sums > 0.3 * 64 * 1024 * 256


def test_the_sinkhorn_rounds_quotient_is_the_division_operators(part):
    """Every mantissa of the divisor, dividends at random and next to ties: 1.2e9 quotients."""
    lib, wrong = part("QUOTIENT"), torch.zeros(1, dtype=torch.int64, device="cuda")
    assert lib.quotients(24, ptr(wrong)) == 0
    torch.cuda.synchronize()
    assert int(wrong) == 0
