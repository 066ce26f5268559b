"""What the two CTAs of a block kernel's pair (csrc/s14_moe_pair.cu) hand over in tensor memory - scale codes that either one's threads have stored,
accumulators that the first one's operations overwrite - goes through barriers at cluster scope, with the tensor operations' fences on either
side.  No run can show that one of these is missing - the hardware may be in order all the same - so the source is looked at."""
import os
import re

from colormlm_b200 import build


def source():
    with open(os.path.join(build.CSRC, "s14_moe_pair.cu")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body(text, name):
    return re.search(name + r"\([^)]*\) \{(.*?)\n\}", text, re.S).group(1)


def test_tensor_memory_is_handed_over_at_cluster_scope():
    text = source()
    for barrier, looks in (("kPBarRows", ["mbar_test_cluster", "mbar_wait_cluster"]), ("kPBarAccFree", ["mbar_test_cluster", "mbar_wait_cluster"])):
        seen = re.findall(r"(\w+)\(bar\(" + barrier, text)
        for alias in re.findall(r"(\w+) = bar\(" + barrier, text):
            seen += re.findall(r"(\w+)\(" + alias + r"\b", text)
        assert sorted(n for n in seen if n != "first_cta") == looks
        base = re.search(r"(\w+) = first_cta\(bar\(" + barrier + r"\)\)", text).group(1)
        arrives = [m.start() for m in re.finditer(r"mbar_arrive_remote\(" + base + r"\b", text)]
        assert len(arrives) == 1 and len(re.findall(r"\w+\(" + base + r"\b", text)) == 1
        assert re.search(r"fence_before\(\);\s+__syncwarp\(\);\s+if \(lane == 0\) $", text[:arrives[0]])
    assert "mbarrier.arrive.relaxed.cluster.shared::cluster" in body(text, "mbar_arrive_remote")
    for name in ("mbar_test_cluster", "mbar_wait_cluster"):
        assert ".relaxed.cluster." in body(text, name)
    # behind either look: fence_after in front of the operations
    issuing = text[text.index("warp == kPMmaWarp) {\n            if (rank == 0u)"):text.index("pair_commit(bar(kPBarAccDone")]
    assert issuing.count("fence_after();") == 2
