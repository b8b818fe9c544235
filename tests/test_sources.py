"""Rules of the instruction set that a GPU run cannot show to be kept, read off the sources (no GPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "juliavision_b200", "csrc")


def sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, re.sub(r"//[^\n]*", "", f.read())


def test_cluster_barriers_bring_the_warp_together_first():
    """barrier.cluster.arrive.aligned is undefined when the lanes of a warp arrive apart, and its callers come out of loops
    whose trip counts differ by lane: whoever issues it converges the warp in the statement before."""
    seen = 0
    for name, text in sources():
        for m in re.finditer(r"[^;{}]*[;{}]\s*asm volatile\(\s*\"[^;]*barrier\.cluster\.arrive", text):
            assert m.group(0).split(";")[0].strip() == "__syncwarp()", (name, m.group(0))
            seen += 1
        assert len(re.findall(r"barrier\.cluster\.arrive", text)) == (1 if name == "ptx.cuh" else 0), name
    assert seen == 1


def test_one_cta_of_a_worker_writes_the_timeline():
    """Every CTA of a worker (a pair, or a cluster along K) runs the lines that record events; only one may write."""
    text = dict(sources())["gemm.cu"]
    writes = [m.start() for m in re.finditer(r"p\.trace\[[^\]]*\] =", text)]
    assert len(writes) == 3
    for at in writes:
        guard = text[text.rindex("if (", 0, at):at]
        assert all(c in guard for c in ("rank == 0", "(!KSPLIT || cluster_ctarank() == 0)", "worker")), guard


def test_what_the_runtime_is_asked_once_is_asked_of_the_right_device_by_one_thread():
    """The K split's room is kept per device and asked for by the plan entry too, with any device current and from any
    thread: the device is set before the question, and the answer is published whole."""
    text = dict(sources())["gemm.cu"]
    ask = text[text.index("static KsplitRoom ksplit_ask("):]
    assert 0 < ask.index("cudaSetDevice(ctx->device)") < ask.index("cudaFuncSetAttribute(") < ask.index("cudaOccupancyMaxActiveClusters(")
    room = text[text.index("ksplit_room(b200_ctx* ctx) {"):]
    assert "std::call_once(" in room[:room.index("\n}\n")]
