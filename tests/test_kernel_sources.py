"""Rules of the kernel sources whose violation shows only as a rare hang, checked on the text (no GPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")


def _read(*parts):
    with open(os.path.join(CSRC, *parts)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_cluster_barriers_bring_the_warp_together_first():
    """`barrier.cluster.*.aligned` is undefined for a diverged warp; callers reach it after loops with per-lane exits."""
    bodies = [b for b in re.findall(r"__device__ __forceinline__ [^{;]*\{(.*?)\n\}", _read("common", "ptx.cuh"), re.S) if "barrier.cluster" in b]
    assert bodies
    for body in bodies:
        assert body.index("__syncwarp()") < body.index("barrier.cluster"), body
    for name in os.listdir(CSRC):
        if name.endswith(".cu"):
            assert "barrier.cluster" not in _read(name), name + ": use the wrapper"


def test_waits_before_warp_wide_instructions_give_the_warp_one_answer():
    """TMEM loads, shuffles and __syncwarp follow the waits of whole warps: lanes that give up (time limit, abort flag) must
    do so together.  The per-lane wait is left to branches of a single thread."""
    for name in ("gemm_sm100.cu", "attention.cu"):
        lone = [line.strip() for line in _read(name).splitlines() if re.search(r"\bwait_parity\(", line)]
        assert all(re.match(r"(bool )?w = ", line) for line in lone), (name, lone)      # issuing thread of the serial attention forward


def test_tensor_memory_is_allocated_before_a_successor_is_admitted():
    """A kernel that is set up while its predecessor runs allocates TMEM before it waits for it.  If the predecessor still had to allocate
    on the same SM, each could hold what the other waits for, without a time limit."""
    admits = r"\b(after_predecessor|admit_successor|gemm_begin)\("
    seen = 0
    for name in ("gemm_sm100.cu", "gemm_transposed.cuh", "gemm_wgrad.cuh", "attention.cu"):
        text = _read(name)
        # bodies of kernels and of what they share: from a template or __global__ / __device__ line to the brace in the first column
        for body in re.findall(r"^__(?:global|device)__[^;{]*\{\n(.*?)^\}", text, re.S | re.M):
            alloc = re.search(r"\btmem_alloc(_pair)?\(", body)
            if alloc is None:
                continue
            seen += 1
            first = re.search(admits, body)
            assert first is not None and first.start() > alloc.start(), (name, body[:120])
    assert seen == sum(len(re.findall(r"\btmem_alloc(?:_pair)?\(", _read(n))) for n in ("gemm_sm100.cu", "gemm_transposed.cuh", "gemm_wgrad.cuh", "attention.cu")) == 8


def test_every_launch_follows_one_rule_for_early_set_up():
    """Programmatic launch pays for grids of up to a number of CTAs: no launcher sets it by itself."""
    for name in sorted(os.listdir(CSRC)) + [os.path.join("common", "host.h")]:
        if name.endswith((".cu", ".cuh", ".h", ".cpp")):
            for value in re.findall(r"programmaticStreamSerializationAllowed = ([^;]*);", _read(name)):
                assert value.startswith("early_setup_pays("), (name, value)
