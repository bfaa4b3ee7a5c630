"""Kernels that may start before the kernel in front of them has finished wait for it: in the sources, without a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "scriptling_llm_lib_b200" / "csrc"
FILES = {p.name: p.read_text() for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh", ".inc")}


def _closing(s, i, pair):
    """Where the bracket that opens at s[i] closes."""
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j
    raise ValueError("unbalanced")


def _bodies():
    """Kernel name -> body, of every __global__ definition."""
    out = {}
    for text in FILES.values():
        for m in re.finditer(r"__global__", text):
            head = re.compile(r"\b(\w+_kernel)\s*\(").search(text, m.end())
            if head is None:
                continue
            close = _closing(text, head.end() - 1, "()")
            brace = text.find("{", close)
            if text[close + 1:brace].strip() == "":
                out[head.group(1)] = text[brace:_closing(text, brace, "{}") + 1]
    return out


def test_every_kernel_launched_ahead_waits_for_the_one_in_front():
    bodies, ahead = _bodies(), set()
    for text in FILES.values():
        ahead |= set(re.findall(r"sllm_launch\(\s*(?:\w+::)*(\w+_kernel)\b", text))
        ahead |= set(re.findall(r"cudaLaunchKernelEx\(&cfg, (\w+_kernel)\b", text))
    ahead |= {"chunk_delta_parts_kernel", "chunk_delta_out_kernel"}             # launched through a pointer
    assert len(ahead) > 40 and ahead <= set(bodies)
    assert not [k for k in sorted(ahead) if "pdl_wait()" not in bodies[k]]


def test_tensor_memory_is_taken_before_dependents_may_start():
    """A dependent's block that took an SM's columns first would wait for a kernel that waits for them."""
    for name, body in _bodies().items():
        taken = max(body.find("tcgen05.alloc"), body.find("u.open("))
        if taken >= 0 and "pdl_launch_dependents()" in body:
            assert body.find("pdl_launch_dependents()") > taken, name


def test_what_a_launcher_sets_up_is_kept_for_each_device():
    """A kernel's limit of shared memory and the blocks that fit are a device's own: a process may run engines on several."""
    for name, text in FILES.items():
        assert not re.findall(r"static (?:bool|int) \w+(?:\[\d+\])? = (?:false|0|\{)[^;]*;", text), name
