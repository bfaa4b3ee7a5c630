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


def _bodies(heads=False):
    """Kernel name -> body (or list of parameters), of every __global__ definition."""
    out = {}
    for text in FILES.values():
        for m in re.finditer(r"__global__", text):
            head = re.compile(r"\b(\w+_kernel)\s*\(").search(text, m.end())
            if head is None:
                continue
            close = _closing(text, head.end() - 1, "()")
            brace = text.find("{", close)
            if text[close + 1:brace].strip() == "":
                out[head.group(1)] = text[head.end():close] if heads else text[brace:_closing(text, brace, "{}") + 1]
    return out


def _ahead():
    names = set()
    for text in FILES.values():
        names |= set(re.findall(r"sllm_launch\(\s*(?:\w+::)*(\w+_kernel)\b", text))
        names |= set(re.findall(r"cudaLaunchKernelEx\(&cfg, (\w+_kernel)\b", text))
    return names | {"chunk_delta_parts_kernel", "chunk_delta_out_kernel"}             # launched through a pointer


def _read_in_front_of_the_wait(head, body):
    """Parameters (pointers, tensor maps, a struct's pointers) that the text in front of the first wait reads through."""
    before = re.sub(r"//[^\n]*", "", body).split("pdl_wait()")[0]
    params = [(a.split()[-1].lstrip("*&"), "*" in a) for a in head.replace("\n", " ").split(",")]
    pointers, others = {n for n, p in params if p}, {n for n, p in params if not p}
    read = pointers & set(re.findall(r"(?<![\w.>])(\w+)\[", before) + re.findall(r"\(\s*\(?[^()]*\*\)\s*\(?(\w+)", before)
                          + re.findall(r"\bld\w*\(\s*(\w+)", before) + re.findall(r"(?<![\w)\]] )\*(\w+)", before))
    read |= {f"{s}.{f}" for s, f in re.findall(r"\b(\w+)\.(\w+)\[", before) if s in others}
    return read | set(re.findall(r"tma_load\w*\([^;]*?&(\w+)", before)) | ({"?"} if re.search(r"\b(ld_dep|ld_stream|load_w|__ldg)\w*\s*\(", before) else set())


# what is read in front of the wait on purpose: weights, which no kernel of a step writes (the few-rows product's lambdas that read
# its input stand in front of the wait and run behind it)
WEIGHTS = {"gemm_small_m_kernel": {"?", "y"}, "gemm_tc_cluster_kernel": {"map_b"}, "gemm_tc_skinny_kernel": {"map_w"}, "add_rms_normed_reg_kernel": {"?"}}


def test_every_kernel_launched_ahead_waits_for_the_one_in_front():
    bodies, heads, ahead = _bodies(), _bodies(heads=True), _ahead()
    assert len(ahead) > 40 and ahead <= set(bodies)
    assert not [k for k in sorted(ahead) if "pdl_wait()" not in bodies[k]]
    early = {k: _read_in_front_of_the_wait(heads[k], bodies[k]) - WEIGHTS.get(k, set()) for k in sorted(ahead)}
    assert not {k: v for k, v in early.items() if v}


def test_only_the_few_rows_product_reads_its_second_operand_ahead():
    """The plain product's may be what the kernel in front writes: where a cluster shares its K it waits first, too."""
    text = FILES["gemm_tcgen05.cu"]
    body = _bodies()["gemm_tc_cluster_kernel"]
    assert 0 < body.find("if (!b_ahead) pdl_wait();") < body.find("tma_load_2d(")
    calls = re.findall(r"(sllm_gemm_tc_\w+)\(|return tc_cluster_launch\(A, B, [^;]*tile_n, ([01]), err", text)
    ahead, fn = {}, None
    for name, flag in calls:
        fn = name or fn
        if flag:
            ahead[fn] = int(flag)
    assert ahead == {"sllm_gemm_tc_fold_bf16": 0, "sllm_gemm_tc_act_bf16": 0, "sllm_gemm_tc_skinny_bf16": 1}


def test_a_read_in_front_of_the_wait_is_found():
    for read in ("float v = x[threadIdx.x];", "float4 v = *(const float4*)(x + 4);", "float v = ld4(x + 3);", "int v = p.rows[0];",
                 "tma_load_2d(dst, &map, 0, 0, bar);", "int n = *count;"):
        head = "const float* __restrict__ x, const int* count, Args p, const __grid_constant__ CUtensorMap map"
        assert _read_in_front_of_the_wait(head, "{ " + read + " pdl_wait(); }") and not _read_in_front_of_the_wait(head, "{ pdl_wait(); " + read + " }")


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
