"""What the launchers keep between calls, read from their sources: a kernel's limit of dynamic shared memory belongs to a device, so no
launcher may remember for the whole process that it was raised (a model on the process's second device would fail at its first launch).  And
what a kernel that lives beside the one in front of it may not do."""
import pathlib
import re

import arle_b200

CSRC = pathlib.Path(arle_b200.__file__).parent / "csrc"


def test_no_launcher_remembers_a_device_setting_per_process():
    sources = sorted(CSRC.glob("*.cu"))
    assert sources
    for f in sources:
        text = f.read_text()
        assert not re.search(r"static\s+bool\s+\w+\s*(\[\w*\])?\s*[={;]", text), f.name
        for flag in re.findall(r"static\s+(?:std::)?(?:atomic<bool>|once_flag)\s+\w+", text):
            raise AssertionError(f"{f.name}: {flag}")


def test_the_limit_is_kept_per_device():
    text = (CSRC / "common.cuh").read_text()
    body = text[text.index("class SharedLimit"):]
    assert "cudaGetDevice(&dev)" in body[: body.index("};")]


def test_kernels_that_always_start_early_read_plainly():
    """The non-coherent load path is for memory that nobody writes while the kernel lives, and a kernel launched programmatically lives beside
    the one in front of it, which may write its weights: waiting for that kernel orders plain loads alone."""
    text = (CSRC / "gemm_skinny.cu").read_text()
    first, last = text.index("uint4 ld_weights("), text.index("struct DirectPlan")
    body = re.sub(r"//[^\n]*", "", text[first:last])
    assert "direct_gemm_kernel(" in body and "pdl_wait();" in body
    assert not re.search(r"\.nc\b|__ldg\(", body)


def test_the_streamed_decode_attention_starts_early_and_reads_plainly():
    text = (CSRC / "attention_decode_stream.cu").read_text()
    assert "launch_kernel_as(prep.on != 0" in text
    kernel = text[text.index("decode_stream_kernel("): text.index("size_t fixed_smem(")]
    for part in (kernel, text[text.index("void prep_head("): text.index("constexpr int kPlanHeader")], text[text.index("void stream_shares("): text.index("void own_units(")]):
        body = re.sub(r"//[^\n]*", "", part)
        assert not re.search(r"\.nc\b|__ldg\(|__restrict__", body)
    body = re.sub(r"//[^\n]*", "", kernel)
    assert body.index("pdl_wait();") < min(body.index(x) for x in ("q_indptr[", "plan[", "rows_plan[i]", "stream_shares(q_indptr", "block_table +") if x in body)


def _functions(text):
    """Name -> arguments and body of the functions that are defined in ``text`` (of all, where several have a name)."""
    found = {}
    for m in re.finditer(r"\b(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += (text[i] == "(") - (text[i] == ")")
            i += 1
        rest = re.match(r"\s*\{", text[i:])
        if rest is None or m.group(1) in ("if", "for", "while", "switch"):
            continue
        depth, j = 1, i + rest.end()
        while depth and j < len(text):
            depth += (text[j] == "{") - (text[j] == "}")
            j += 1
        found[m.group(1)] = found.get(m.group(1), "") + text[m.end(): j]
    return found


def test_kernels_that_are_launched_early_read_plainly():
    """Every kernel that goes through launch_early, or through launch_kernel_as with a condition of its own: no restrict on what it reads, no
    __ldg in it nor in a function that it calls, and a wait before anything else."""
    headers = {f: re.sub(r"//[^\n]*", "", f.read_text()) for f in CSRC.glob("*.cuh")}
    shared = _functions("\n".join(headers.values()))
    found = set()
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        here = _functions(text)
        kernels = set(re.findall(r"__global__[^;{]*?\b(\w+)\s*\((?!\s*(?:THREADS|\d))", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text)))
        for m in re.finditer(r"launch_(?:early\(|kernel_as\()([^;]*);", text):
            names = kernels & set(re.findall(r"\b\w+\b", m.group(1)))
            for var in set(re.findall(r"\bauto (\w+) =", text[: m.start()])) & set(re.findall(r"\b\w+\b", m.group(1))):
                names |= kernels & set(re.findall(r"\b\w+\b", text[text.rindex(f"auto {var} =", 0, m.start()): m.start()]))
            assert names, f"{f.name}: {m.group(0)[:80]}"
            for name in names - {"skinny_gemm_kernel"}:                 # early where a switch asks for it alone
                body = here[name]
                called = {name} | (set(re.findall(r"\b(\w+)\s*(?:<[^<>;]*>)?\s*\(", body)) & (set(here) | set(shared)))
                for c in called - {"launch_early"}:
                    assert not re.search(r"\.nc\b|__ldg\(", here.get(c) or shared[c]), (name, c)
                if name == "direct_gemm_kernel":                         # its weights and rows go through loads of their own
                    continue
                assert "__restrict__" not in body and "pdl_wait();" in body, name
                found.add(name)
    assert {"moe_plan_kernel", "moe_rows_kernel", "moe_combine_kernel", "moe_select_warp_kernel", "latent_prep_kernel", "latent_gather_kernel",
            "latent_plan_kernel", "rms_rows_block_kernel", "rmsnorm_vec_kernel", "silu_mul_bf16_vec_kernel", "decode_stream_kernel",
            "delta_gates_kernel", "ssm_gates_kernel", "rotary_angles_kernel"} <= found
