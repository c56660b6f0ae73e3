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


def test_kernels_that_are_launched_early_read_plainly():
    """Every kernel that goes through launch_early, or through launch_kernel_as with a condition of its own: no restrict on what it reads, no
    __ldg, and a wait before anything else."""
    found = set()
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        names = set()
        for m in re.finditer(r"launch_(?:early\(|kernel_as\()([^;]*);", text):
            names |= set(re.findall(r"\b\w+_kernel\b", m.group(1)))
            if re.match(r"\s*kernel\b", m.group(1)):
                names |= set(re.findall(r"\b\w+_kernel\b", text[text.rindex("auto kernel", 0, m.start()): m.start()]))
        for name in names:
            at = re.search(r"__global__[^;{]*?\b" + name + r"\s*\(", text)
            if at is None:
                continue
            end = text.index("\n}\n", at.end())
            body = text[at.end(): end]
            assert not re.search(r"\.nc\b|__ldg\(", body), name
            if name in ("skinny_gemm_kernel", "direct_gemm_kernel"):      # their weights and rows go through loads of their own
                continue
            assert "__restrict__" not in body and "pdl_wait();" in body, name
            found.add(name)
    assert {"moe_plan_kernel", "moe_rows_kernel", "moe_combine_kernel", "moe_select_warp_kernel", "latent_prep_kernel", "latent_gather_kernel",
            "latent_plan_kernel", "rms_rows_block_kernel", "rmsnorm_vec_kernel", "silu_mul_bf16_vec_kernel", "decode_stream_kernel",
            "delta_gates_kernel", "ssm_gates_kernel", "rotary_angles_kernel"} <= found
