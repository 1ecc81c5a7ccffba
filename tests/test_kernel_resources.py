"""What no result shows.  Registers and spills of the kernels that read partial sums, as the compiler reports them (build/*.ptxas): a kernel that holds
the values of many slabs where a prompt has one finished matrix loses warps in flight, or spills.  And the pointers of kernels that may start
before the one in front of them has finished."""
import glob
import os
import re

import pytest

from nn_b200 import build

if not os.path.exists(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")):
    pytest.skip("no nvcc", allow_module_level=True)


@pytest.fixture(scope="module")
def report():
    """{mangled name: (registers, bytes spilled)}"""
    build.make()
    found = {}
    for file in os.listdir(os.path.join(build.CSRC, "build")):
        if file.endswith(".ptxas"):
            text = open(os.path.join(build.CSRC, "build", file)).read()
            for name, spill, regs in re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill loads.*?Used (\d+) registers", text, re.S):
                found[name] = (int(regs), int(spill))
    return found


# of every size the kernel is built for: registers that the smallest build may have (65536 a SM), bytes that any build may spill
@pytest.mark.parametrize("kernel,most_registers,most_spilled", [
    ("ns_lightning_chunk_kernel", 255, 32),
    ("ns_glu_rows_kernel", 48, 0), ("ns_copy_cols_kernel", 32, 0), ("ns_rms_rows_kernel", 40, 0), ("ns_rms_post_rows_kernel", 40, 0),
    ("ns_window_append_kernel", 48, 40), ("ns_short_conv_kernel", 72, 20), ("ns_short_conv_slide_kernel", 168, 32),
    ("ns_rotate_heads_kernel", 32, 0), ("ns_latent_append_kernel", 40, 0), ("ns_gated_norm_kernel", 48, 0), ("ns_delta_chunk_kernel", 254, 0),
    ("ns_delta_recurrent_kernelILi16E", 128, 0), ("ns_lightning_recurrent_kernelILi8E", 64, 24),
    # 16 warps of two units in flight; the launch's registers that setmaxnreg deals out (tiles of one group spill a few words); five CTAs an SM
    ("ns_stream_bf16_kernel", 128, 0), ("ns_attention_prompt_kernelILb0E", 168, 0), ("ns_attention_prompt_kernelILb1E", 168, 96), ("ns_attention_decode_kernelILi\\d+ELi2ELi5E", 96, 0),
])
def test_kernels_of_many_rows_stay_small(report, kernel, most_registers, most_spilled):
    builds = {n: v for n, v in report.items() if re.search(r"\d" + kernel, n)}
    assert builds
    # builds of one size differ in the last template argument, the number of slabs read together (and the CTAs an SM is to hold)
    ways = 2 if "recurrent" in kernel else 1
    sizes = {}
    for name, (regs, spill) in builds.items():
        assert spill <= most_spilled, (name, spill)
        key = re.sub(r"(Li\d+E){%d}E" % ways, "E", name)
        sizes[key] = min(regs, sizes.get(key, 1 << 30))
    assert max(sizes.values()) <= most_registers, sizes


def _programmatic():
    """Kernels that are launched programmatically: named in the call, or what `kernel` stands for in the function around it."""
    names = set()
    for path in sorted(glob.glob(os.path.join(build.CSRC, "*.cu"))):
        text = open(path).read()
        names |= set(re.findall(r"ns_launch_pdl\(\s*(ns_\w+?)(?:<[^(]*>)?,", text))
        for call in re.finditer(r"ns_launch_pdl\(\s*kernel,", text):
            start = max(m.start() for m in re.finditer(r"^(?:extern \"C\" |template |static )?[\w*<> ,]+\(?.*$", text[:call.start()], re.M) if m.group()[0] not in " }")
            body = text[start:text.index("\n}", call.start())]
            found = re.findall(r"auto kernel = (ns_\w+)", body) + re.findall(r"launch\((ns_\w+)<", body)
            assert found, (path, body)
            names |= set(found)
    return names


def test_programmatic_launches_read_nothing_early():
    """The compiler may move a load through a const __restrict__ pointer, or an __ldg, above griddepcontrol.wait, unless the pointer comes out of ns_after_wait.
    Weights are exempt: they are read by volatile instructions, before the wait only where no kernel writes them (prefetch_b)."""
    source = "\n".join(open(f).read() for f in sorted(glob.glob(os.path.join(build.CSRC, "*.cu"))))
    names = _programmatic()
    assert {"ns_f32_linear_kernel", "ns_f32_attention_step_kernel", "ns_stream_bf16_kernel", "ns_rms_rows_kernel", "ns_rms_post_rows_kernel", "ns_rms_post_rows_vec_kernel",
            "ns_gemv_i8_kernel", "ns_stream_i8_kernel", "ns_gemm_tc_kernel", "ns_gemm_tail_kernel"} <= names
    for name in names:
        parameters, body = re.search(name + r"\(([^)]*)\)\s*\{(.*?)\n\}", source, re.S).groups()
        for pointer in re.findall(r"const\s+\w+\*\s*__restrict__\s+(\w+)", parameters):
            waits = re.search(r"\b%s = ns_after_wait\(%s\)" % (pointer, pointer), body)
            streamed = pointer == "w" and "load_stream(" in body and not re.search(r"__ldg\([^;]*\bw\b|[^\w.]w\[", body)
            assert waits or streamed, (name, pointer)
        # through the fields of a struct: kernels that do something before their wait, other than these int8 ones, whose scales and biases stand in conditional
        # code of their loops
        early = body[:body.index("ns_pdl_wait()")] if "ns_pdl_wait()" in body else ""
        if name not in ("ns_gemv_i8_kernel", "ns_stream_i8_kernel") and re.search(r"prefetch|load|fill", early):
            assert not re.search(r"__ldg\((?:reinterpret_cast<[^>]*>\()?&?[ap]\.", body), name


def test_a_row_ahead_fits_the_longest_rows(report):
    """16384 columns take 1024 threads: 64 registers each."""
    (regs, spill), = [v for n, v in report.items() if "ns_quantize_rows_reg_kernelILi2ELb1ELb1E" in n]
    assert regs <= 64 and spill == 0
