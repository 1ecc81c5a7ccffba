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


def test_programmatic_launches_read_nothing_early():
    """The compiler may move a load through a const __restrict__ pointer above griddepcontrol.wait, unless the pointer comes out of ns_after_wait."""
    source = "\n".join(open(f).read() for f in sorted(glob.glob(os.path.join(build.CSRC, "*.cu"))))
    names = set(re.findall(r"ns_launch_pdl\(\s*(ns_\w+?)(?:<[^(]*>)?,", source))
    assert "ns_f32_linear_kernel" in names and "ns_f32_attention_step_kernel" in names
    for name in names:
        parameters, body = re.search(name + r"\(([^)]*)\)\s*\{(.*?)\n\}", source, re.S).groups()
        for pointer in re.findall(r"const\s+\w+\*\s*__restrict__\s+(\w+)", parameters):
            assert re.search(r"\b%s = ns_after_wait\(%s\)" % (pointer, pointer), body), (name, pointer)
