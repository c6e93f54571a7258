"""Host-side rules of the kernel launchers, read from the sources."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shared_memory_limits_are_set_per_device():
    """A kernel's dynamic shared-memory limit belongs to a device: a launcher that remembers having set it once per process fails on a second GPU. So the limit
    is set by allow_smem (a bit per device), behind an array with an entry per device, or at every launch."""
    sets = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "vyomai_b200", "csrc", "*.cu*"))):
        src = open(path).read()
        for m in re.finditer(r"cudaFuncSetAttribute\(", src):
            before = src[max(0, m.start() - 250):m.start()]
            kept = re.search(r"\bstatic\s+(bool|size_t|std::once_flag)\s+\w+(\[\w+\])?\s*[={;]", before)
            assert kept is None or "[dev]" in before, (path, src[m.start():m.start() + 100])
            sets += 1
    assert sets > 0


def test_register_shares_that_a_build_does_not_have_choose_another_form():
    """Kernels whose warps share registers out (setmaxnreg) run only where the compiler gave the count that the shares add up to. Whether it did belongs to the rule that
    chooses the form - another toolkit's build then takes the forms beside them - and is no error of the call. The build that is here has it."""
    kernels = {"window_attn_tc": ("window_attn_tc_applies", "TC_REGS", 4, "window_attn_tc_kernel"), "linear_attn_tc": ("linear_attn_tc_applies", "LT_REGS", 1, "la_outputs_tc_kernel")}
    csrc = os.path.join(ROOT, "vyomai_b200", "csrc")
    for path in glob.glob(os.path.join(csrc, "*.cu")):
        if "setmaxnreg" in open(path).read():
            assert os.path.basename(path)[:-3] in kernels
    for name, (rule, regs, forms, kernel) in kernels.items():
        src = open(os.path.join(csrc, name + ".cu")).read()
        assert "cudaErrorInvalidConfiguration" not in src
        count = int(re.search(rf"\b{regs} = (\d+)", src).group(1))
        body = src[src.index(f"bool {rule}("):]
        body = body[:body.index("\n}")]
        assert "registers" in body and re.search(r"\) return false;|!enough\) return false;", body)
        log = os.path.join(csrc, "build", name + ".ptxas.log")
        if os.path.exists(log):
            used = re.findall(rf"entry function '[^']*{kernel}[^']*'(?:(?!entry function).)*?Used (\d+) registers", open(log).read(), re.S)
            assert len(used) == forms and all((int(u) + 7) // 8 * 8 == count for u in used)


def test_register_shares_of_builds_made_by_including_a_file():
    """linear_attn_tc_fixed.cu builds linear_attn_tc.cu's kernels once more, with registers of its own: its rule asks for the same count, and the build that is here has it."""
    csrc = os.path.join(ROOT, "vyomai_b200", "csrc")
    for path in glob.glob(os.path.join(csrc, "*.cu")):   # every file that builds such kernels by including them
        src = open(path).read()
        if re.search(r'#include "\w+\.cu"', src):
            assert os.path.basename(path) == "linear_attn_tc_fixed.cu" and '#include "linear_attn_tc.cu"' in src
    src = open(os.path.join(csrc, "linear_attn_tc.cu")).read()
    count = int(re.search(r"\bLT_REGS = (\d+)", src).group(1))
    assert "la_fixed_registers()" in src[src.index("bool linear_attn_tc_applies("):] and re.search(r"bool la_fixed_registers\(\) \{ return la_registers<false, VY_UACT_SILU>\(\); \}", src)
    log = os.path.join(csrc, "build", "linear_attn_tc_fixed.ptxas.log")
    if os.path.exists(log):
        used = re.findall(r"entry function '[^']*la_outputs_tc_kernel[^']*'(?:(?!entry function).)*?Used (\d+) registers", open(log).read(), re.S)
        assert len(used) == 1 and (int(used[0]) + 7) // 8 * 8 == count
