"""The shared-memory limit of a kernel is an attribute of the device: where a
launch needs more than the default, the host raises it on every call and not
once per process, and with one value for all sizes."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# kernels of the FP64 form that run with more than 48 KB
KERNELS = ["stencilInt", "exactGramKernel", "exactVCKernel", "cholInvKernel",
           "cholDropSmemKernel", "refJacobiKernel", "hhTridiagDfKernel"]


def _sources():
    files = glob.glob(os.path.join(ROOT, "nuclearcgm_gb300", "csrc", "*.cu"))
    return "\n".join(open(f).read() for f in files)


def test_limits_are_raised_on_every_call():
    once = "\n".join(re.findall(r"static const bool \w+ = \[\]\s*\{.*?\}\(\);",
                                _sources(), re.S))
    assert [k for k in KERNELS if re.search(r"\b%s\b" % k, once)] == []


def test_inverse_factor_has_one_limit():
    set_to = re.findall(r"cudaFuncSetAttribute\(cholInvKernel<true>,\s*"
                        r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*"
                        r"\(int\)(\w+)\)", _sources())
    assert set_to == ["kMaxSmem"]
