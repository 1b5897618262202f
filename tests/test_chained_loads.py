"""Kernels that are launched while the one before them still runs must not read
its vectors through the read-only path: ld.global.nc and __ldg (and what the
compiler makes of const __restrict__ pointers) want data that nothing writes
while the kernel lives.  Tables are uploaded before any of the kernels start and
may be read that way.  Checked on the sources: in the files whose kernels are
launched that way, vectors are the pointers to the element type T (in the adjoint
kernels, which are FP64 only, the parameters named in VECTORS)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ed_solver_b200", "csrc")
FILES = ["edk_kernels.cu", "edk_rows_fast.cuh", "edk_rows_tma.cuh", "edk_sz.cu", "edk_grad_kernels.cu", "edk_device.cuh"]
VECTORS = ["a", "b", "w", "r", "vkm1", "vk", "vbn", "vbc", "wbar", "vkp", "vkk", "vkm", "hw", "ap", "p", "psi"]
# kernels of these files that are launched plainly, after the grid before them has ended
PLAIN = {"edk_kernels.cu": ["combine_kernel"], "edk_sz.cu": ["sz_apply_c_kernel"]}


def _source(name):
    s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    for k in PLAIN.get(name, []):
        s = re.sub(r"__global__[^;{]*\b%s\(.*?\n}\n" % k, "", s, flags=re.S)
    return s


@pytest.mark.parametrize("name", FILES)
def test_vectors_keep_off_the_read_only_path(name):
    s = _source(name)
    assert "launch_chained" in s or name.endswith(".cuh")
    assert ".nc" not in "".join(re.findall(r'asm volatile\(\s*"ld[^"]*"', s))
    assert not re.search(r"\bldr[124]\(", s)              # the plainly launched kernels' loads
    for m in re.finditer(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?(\w+)", s):
        kinds = re.findall(r"(\w+) \*(?:__restrict__ )?%s\b" % m.group(1), s[:m.start()])
        assert not kinds or kinds[-1] not in ("T", "int4"), m.group(0)
    assert not re.search(r"\bT \*__restrict__", s)
    if name == "edk_grad_kernels.cu":
        assert not [v for v in VECTORS if re.search(r"double \*__restrict__ %s\b" % v, s)]
