"""Rules that the kernel sources have to keep and that no run shows reliably (CPU only)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "expertscattergather_b200", "csrc")


def _kernels():
    """(file, name, parameters, body) of every kernel."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s", text):
            k = re.compile(r"(\w+_kernel\w*)\s*\(").search(text, m.end())
            i = k.end()
            j = text.index("{", i)
            depth, end = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield os.path.basename(path), k.group(1), text[i:j], text[j:end]


KERNELS = list(_kernels())


def test_kernels_are_found():
    names = {k[1] for k in KERNELS}
    assert {"strict_kernel", "dense16_kernel", "generic_rowgemm_kernel", "scatter_prepare_kernel", "csr_batch_place_kernel"} <= names


DEPENDENTS = [k for k in KERNELS if "pdl_wait" in k[3]]


@pytest.mark.parametrize("kernel", DEPENDENTS, ids=[k[1] for k in DEPENDENTS])
def test_dependent_kernels_promise_nothing_about_aliases(kernel):
    """A kernel that may start under the one before it must not tell the compiler that nobody writes its inputs meanwhile: loads
    through `__restrict__` pointers are not bound by the wait."""
    file, name, params, body = kernel
    assert "__restrict__" not in params + body, f"{file}: {name}"


def test_ctas_that_count_for_themselves_are_resident_together():
    """The grid of the kernel that counts ids and fills has four CTAs for an SM; one that has to wait for the others counts and fills after them."""
    text = open(os.path.join(CSRC, "egs_generic.cu")).read()
    assert re.search(r"__launch_bounds__\(kPrepThreads, 4\)\s+scatter_prepare_kernel", text)
    assert "size_t grid = 4 * 148;" in text
