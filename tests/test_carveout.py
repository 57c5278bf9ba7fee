"""Every kernel that runs beside another lane's asks for the largest shared-memory
carveout (the reason stands at stage1_configure): each one's name is in its file's
list, or in the function that the list is made from."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "projekt-2012_b200", "csrc")


@pytest.mark.parametrize("file,func", [("stage1.cu", "stage1_configure"), ("batch.cu", "batch_configure"),
                                       ("traceback.cu", "walker_configure")])
def test_every_kernel_is_configured(file, func):
    text = open(os.path.join(CSRC, file)).read()
    kernels = set(re.findall(r"__global__ void(?:\s+__launch_bounds__\((?:[^()]|\([^()]*(?:\([^()]*\)[^()]*)*\))*\))?\s+(\w+)\(", text))
    assert len(kernels) == len(re.findall(r"__global__ void", text))
    body = text[text.index(f"cudaError_t {func}()"):]
    body = body[:body.index("\n}\n")]
    if "kernel_of(" in body:  # the kernels that launches choose from
        body += "".join(re.findall(r"^KernelRef \w+\(.*?^}$|^template[^\n]*\nKernelRef \w+\(.*?^}$", text, re.M | re.S))
    missing = {k for k in kernels if not re.search(rf"\b{k}\b", body)}
    assert not missing
