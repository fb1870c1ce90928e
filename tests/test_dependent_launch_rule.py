"""Under programmatic dependent launch a kernel may begin before the kernel in front of it has ended (csrc/common.cuh)."""

import os
import re

import pytest

import ullm_b200.csrc.build as build

def files():
    return sorted(f for f in os.listdir(build.HERE) if f.endswith((".cu", ".cuh")))


def text(name):
    with open(os.path.join(build.HERE, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", files())
def test_every_kernel_that_is_launched_so_waits(name):
    """Each kernel of a file that launches through `ullm_launch_kernel` waits for the kernel in front of it."""
    s = text(name)
    for kernel in set(re.findall(r"ullm_launch_kernel\((\w+)", s)):
        at = re.search(r"__global__[^;{]*?\b%s\(" % kernel, s)
        if at is not None:
            body = s[at.end():]
            body = body[:body.find("__global__")] if "__global__" in body else body
            assert "pdl_wait();" in body, kernel
