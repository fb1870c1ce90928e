"""Under programmatic dependent launch a kernel may begin before the kernel in front of it has ended.  What that kernel writes must then
not be declared unchanging (csrc/common.cuh): `__restrict__` and `__ldg` are for weights and tables, and `__restrict__` for results that
a kernel writes and does not read."""

import os
import re

import pytest

import ullm_b200.csrc.build as build

# weights, and tables made of constants, by the name they have in every kernel
FIXED = set("""w w0 w2 wa wb wo wq wk q_w k_w w_c conv_w conv_b weights table mu mix inv_freq cos_t sin_t bias bias_i bias_f b1 b2 bz bx
alpha alpha2 pq dt_bias a_log d_skip bonus correction extra_vec vmix_lambda q_head_scale""".split())
FIXED_IN = {("moe_combine_add_norm_kernel", "scale"), ("norm_rows_kernel", "b")}
# results
WRITTEN = set("""out out_f32 part_o part_ml parts q_out k_cache v_cache k_pages v_pages pk_pages pv_pages terms y copy rows_out xbc dt
log_decay scores choice weight total""".split())
WRITTEN_IN = {("gla_fold_kernel", "fold"), ("mingru_fold_kernel", "fold_a"), ("mingru_fold_kernel", "fold_b")}
# launched by itself, while products are timed
NOT_LAUNCHED_SO = {"lt_flush_read_kernel"}

LDG = {"brow", "bp", "p.norm_w", "p.bias", "p.pre_w", "reinterpret_cast<const float4*>(src"}  # (src: rows of w)


def files():
    return sorted(f for f in os.listdir(build.HERE) if f.endswith((".cu", ".cuh")))


def text(name):
    with open(os.path.join(build.HERE, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def restricted(s):
    """(function, const or not, parameter) of every `__restrict__` in a parameter list; how many stand elsewhere."""
    found = []
    lists = re.compile(r"(\w+)\(([^()]*__restrict__[^()]*(?:\([^()]*\)[^()]*)*)\)")
    for m in lists.finditer(s):
        for const, name in re.findall(r"(const )?\b[\w:]+\s*\*+\s*__restrict__ (\w+)", m.group(2)):
            found.append((m.group(1), bool(const), name))
    return found, s.count("__restrict__") - len(found)


@pytest.mark.parametrize("name", files())
def test_only_what_no_step_writes_is_declared_unchanging(name):
    s = text(name)
    found, elsewhere = restricted(s)
    assert elsewhere == 0
    for function, const, parameter in found:
        if function not in NOT_LAUNCHED_SO:
            allowed, here = (FIXED, FIXED_IN) if const else (WRITTEN, WRITTEN_IN)
            assert parameter in allowed or (function, parameter) in here, (function, parameter)
    for read in re.findall(r"__ldg\(([^;]*)", s):
        assert any(read.startswith(k) for k in LDG), read


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
