"""Kernels launched dependent (csrc/pdl.cuh) exist while their predecessor still
writes, so what it writes may not be read through the read-only path: no __ldg
and no const __restrict__ parameter, but for data that no running predecessor
writes."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lbman3d_b200", "csrc")
# weights, biases and scales; pre-activations the forward pass stored
SETTLED = {"bimg", "bias", "pre_below", "shift", "inv_scale", "out_scale"}


def _block(text, at, pair):
    depth, i = 0, text.index(pair[0], at)
    for j in range(i, len(text)):
        depth += (text[j] == pair[0]) - (text[j] == pair[1])
        if depth == 0:
            return text[i + 1:j], j + 1
    raise AssertionError("unbalanced source")


def _dependent_kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cuh", ".cu")):
            continue
        with open(os.path.join(CSRC, name)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__\s+void\s+", text):
            at = m.end()
            bounds = re.match(r"__launch_bounds__", text[at:])
            if bounds:
                _, at = _block(text, at, "()")
            kernel = re.match(r"\s*(\w+)", text[at:]).group(1)
            params, at = _block(text, at, "()")
            body, _ = _block(text, at, "{}")
            if "pdl_begin()" in body:
                yield name, kernel, params


KERNELS = list(_dependent_kernels())


def test_the_dependent_kernels_are_found():
    assert {k for _, k, _ in KERNELS} >= {"qpoint_kernel", "qpoint2_kernel", "point_force_kernel", "lbm_aa_point_kernel",
                                          "lbm_aa_point_h2_kernel", "conv_dhalo_kernel", "wgrad_march_kernel",
                                          "sum_partials_kernel", "features_kernel", "loss_kernel", "apply_kernel"}


@pytest.mark.parametrize("file,kernel,params", KERNELS, ids=[k for _, k, _ in KERNELS])
def test_inputs_are_not_declared_read_only(file, kernel, params):
    read_only = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
    assert read_only <= SETTLED, (file, kernel, read_only - SETTLED)


@pytest.mark.parametrize("file", sorted({f for f, _, _ in KERNELS}))
def test_no_read_only_loads_beside_them(file):
    with open(os.path.join(CSRC, file)) as fh:
        assert "__ldg" not in fh.read()


def test_the_point_update_takes_plain_pointers():
    # the device functions of the point kernels hand the pointers on
    with open(os.path.join(CSRC, "qpoint.cuh")) as fh:
        assert not re.findall(r"const\s+\w+\s*\*\s*__restrict__", fh.read())
