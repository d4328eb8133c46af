"""Kernels that may start while the one before them drains (let_next_start) read nothing that a kernel
writes before they wait for it: the flags that leave out instances, the reference pressures and the
solver's counters. Read from the sources: a stale flag shows on a GPU only once in a great while."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "teal_b200", "csrc")
WRITTEN = re.compile(r"leaves_out\(|left_out\(|active\[|pr_ref\)?\.of|\.newton\(|\.arnoldi\(|\bgb\.(ctl|sc|part)\b|\bst\.\w+\[")
LEAVE = re.compile(r"if \((.*)\) \{\s*wait_for_previous\(\);\s*return;\s*\}")


def kernels():
    for name in ("aux_kernels.cuh", "kernels.cuh", "face.cuh", "gmres.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//.*", "", f.read())
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\([^{;]*\)\s*\{", text):
            end, depth = m.end(), 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            if "let_next_start();" in text[m.end():end]:
                yield m.group(1), text[m.end():end]


KERNELS = dict(kernels())


def test_every_early_kernel_is_found():
    assert {"k_boundary", "k_gradient", "k_cell", "k_face", "k_face_staged", "k_face_sides", "k_cell_fluxes",
            "k_step_end", "k_newton_residual", "k_arnoldi_dots", "k_arnoldi_update"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_flags_are_read_behind_the_wait(name):
    # threads with nothing to do wait and leave: only their condition comes before the others' wait
    body = LEAVE.sub(r"\1", KERNELS[name])
    before = body.split("wait_for_previous();")[0]
    assert not WRITTEN.search(before), WRITTEN.search(before).group(0)
