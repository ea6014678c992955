"""The debug build's index checks are in the sources: every load of the interpolation kernels'
images, sinograms and planes stands behind CT_DCHECK, CT_DLOAD or a checked ldg_v8 (dbgcheck.cuh).
Read from the text, as no test plants an out-of-range index."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fanbeamctrecon_tensorflowop_gb300" / "csrc"
CHECK = re.compile(r"CT_DCHECK|CT_DLOAD|ldg_v8\(")


@pytest.mark.parametrize("name", ["fp_body.cuh", "fp_adjoint.cu", "bp_body.cuh", "bp_gather.cu",
                                  "cone.cu"])
def test_every_interpolation_file_checks_its_indexes(name):
    assert CHECK.search((CSRC / name).read_text())


def test_every_pixel_load_of_the_gather_transpose_is_checked():
    lines = (CSRC / "bp_gather.cu").read_text().splitlines()
    loads = [k for k, line in enumerate(lines) if re.search(r"\bx\.load\(", line)]
    assert len(loads) >= 4
    for k in loads:
        assert any("CT_DCHECK(in(" in line for line in lines[max(0, k - 2):k + 1]), lines[k]
