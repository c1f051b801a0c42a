"""The tile kernels of the time loop start while the kernel before them is
still writing the step's arrays (programmatic dependent launch).  Those arrays
are not constant for the kernel's lifetime, so none of the kernels, nor of the
device functions they call, may declare them __restrict__."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "optimisation2forme_b200" / "csrc"
WRITTEN = {"U", "Uold", "U32", "keep", "R", "eL", "eR", "ctq", "ctqy", "grad", "alpha", "vq_out", "part", "hist", "st"}
FUNCTIONS = {
    "kernels_tile.cuh": ["tile_gradient", "tile_fluxes", "k_tile_gradient", "k_tile_residual"],
    "kernels.cuh": ["vertex_state_of", "vertex_visc_of", "cell_gradient_body", "cell_gradient_plain",
                    "cell_gradient_from", "cell_residual_sum", "cell_residual_plain", "cell_residual_from"],
    "kernels_f32.cuh": ["cell_residual_mixed_from"],
    "solver_f32.cu": ["k_tile_residual_mixed"],
}


def _parameters(text: str, name: str) -> str:
    m = re.search(r"(?:void|bool|double|Vec4<T>|__launch_bounds__\([^)]*\))\s+" + name + r"\(([^{;]*)\)\s*\{", text)
    assert m, name
    return m.group(1)


@pytest.mark.parametrize("file,name", [(f, n) for f, ns in FUNCTIONS.items() for n in ns])
def test_step_arrays_are_not_restrict(file, name):
    text = re.sub(r"//[^\n]*", "", (CSRC / file).read_text())
    declared = set(re.findall(r"__restrict__\s+(\w+)", _parameters(text, name)))
    assert not declared & WRITTEN


def test_every_dependent_kernel_is_covered():
    """The kernels that wait for the one before them are the ones above."""
    waiting = set()
    for f in ("kernels_tile.cuh", "solver_f32.cu"):
        text = re.sub(r"//[^\n]*", "", (CSRC / f).read_text())
        waiting |= {n for n in re.findall(r"\b(k_tile_\w+)\(", text)}
    assert waiting <= {n for ns in FUNCTIONS.values() for n in ns}
