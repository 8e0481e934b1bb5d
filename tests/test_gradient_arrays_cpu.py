"""Which gradient arrays each form of the per-Gaussian backward asks for: the arguments are
checked before any device work, so a refusal shows without a GPU."""
from __future__ import annotations

import ctypes as C

import pytest

INVALID_ARGUMENT = 1
ARRAYS = ("dL_dmeans2D", "dL_dcolors", "dL_dopacity", "dL_dmeans3D", "dL_dcov3D", "dL_dsh", "dL_dscales", "dL_drotations")


def _status(form, missing, precomputed):
    from cfgs import native
    lib = native.load()
    s, g, gr = native.Settings(), native.Gaussians(), native.Gradients()
    s.image_width = s.image_height = 16
    s.viewmatrix = s.projmatrix = s.campos = 256
    g.num_gaussians = 1
    g.sh_coeffs = 1
    g.means3D = g.opacities = 256
    if precomputed:
        g.colors_precomp = g.cov3D_precomp = 256
    else:
        g.shs = g.scales = g.rotations = 256
    for a in ARRAYS:
        setattr(gr, a, None if a in missing else 256)
    return getattr(lib, form)(C.byref(s), C.byref(g), 256, 256, 256, 1, 256, C.byref(gr), None)


@pytest.mark.parametrize("missing", ["dL_dcolors", "dL_dcov3D", "dL_dmeans2D", "dL_dopacity", "dL_dmeans3D"])
@pytest.mark.parametrize("precomputed", [False, True])
def test_the_full_form_asks_for_every_array(missing, precomputed):
    assert _status("cfgs_preprocess_backward", {missing}, precomputed) == INVALID_ARGUMENT


@pytest.mark.parametrize("missing,precomputed", [("dL_dcolors", True), ("dL_dcov3D", True), ("dL_dmeans2D", False),
                                                 ("dL_dopacity", False), ("dL_dmeans3D", True), ("dL_dscales", False),
                                                 ("dL_drotations", False)])
def test_the_inputs_form_asks_for_its_inputs(missing, precomputed):
    assert _status("cfgs_preprocess_backward_inputs", {missing}, precomputed) == INVALID_ARGUMENT
