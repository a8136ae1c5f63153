"""The pointwise pass on pixel models, at odd sizes.

Oracle: an extruded image of one layer solved by the 3D passes for any matrix has the tensor of its
2D image (the solution does not depend on z).
"""
import zlib

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multirhs", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,nmat", [((1, 2), 2), ((5, 7), 2), ((33, 31), 4), ((8, 34), 3), ((64, 128), 2)])
@pytest.mark.parametrize("analysis", ["conductivity", "elasticity"])
def test_pixels_equal_one_layer_of_voxels(monkeypatch, analysis, shape, nmat, precision, multirhs):
    from chfem_b200 import compute_property
    monkeypatch.setenv("CHFEM_B200_THERMAL_OP", "generic")
    monkeypatch.setenv("CHFEM_B200_BLOCK_OP", "element")
    img = H.small_image(shape, nmat, seed=zlib.crc32(repr(shape).encode()) % 1000)
    vals = [(1.0, 0.3), (10.0, 0.2), (4.0, 0.25), (0.5, 0.35)]
    props = {int(c): (vals[i] if analysis == "elasticity" else vals[i][0]) for i, c in enumerate(np.unique(img))}
    kw = dict(mat_props=props, solver_tolerance=1e-9 if precision == "fp64" else 1e-7, solver_maxiter=20000, precision=precision)
    C2 = np.array(compute_property(analysis, img, multirhs=multirhs, **kw))
    C3 = np.array(compute_property(analysis, img[None], **kw))
    ax = [0, 1, 5] if analysis == "elasticity" else [0, 1]  # plane strain: xx, yy, xy
    # both stop at tol: the tensor's error is of the order tol; FP32 fields add theirs
    assert H.rel_to_max(C2, C3[np.ix_(ax, ax)]) < (1e-6 if precision == "fp64" else 1e-4)
