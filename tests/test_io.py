"""chfem .nf / .raw formats (chfem/io.py) and the compute_property argument checks."""
import numpy as np
import pytest

from chfem_b200 import compute_property, export_for_chfem, import_nf, import_raw
from tests import helpers as H


def test_nf_roundtrip(tmp_path):
    img = H.small_image((4, 5, 6), 2, seed=1)
    d = export_for_chfem(str(tmp_path / "a.raw"), img, 1, mat_props={0: (1.0, 0.3), 255: (10.0, 0.2)}, voxel_size=2.0,
                         solver_tolerance=1e-5, solver_maxiter=77)
    nf = import_nf(str(tmp_path / "a.nf"))
    assert nf["image_dimensions"] == (4, 5, 6)
    assert nf["type_of_analysis"] == 1 and nf["number_of_iterations"] == 77
    assert nf["properties_of_materials"] == [(0, 1.0, 0.3), (255, 10.0, 0.2)]
    assert abs(nf["solver_tolerance"] - 1e-5) < 1e-20 and nf["voxel_size"] == 2.0
    back = import_raw(str(tmp_path / "a.raw"), (4, 5, 6))
    assert np.array_equal(back, img)
    assert d["image_dimensions"] == [6, 5, 4]


def test_golden_nf_parses():
    g = H.golden()
    nf = import_nf(H.GOLDEN + "/" + g["fluid_fibers"]["nf"])
    assert nf["refinement"] == 2 and nf["image_dimensions"] == (10, 100, 100)


def test_compute_property_argument_errors():
    a = np.zeros((4, 4, 4), np.uint8)
    with pytest.raises(ValueError, match="Invalid property"):
        compute_property("viscosity", a)
    with pytest.raises(ValueError, match="Invalid direction"):
        compute_property("conductivity", a, mat_props={0: 1.0}, direction="w")
    with pytest.raises(ValueError, match="Invalid solver"):
        compute_property("conductivity", a, mat_props={0: 1.0}, solver="gmres")
    with pytest.raises(ValueError, match="uint8"):
        compute_property("conductivity", a.astype(np.int32), mat_props={0: 1.0})
    with pytest.raises(ValueError, match="No fluid phase"):
        compute_property("conductivity", a + 3, mat_props={3: 1.0})
    with pytest.raises(ValueError, match="Material properties"):
        compute_property("conductivity", a)


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 7), (2, 40, 33), (17, 64, 128)])
def test_colour_histogram_equals_bincount(shape):
    """The native count (threads over chunks of the image) is numpy's for every size and colour."""
    from chfem_b200.io import _color_histogram
    img = np.random.default_rng(5).integers(0, 256, size=shape).astype(np.uint8)
    for a in (img, np.full(shape, 255, np.uint8)):
        hist = _color_histogram(a)
        assert hist.dtype == np.int64 and np.array_equal(hist, np.bincount(a.reshape(-1), minlength=256))


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 2, 3), (4, 1, 5), (3, 5, 1), (6, 7, 9)])
def test_node_keys_name_the_eight_voxels(tmp_path, shape):
    """2 bits per local node e: the material of the voxel in which the node is corner e, on the
    periodic grid (x: +columns, y: -rows, z: -layers; nodes stored rows fastest)."""
    from tests.test_gpu_parity import host_arrays
    img = H.small_image(shape, 4, seed=3)
    nf, raw = H.write_small_case(str(tmp_path), "keys", img, 0)
    keys = host_arrays(nf, raw)["keys"]
    mat = np.searchsorted(np.unique(img), img).transpose(0, 2, 1)  # (layers, columns, rows)
    ref = np.zeros(mat.shape, np.int64)
    for e, (dl, dc, dr) in enumerate([(0, 0, 1), (0, 1, 1), (0, 1, 0), (0, 0, 0), (1, 0, 1), (1, 1, 1), (1, 1, 0), (1, 0, 0)]):
        ref |= np.roll(mat, (dl, dc, dr), axis=(0, 1, 2)) << (2 * e)
    assert np.array_equal(keys, ref.reshape(-1))
