"""Polygon-cage bindings of scenes with an odd number of Gaussians, whose
slot array ends between two 64-bit words: the scan behind it keeps 64-bit
words in the same buffer. The bound set equals the oracle's exactly."""
import numpy as np
import pytest

import oracle
from cindergs_b200 import GpuPipelineState, PolyCageMesh, random_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 599, 4097])
def test_bindings_of_odd_counts(n):
    cage = PolyCageMesh.icosphere([0, 0, 0], 1.15, 2)
    scene = random_scene(n, seed=5)  # means ~ N(0, I): some outside the cage
    scene.positions[0] = 0.1
    inside, _ = oracle.mvc_bind(scene.positions, cage.rest_vertices, cage.triangles)
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        st.upload_cages(None)
        st.mvc_cage_upload(cage)
        assert st.mvc_bind() == int(inside.sum())
        np.testing.assert_array_equal(st.mvc_read_bindings()[0], np.nonzero(inside)[0])
        st.mvc_field_create(seed=3)
        assert st.mvc_bind_learned(threshold=1e9) == (int(inside.sum()), 0)
        assert st.mvc_bind_learned(threshold=0.0) == (int(inside.sum()),) * 2
    finally:
        st.close()
