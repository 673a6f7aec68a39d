"""Fields of several cages in one context: what a batch's buffers hold follows
the cage as well as the rows, so a cage with more vertices after one with fewer
(at the same or a smaller batch) trains and evaluates as in a fresh context,
bit for bit."""
import numpy as np
import pytest

from cindergs_b200 import GpuPipelineState, PolyCageMesh

pytestmark = pytest.mark.gpu


def work(st, level, batch, steps):
    """Parameters, gradients and weights after training a cage's field."""
    cage = PolyCageMesh.icosphere([0, 0, 0], 1.15, level)
    st.mvc_cage_upload(cage)
    st.mvc_field_create(seed=level)
    rng = np.random.default_rng(level)
    n, V = 2 * batch, cage.num_vertices
    pts = (rng.uniform(-0.5, 0.5, (n, 3))).astype(np.float32)
    w = rng.random((n, V), dtype=np.float32) ** 4
    w = (w / w.sum(1, keepdims=True)).astype(np.float32)
    st.mvc_field_train(pts, w, steps=steps, batch=batch, lr=2e-3, lam=0.05, seed=3)
    p = st.mvc_field_params()
    g, _ = st.mvc_field_grads(pts[:batch], w[:batch], lam=0.05)
    return p, g, st.mvc_field_eval(pts)


# (cage level, batch) one after another: 42, 162 and 642 vertices; 65,536 rows
# leave room for every buffer of 16,384 rows of the larger cage but the weight
# gradients' partial sums
@pytest.mark.parametrize("sequence", [[(2, 4096), (3, 4096)], [(1, 264), (3, 264), (2, 264)],
                                      [(2, 65_536), (3, 16_384)]])
def test_cages_one_after_another(sequence):
    st = GpuPipelineState(0)
    try:
        for level, batch in sequence:
            got = work(st, level, batch, 2)
            fresh = GpuPipelineState(0)
            try:
                want = work(fresh, level, batch, 2)
            finally:
                fresh.close()
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
                assert np.isfinite(a).all()
    finally:
        st.close()
