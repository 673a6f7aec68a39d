"""Adam at a learning rate that underflows: the step counts and the moments go
on, so a later step at a usual rate starts from them."""
import numpy as np
import pytest

from cindergs_b200 import GpuPipelineState, PolyCageMesh

pytestmark = pytest.mark.gpu


def test_moments_go_on_where_the_rate_underflows():
    cage = PolyCageMesh.icosphere([0, 0, 0], 1.15, 1)
    V = cage.num_vertices
    rng = np.random.default_rng(4)
    # eight equal rows, so that every batch is the same whatever rows are drawn
    data = []
    for _ in range(2):
        w = rng.random(V) ** 4
        data.append((np.repeat(rng.uniform(-0.4, 0.4, (1, 3)), 8, 0).astype(np.float32),
                     np.repeat((w / w.sum())[None], 8, 0).astype(np.float32)))
    st = GpuPipelineState(0)
    try:
        st.mvc_cage_upload(cage)
        st.mvc_field_create(seed=2)
        p0 = st.mvc_field_params().astype(np.float64)
        g = [st.mvc_field_grads(*d, lam=0.05)[0].astype(np.float64) for d in data]
        # the smallest float32 number, times the schedule's factor of 1 down to
        # 0.05: 0 from below a half on; no parameter moves
        steps = 20
        st.mvc_field_train(*data[0], steps=steps, batch=8, lr=1.4e-45, lam=0.05)
        np.testing.assert_array_equal(st.mvc_field_params(), p0.astype(np.float32))
        st.mvc_field_train(*data[1], steps=1, batch=8, lr=1e-3, lam=0.05)
        p1 = st.mvc_field_params().astype(np.float64)
    finally:
        st.close()
    m, v = np.zeros_like(p0), np.zeros_like(p0)
    for k in range(steps + 1):
        gk = g[0] if k < steps else g[1]
        m, v = 0.9 * m + 0.1 * gk, 0.999 * v + 0.001 * gk * gk
    t = steps + 1
    want = 1e-3 * (m / (1 - 0.9**t)) / (np.sqrt(v / (1 - 0.999**t)) + 1e-8)
    # where neither gradient is near the 1e-8 of the denominator; a parameter
    # (at most 1 here) is rounded to 2^-24 of itself, the moments to 1e-6 of the
    # step of at most 3e-3
    on = (np.abs(g[0]) > 1e-6) & (np.abs(g[1]) > 1e-6) & (np.abs(p0) <= 1.0)
    assert on.sum() > 1000
    np.testing.assert_allclose((p0 - p1)[on], want[on], atol=1e-6, rtol=0)
