"""Gradients of the learned field against the oracle's float64 backward pass
where the training kernels change their course: cages at the edges of the loss
kernel's columns per lane and at the largest size, vertex counts that are no
multiple of 8, batches of one and of many ranges of the weight gradients' sums
(512 rows: two, 4,096: sixteen, 4,104: thirteen that hold rows), and batches
that end inside a 128-row tile, a 64-row block or a 32-row group.

Bound: 2% of each parameter block's norm, as for one cage and batch in
test_gpu_field: the two sides round fp32 sums that differ in the last bits, so
an occasional bf16 rounding goes the other way."""
import numpy as np
import pytest

from oracle import mvc_field as of
from cindergs_b200 import GpuPipelineState, PolyCageMesh

pytestmark = pytest.mark.gpu


def globe(V):
    """Closed mesh of V vertices: rings of equal size between two poles."""
    m = V - 2
    rings = max(r for r in range(1, 40) if m % r == 0 and m // r >= 3)
    seg = m // rings
    lat = np.pi * np.arange(1, rings + 1) / (rings + 1)
    lon = 2 * np.pi * np.arange(seg) / seg
    body = np.stack([np.sin(lat)[:, None] * np.cos(lon), np.sin(lat)[:, None] * np.sin(lon),
                     np.cos(lat)[:, None] + 0 * lon], 2).reshape(-1, 3)
    v = 1.2 * np.concatenate([[[0, 0, 1]], body, [[0, 0, -1]]])
    at = lambda r, s: 1 + r * seg + s % seg  # noqa: E731
    t = [[0, at(0, s), at(0, s + 1)] for s in range(seg)]
    for r in range(rings - 1):
        for s in range(seg):
            t += [[at(r, s), at(r + 1, s), at(r + 1, s + 1)], [at(r, s), at(r + 1, s + 1), at(r, s + 1)]]
    t += [[V - 1, at(rings - 1, s + 1), at(rings - 1, s)] for s in range(seg)]
    return PolyCageMesh.new(v.astype(np.float32), t)


@pytest.mark.parametrize("V,B", [(5, 8), (162, 40), (192, 512), (193, 136), (642, 4096),
                                 (42, 4104), (672, 72), (673, 1000), (1022, 264), (1024, 2048)])
def test_gradients(V, B):
    cage = globe(V)
    st = GpuPipelineState(0)
    try:
        st.mvc_cage_upload(cage)
        st.mvc_field_create(seed=V)
        off, _, enc = st.mvc_field_layout()
        p = st.mvc_field_params().astype(np.float64)
        rng = np.random.default_rng(V + B)
        p[off["W5"]:off["W5"] + V * 128] = rng.normal(0, 0.02, V * 128)
        for k in ("b1", "b2", "b3", "b4"):
            p[off[k]:off[k] + 128] = rng.normal(0, 0.1, 128)
        p[off["b5"]:off["b5"] + V] += rng.normal(0, 1e-3, V)
        p = p.astype(np.float32)
        st.mvc_field_params(p)
        pts = rng.uniform(-0.6, 0.6, (B, 3)).astype(np.float32)
        w = rng.random((B, V)) ** 4
        w = (w / w.sum(1, keepdims=True)).astype(np.float32)
        g, loss = st.mvc_field_grads(pts, w, lam=0.5)
        (lw, lr), go = of.loss_and_grads(of.unpack(p, off, V), pts, w, cage.rest_vertices, enc, 0.5)
        assert abs(loss[0] - lw) <= 1e-3 * lw and abs(loss[1] - lr) <= 1e-3 * lr + 1e-9
        for k in of.NAMES:
            ref = go[k].reshape(-1)
            got = g[off[k]:off[k] + ref.size].astype(np.float64)
            assert np.linalg.norm(got - ref) < 2e-2 * np.linalg.norm(ref), k
    finally:
        st.close()
