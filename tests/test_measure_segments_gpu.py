"""Area and volume of components that each reach through many triangle
chunks (parallel rods along z, the order bricks come in): more (component,
chunk) partials than the measure first makes room for.  Equal to the oracle's
sums bit for bit, as are the mesh's bytes, so no tolerance applies."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rods,length", [(1, 12), (24, 130)])
def test_rods_equal_oracle(rods, length):
    from sesmesh_b200 import surface as S
    s = np.array([[6.0 * (k % 6), 6.0 * (k // 6), 1.1 * z, 1.7] for k in range(rods) for z in range(length)])
    h = 0.3
    out = S.compute_surface(s, S.SurfaceParams.vdw().with_spacing(h))
    ref = O.Surface(s, 0.0, h, kind="vdw")
    nt, nc = out.stats["triangles"], out.stats["components"]
    assert nc == rods == int(ref.stats["components"]) and nt == int(ref.stats["triangles"])
    chunks = -(-nt // 16384)
    if rods > 1:  # more partials than four per component and chunk
        comp = out.vertex_component[out.triangles[:, 0]]
        assert rods * chunks > 4 * (nc + chunks) + 256 and len(np.unique(comp)) == rods
    assert out.stats["area"] == ref.stats["area"] and out.stats["volume"] == ref.stats["volume"]
    m = ref.mesh()
    assert np.array_equal(out.positions.view(np.uint32), m["positions"].view(np.uint32))
    assert np.array_equal(out.triangles, m["triangles"])
