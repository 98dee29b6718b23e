"""The exact refinement's block passes at the edges of their ranges: few
sub-blocks (wide blocks), long lists (one block to an SM), lists over a
block's shared memory (left to the global slabs, and those over a slab to
the host) and the single edges that fast mode leaves.  Vertices are the host
refinement's byte for byte, so no tolerance applies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sets():
    from sesmesh_b200 import workloads
    g = workloads.globule330()["spheres"]
    u = workloads.globule2800()["spheres"]
    return {"2 spheres": np.array([[0, 0, 0, 1.7], [2.5, 0.3, 0.1, 1.5]]), "33 spheres": g[:33],
            "330 spheres": g, "2800 spheres": u}


@pytest.mark.parametrize("refine", ["exact", "fast"])
@pytest.mark.parametrize("name,h,brick", [("2 spheres", 0.5, 10), ("33 spheres", 0.37, 10), ("330 spheres", 0.2, 8),
                                          ("330 spheres", 0.8, 16), ("2800 spheres", 0.5, 8),
                                          ("2800 spheres", 1.0, 10), ("2800 spheres", 1.3, 10)])
def test_block_passes_equal_host(name, h, brick, refine):
    from sesmesh_b200 import surface as S
    p = S.SurfaceParams.ses(1.4).with_spacing(h).with_brick_size(brick).with_refine(refine)
    got = []
    for on in (True, False):
        eng = S.SurfaceEngine(_sets()[name], p)
        eng.set_exact_on_device(on)
        out = eng.mesh()
        got.append((out.obj(), [out.stats[k] for k in ("vertices", "triangles", "area", "volume",
                                                        "refine_evaluations")]))
        out.close()
        eng.close()
    assert got[0] == got[1]
