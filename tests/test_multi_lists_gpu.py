"""One batch of structures whose candidate lists span the batch passes'
ranges: short lists, lists over the small regions of the sampling and the
refinement (their second passes) and lists past the first pools (gathered
again).  Meshes equal the single-structure path's byte for byte at the same
brick edge, linear and warm start, so no tolerance applies."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("brick", [8, 16])
def test_mixed_list_lengths_equal_single(brick, warm):
    from sesmesh_b200 import native, surface as S, warm_start, workloads
    g = workloads.globule330()["spheres"]
    u = workloads.globule2800()["spheres"]
    structs = [(g[:1], 0.3), (g[:41], 0.1), (g, 0.25), (u[:1500], 0.6), (u, 0.9)]
    structs = [(s, S.SurfaceParams.ses(1.4).with_spacing(h).with_refine("fast").with_brick_size(brick))
               for s, h in structs]
    mlp = native.Mlp(S._device(0), warm_start.load()) if warm else None
    b = S.MultiBatch(structs, config=(brick, 0, 4), warm=mlp)
    b.run()
    for i, (s, p) in enumerate(structs):
        eng = S.SurfaceEngine(s, p)
        if warm:
            eng.set_warm_start(mlp)
        want = eng.mesh()
        assert b.surface(i).obj() == want.obj(), i
        want.close()
        eng.close()
    b.close()
