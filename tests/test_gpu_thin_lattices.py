"""Every sweep schedule on lattices one or two voxels wide, where a voxel's neighbours along an
axis may all lie outside: bit-identical grids, equal to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCHEDULES = (0, 12, 13, 14, 15, 16, 21, 31, 41, 51, 43, 44, 46, 53)


@pytest.mark.parametrize("dims", [(1, 21, 20), (1, 65, 9), (2, 33, 18), (3, 20, 21), (1, 1, 40), (1, 40, 1), (40, 1, 1), (1, 1, 1)])
def test_thin_lattices(engine, oracle, dims):
    from gbsdf import meshgen

    # a slab of a sphere's shell: the band does not reach the far ends
    v, f = meshgen.perturbed_sphere(seed=4, n_lat=16, n_lon=32, base_radius=7.0)
    tris = meshgen.to_triangles(np.asarray(v) + (0.2, 0.3, 0.1), np.asarray(f))
    mn = -(np.asarray(dims) // 3)
    mx = mn + np.asarray(dims) - 1
    st, ref, _, _ = oracle.fast_sdf(tris, 1.0, mn, mx, fsm_mode=0, gwn_mode=1, signed_parity=True)
    for sched in (11,) + SCHEDULES:
        out, res = engine.compute_mesh_sdf(tris, 1.0, mn, mx, mode=engine.MODE_EXACT_SIGNS, path=engine.PATH_FAST,
                                           sweep_schedule=sched, raise_on_error=False)
        assert res.status == st, sched
        if st == oracle.OK:
            assert np.array_equal(out.view(np.uint32), ref.view(np.uint32)), sched
