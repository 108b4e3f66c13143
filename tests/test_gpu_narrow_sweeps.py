"""The eikonal's narrow-tile schedules (x 6 and walk 5: tiles of 32 x 4 lines) against the
wide ones, bit for bit, for both update rules; the default plan's line between them; and
their bounded waits, which end in an error status and leave the output untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(dims, h=1.0):
    from gbsdf import meshgen

    tris, mn, mx, h = meshgen.workload("mug_c1_128", dims=dims, h=h)
    return tris, mn, mx, h


# tiles' edges (32, 4), batches of 4 slices and rings of 8 batches: less than one, one, remainders,
# and lattices one voxel thick along each walked axis; a voxel size outside the packed update's range
@pytest.mark.parametrize("dims,h", [((32, 32, 32), 1.0), ((36, 33, 29), 1.0), ((97, 5, 41), 1.0), ((96, 1, 44), 1.0),
                                    ((96, 40, 1), 1.0), ((31, 67, 3), 1.0), ((44, 37, 70), 0.37),
                                    ((40, 36, 44), 3e6)])
@pytest.mark.parametrize("mode", ["EXACT", "EXACT_SIGNS"])
def test_narrow_schedules_identical(engine, dims, h, mode):
    tris, mn, mx, h = _case(dims, h)
    outs = []
    for sched in (11, 43, 53, 46, 56, 0):
        out, res = engine.compute_mesh_sdf(tris, h, mn, mx, mode=getattr(engine, "MODE_" + mode), path=engine.PATH_FAST,
                                           sweep_schedule=sched)
        assert res.ok
        assert sched == 0 or res.stats["sweep_schedule"] == sched
        outs.append(out.view(np.uint32))
    for o in outs[1:]:
        assert np.array_equal(outs[0], o)


# (32 x 16 tiles of the walks, 32 x 8 tiles of the x sweep): 228 / 240 and 234 / 210
@pytest.mark.parametrize("dims,narrow_w,narrow_x", [((378, 300, 300), True, False), ((380, 310, 160), False, True)])
def test_default_plan_by_tiles(engine, dims, narrow_w, narrow_x):
    tris, mn, mx, h = _case(dims)
    _, res = engine.compute_mesh_sdf(tris, h, mn, mx, mode=engine.MODE_EXACT_SIGNS, path=engine.PATH_FAST)
    first = res.stats["sweep_schedule_first"]
    assert (first // 10 == 5) == narrow_w and (first % 10 == 6) == narrow_x
    _, res = engine.compute_mesh_sdf(tris, h, mn, mx, mode=engine.MODE_EXACT, path=engine.PATH_FAST)
    assert res.stats["sweep_schedule"] // 10 == 5


@pytest.mark.parametrize("sched", [53, 46])
@pytest.mark.parametrize("mode", ["REFERENCE", "EXACT"])
def test_narrow_wait_timeout_reports_error(engine, sched, mode):
    from gbsdf import _lib

    tris, mn, mx, h = _case((48, 48, 52))
    mode = getattr(engine, "MODE_" + ("EXACT_SIGNS" if mode == "REFERENCE" else mode))
    buf = np.full(int(np.prod(mx.astype(np.int64) - mn + 1)), 7.0, np.float32)
    _, res = engine.compute_mesh_sdf(tris, h, mn, mx, out=buf, mode=mode, path=engine.PATH_FAST,
                                     sweep_schedule=sched, wait_poll_limit=-1, raise_on_error=False)
    assert res.status == _lib.ECUDA and "timed out" in res.message
    assert np.all(buf == 7.0)
    _, res = engine.compute_mesh_sdf(tris, h, mn, mx, mode=mode, path=engine.PATH_FAST, sweep_schedule=sched)
    assert res.ok
