"""A planned batch's kernel_launches counts what the run launched: the recorded graph, and from the
host the patch rounds and output of the members whose first probe found mismatches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_launches_of_patch_rounds_are_counted(engine):
    from gbsdf import meshgen

    v, f = meshgen.perturbed_sphere(seed=1, n_lat=24, n_lon=48, base_radius=10.0, degree=3, coeff_scale=1.0)
    patching = meshgen.to_triangles(np.asarray(v) + (0.3, 0.2, 0.1), f)
    # the triangles about the poles collapsed: so many mismatches that the first probe ends the build
    diverging = patching.copy()
    c = patching[:, :9].reshape(-1, 3, 3).mean(1)
    hole = np.hypot(c[:, 0], c[:, 1]) < 4.0
    diverging[hole, 3:9] = np.tile(diverging[hole, :3], 2)
    t = diverging.copy()  # the batch reads this array in each run
    with engine.Batch([(t, 1.0, np.full(3, -16, np.int32), np.full(3, 16, np.int32))]) as b:
        st, s0 = b.run()
        assert st[0] != 0 and s0[0]["patch_rounds"] == 0
        t[:] = patching  # new contents in place
        st, s1 = b.run()
        assert st[0] == 0 and s1[0]["patch_rounds"] == 1 and s1[0]["probes"] == 2
        # at least the patch box's marks, blocks, walks and re-checks, the probe and the output
        assert s1[0]["kernel_launches"] >= s0[0]["kernel_launches"] + 10
        t[:] = diverging
        st, s2 = b.run()
        assert s2[0]["kernel_launches"] == s0[0]["kernel_launches"]
