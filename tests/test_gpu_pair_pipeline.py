"""The paired x pipeline (schedule 4) writes each chunk's results through two staging buffers: a
buffer may be written again only when the stores of two chunks ago have read it, also where a
warp has one line inside the lattice and one beyond it (dz not a multiple of 8)."""
import re
from pathlib import Path

import numpy as np
import pytest

SRC = Path(__file__).resolve().parent.parent / "rhizome_v24.15_gb300" / "csrc" / "k_eikonal.cu"


def _kernels():
    """{name: body} of the kernels that store through a descriptor."""
    text = re.sub(r"//[^\n]*", "", SRC.read_text())
    out = {}
    for m in re.finditer(r"__global__[^{;]*?\b(\w+)\(const __grid_constant__[^{;]*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        body = text[m.end():i]
        if "tma_store_3d" in body:
            out[m.group(1)] = body
    return text, out


def test_one_bulk_group_a_chunk():
    # `wait_group.read n` counts groups: whatever the number of stores of a chunk, they are one
    # group, committed on every path, and at most one group is left reading before the next chunk
    text, kernels = _kernels()
    assert {"sweep_x_pipe_kernel", "sweep_x_pipe2_kernel"} <= set(kernels)
    helper = text[text.index("void tma_store_3d("):]
    assert "commit_group" not in helper[: helper.index("\n}")]
    for name, body in kernels.items():
        tail = body[body.index("tma_store_3d"):]
        stmts = [s.strip() for s in tail[: tail.index("}")].split(";")]
        stores = [k for k, s in enumerate(stmts) if "tma_store_3d" in s]
        commits = [k for k, s in enumerate(stmts) if s == "tma_store_commit()"]
        waits = [k for k, s in enumerate(stmts) if s == "tma_store_wait_read1()"]
        assert len(commits) == len(waits) == 1, name
        assert max(stores) < commits[0] < waits[0], name
        assert body.count("tma_store_3d") == len(stores) and body.count("tma_store_commit") == 1, name


@pytest.mark.gpu
@pytest.mark.parametrize("dz", [1, 2, 4, 5, 7, 9, 12, 15, 20, 31])
def test_pair_pipeline_ragged_tiles(engine, dz):
    from gbsdf import meshgen

    # rows of 128 chunks, and enough of them to fill the chip: a window of dz slices of the mug
    tris, mn, mx, h = meshgen.workload("mug_c1_128", dims=(161, 161, 161), h=0.5)
    mn, mx = np.array([-300, mn[1], 10]), np.array([723, mx[1], 9 + dz])
    outs = []
    for sched in (11, 14):
        out, res = engine.compute_mesh_sdf(tris, h, mn, mx, mode=engine.MODE_EXACT_SIGNS, path=engine.PATH_FAST,
                                           sweep_schedule=sched)
        assert res.ok and res.stats["sweep_schedule"] == sched
        outs.append(out.view(np.uint32))
    assert np.array_equal(outs[0], outs[1])
