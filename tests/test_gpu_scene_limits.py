"""Trees that the two-level traversal's 31-bit references cannot hold are
refused when the scene is bound, from the counts alone (the arrays here are as
small as a scene of one triangle needs; no call below reads past them)."""
import ctypes

import numpy as np
import pytest

from marigold_b200 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

HALF = 1 << 31


def _bind(tracer, *, tlas_nodes=1, instances=1, tlas_lens=False, blas_nodes=1, mesh_triangles=1, blas_lens=False):
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    node = torch.zeros(8, dtype=torch.int32, device="cuda")
    one = torch.ones(1, dtype=torch.int32, device="cuda")
    inst = torch.zeros(20, dtype=torch.int32, device="cuda")
    mesh = np.array([0, 0, mesh_triangles, 0], np.uint32)
    meshes = torch.from_numpy(mesh.view(np.int32)).cuda()
    verts = torch.eye(3, device="cuda")
    tris = torch.arange(3, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return tracer.L.mgbvh_tracer_set_scene_dev(
        tracer.ptr, vp(node), tlas_nodes, vp(one) if tlas_lens else None, vp(inst), instances, vp(meshes), 1,
        vp(node), blas_nodes, vp(one) if blas_lens else None, vp(verts), 12, 3, vp(tris), mesh_triangles, None)


@pytest.mark.parametrize("kw,status", [
    ({}, _lib.OK),
    # arrays longer than any tree over their objects
    ({"tlas_nodes": HALF + 1, "instances": HALF // 2}, _lib.OK),
    ({"blas_nodes": 2 * HALF - 1}, _lib.OK),
    # as many instances as there are references for, or lens beside them
    ({"instances": HALF}, _lib.OK),
    ({"instances": HALF + 1, "tlas_lens": True}, _lib.OK),
    ({"tlas_nodes": HALF + 1, "instances": HALF // 2 + 1}, _lib.ERR_UNSUPPORTED),
    ({"tlas_nodes": HALF + 1, "instances": HALF // 2 + 1, "tlas_lens": True}, _lib.ERR_UNSUPPORTED),
    ({"instances": HALF + 1}, _lib.ERR_UNSUPPORTED),
    ({"blas_nodes": HALF + 1, "mesh_triangles": HALF // 2 + 1}, _lib.ERR_UNSUPPORTED),
    ({"blas_nodes": HALF + 1, "mesh_triangles": HALF // 2 + 1, "blas_lens": True}, _lib.ERR_UNSUPPORTED),
    ({"mesh_triangles": HALF + 1}, _lib.ERR_UNSUPPORTED),
])
def test_scene_reference_limits(kw, status):
    tr = _lib.Tracer(0)
    assert _bind(tr, **kw) == status
    tr.close()
