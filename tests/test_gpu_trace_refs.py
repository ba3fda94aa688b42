"""The edges of the traversal kernels' dispatch and stacks (needs a B200):
node arrays at every alignment they are taken at, leaves of one and of several
objects, trees deeper than the part of the stack in shared memory and up to the
stack's limit, and ray counts around a warp and a CTA. The trees are written by
hand as combs whose visits can be counted: a ray that meets the boxes from the
deep end visits every node, holds one leaf per level on its stack and tests
every triangle. Hits must be brute force's bit for bit."""
import ctypes

import numpy as np
import pytest

from marigold_b200 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NODE = np.dtype([("lo", "<f4", 3), ("start", "<u4"), ("hi", "<f4", 3), ("child", "<u4")])


def _vp(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def comb(levels, per_leaf=1):
    """Leaf i of the comb at z = i, in front of (below) the rest: nodes, lengths,
    vertices and triangles."""
    n = levels * per_leaf
    verts = np.zeros((n, 3, 3), np.float32)
    tri = np.array([[-1, -1, 0], [1, -1, 0], [0, 1, 0]], np.float32)
    for i in range(n):
        verts[i] = tri
        verts[i, :, 2] = i // per_leaf + (i % per_leaf) / 16
    nodes = np.zeros(2 * levels - 1, NODE)
    lens = np.zeros(2 * levels - 1, np.uint32)

    def put(k, a, b, child):  # a node over leaves [a, b)
        nodes[k]["lo"] = verts[a * per_leaf:b * per_leaf].min((0, 1))
        nodes[k]["hi"] = verts[a * per_leaf:b * per_leaf].max((0, 1))
        nodes[k]["start"], nodes[k]["child"], lens[k] = a * per_leaf, child, (b - a) * per_leaf

    k = 0
    for i in range(levels - 1):  # node k holds leaves [i, levels); its children: leaf i, the rest
        put(k, i, levels, 2 * i + 1)
        put(2 * i + 1, i, i + 1, 0)
        k = 2 * i + 2
    put(k, levels - 1, levels, 0)
    return nodes, lens, verts.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def on_device(nodes, offset):
    """The node array `offset` bytes past a 256-byte boundary."""
    words = nodes.view(np.int32).reshape(-1)
    buf = torch.zeros(words.size + 64, dtype=torch.int32, device="cuda")
    at = offset // 4
    buf[at:at + words.size] = torch.from_numpy(words.copy()).cuda()
    return buf[at:at + words.size]


def rays_from_deep_end(m, levels):
    r = np.zeros((m, 8), np.float32)
    g = np.random.default_rng(m)
    r[:, 0] = g.uniform(-0.2, 0.2, m)
    r[:, 1] = g.uniform(-0.4, 0.2, m)
    r[:, 2] = levels + 1
    r[:, 6] = -1.0
    return torch.from_numpy(r).cuda()


@pytest.mark.parametrize("levels", [1, 2, 16, 17, 18, 33, 63, 64])
@pytest.mark.parametrize("offset", [0, 16])
@pytest.mark.parametrize("per_leaf", [1, 3])
def test_comb(levels, offset, per_leaf):
    nodes, lens, verts, tris = comb(levels, per_leaf)
    n = tris.shape[0]
    dn = on_device(nodes, offset)
    dl = torch.from_numpy(lens.view(np.int32)).cuda() if per_leaf > 1 else None
    dv, dt = torch.from_numpy(verts).cuda(), torch.from_numpy(tris.view(np.int32)).cuda()
    dp = torch.arange(n, dtype=torch.int32, device="cuda")
    tr = _lib.Tracer(0)
    L = tr.L
    tr.check(L.mgbvh_tracer_set_blas_dev(tr.ptr, _vp(dn), nodes.size, _vp(dl), _vp(dv), 12, verts.shape[0], _vp(dt),
                                         _vp(dp), n, None))
    for m in (1, 31, 33, 127, 129, 1000):
        dr = rays_from_deep_end(m, levels)
        out = torch.empty((4, m), dtype=torch.int32, device="cuda")
        counts = (ctypes.c_uint64 * 3)()
        for cnt in (counts, None):
            tr.check(L.mgbvh_trace_closest_dev(tr.ptr, _vp(dr), m, _vp(out[0]), _vp(out[1]), cnt, None, None))
            if cnt is not None:
                nb = 2 * levels - 1
                assert list(cnt) == [m * nb, m * nb, m * n]
            tr.check(L.mgbvh_trace_bruteforce_dev(tr.ptr, _vp(dr), m, _vp(out[2]), _vp(out[3]), None))
            torch.cuda.synchronize()
            assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])
            assert (out[1] == n - 1).all()
    tr.close()


def test_comb_past_the_stack():
    """One level more than the stack's 64 entries are enough for is an error, as ever."""
    nodes, _, verts, tris = comb(65)
    dn, dv = on_device(nodes, 0), torch.from_numpy(verts).cuda()
    dt = torch.from_numpy(tris.view(np.int32)).cuda()
    dp = torch.arange(65, dtype=torch.int32, device="cuda")
    tr = _lib.Tracer(0)
    L = tr.L
    tr.check(L.mgbvh_tracer_set_blas_dev(tr.ptr, _vp(dn), nodes.size, None, _vp(dv), 12, verts.shape[0], _vp(dt),
                                         _vp(dp), 65, None))
    dr = rays_from_deep_end(40, 65)
    out = torch.empty((2, 40), dtype=torch.int32, device="cuda")
    rc = L.mgbvh_trace_closest_dev(tr.ptr, _vp(dr), 40, _vp(out[0]), _vp(out[1]), None, None, None)
    assert rc == _lib.ERR_CAPACITY
    tr.close()


@pytest.mark.parametrize("t_levels,b_levels", [(1, 1), (2, 3), (16, 2), (17, 20), (48, 49), (48, 50)])
@pytest.mark.parametrize("offsets", [(0, 0), (16, 0), (0, 16)])
@pytest.mark.parametrize("lens", [(False, False), (True, False), (False, True), (True, True)])
def test_scene_comb(t_levels, b_levels, offsets, lens):
    """A comb of instances of one comb mesh, each shifted by a comb's length:
    the ray meets the last instance's last triangle first."""
    pb = 2 if lens[1] else 1
    pt = 2 if lens[0] else 1  # instances per TLAS leaf
    bn, bl, verts, tris = comb(b_levels, pb)
    n_inst = t_levels * pt
    tn, tl, _, _ = comb(t_levels, pt)
    shift = np.array([b_levels * i for i in range(n_inst)], np.float32)
    for k in range(tn.size):
        a, c = int(tn[k]["start"]), int(tl[k])
        tn[k]["lo"] = [-1, -1, shift[a]]
        tn[k]["hi"] = [1, 1, shift[a + c - 1] + b_levels]
    inst = np.zeros((n_inst, 20), np.float32)
    inst[:, [0, 5, 10, 15]] = 1.0
    inst[:, 14] = -shift
    mesh = np.array([[0, 0, tris.shape[0], 0]], np.int32)
    dtn, dbn = on_device(tn, offsets[0]), on_device(bn, offsets[1])
    dtl = torch.from_numpy(tl.view(np.int32)).cuda() if lens[0] else None
    dbl = torch.from_numpy(bl.view(np.int32)).cuda() if lens[1] else None
    di, dm = torch.from_numpy(inst).cuda(), torch.from_numpy(mesh).cuda()
    dv, dt = torch.from_numpy(verts).cuda(), torch.from_numpy(tris.view(np.int32)).cuda()
    tr = _lib.Tracer(0)
    L = tr.L
    tr.check(L.mgbvh_tracer_set_scene_dev(tr.ptr, _vp(dtn), tn.size, _vp(dtl), _vp(di), n_inst, _vp(dm), 1, _vp(dbn),
                                          bn.size, _vp(dbl), _vp(dv), 12, verts.shape[0], _vp(dt), tris.shape[0], None))
    for m in (1, 33, 129):
        dr = rays_from_deep_end(m, n_inst * b_levels + b_levels)
        out = torch.empty((6, m), dtype=torch.int32, device="cuda")
        counts = (ctypes.c_uint64 * 3)()
        rc = L.mgbvh_trace_scene_dev(tr.ptr, _vp(dr), m, _vp(out[0]), _vp(out[1]), _vp(out[2]), counts, None, None)
        if (t_levels - 1) + (b_levels - 2) + 2 > 96:  # at the deepest pair the stack holds a leaf per level above
            assert rc == _lib.ERR_CAPACITY
            continue
        tr.check(rc)
        tr.check(L.mgbvh_trace_scene_bruteforce_dev(tr.ptr, _vp(dr), m, _vp(out[3]), _vp(out[4]), _vp(out[5]), 0, None))
        torch.cuda.synchronize()
        assert torch.equal(out[:3], out[3:])
        assert (out[2] == tris.shape[0] - 1).all()
        assert counts[1] >= m * (2 * t_levels - 1) and counts[2] > 0
    tr.close()
