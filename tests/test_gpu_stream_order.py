"""Calls on device tensors run after what the current stream still has to do,
torch's default stream (handle 0) included: the inputs and the output buffers
of every call below are written by work that is still queued when it is made.
Before the queued writes the buffers hold other valid values, so a call that
ran too early would only give another result.
"""
import numpy as np
import pytest

from marigold_b200 import BvhSettings, _lib, build_batch_device, learned, synth
from marigold_b200.bvh import build_device, instance_aabbs_device
from tests.treecheck import compare_exact

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

BUSY = 100_000_000  # clock cycles of the queued work before the writes, about 50 ms


def _boxes(n, seed):
    rng = np.random.default_rng(seed)
    lo = rng.uniform(-50, 50, (n, 3)).astype(np.float32)
    return np.concatenate([lo, lo + rng.uniform(0.1, 3.0, (n, 3)).astype(np.float32)], 1)


def _outputs(n):
    return (torch.zeros((2 * n - 1) * 8, dtype=torch.int32, device="cuda"),
            torch.zeros(2 * n - 1, dtype=torch.int32, device="cuda"),
            torch.zeros(n, dtype=torch.int32, device="cuda"))


def _check(oracle, boxes, count, nodes, lens, perm, **kw):
    want = oracle.build(aabbs=boxes, **kw)
    u32 = lambda t: t.cpu().numpy().view(np.uint32)  # noqa: E731
    msg = compare_exact(u32(nodes).reshape(-1, 8)[:count], u32(lens)[:count], u32(perm),
                        want["nodes"], want["lens"], want["perm"])
    assert msg is None, msg


@pytest.mark.parametrize("side", [False, True])  # the default stream and another current stream
@pytest.mark.parametrize("n", [40, 5000])
def test_build_waits_for_its_input(oracle, n, side):
    first, second = _boxes(n, 1), _boxes(n, 2)
    buf, src = torch.from_numpy(first).cuda(), torch.from_numpy(second).cuda()
    nodes, lens, perm = _outputs(n)
    ctx = _lib.Context(0)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if side else torch.cuda.default_stream()):
        build_device(ctx, BvhSettings(), nodes, perm, aabbs=buf, out_lens=lens)  # scratch is allocated
        torch.cuda._sleep(BUSY)
        buf.copy_(src)
        count, _, _ = build_device(ctx, BvhSettings(), nodes, perm, aabbs=buf, out_lens=lens)
    torch.cuda.synchronize()
    _check(oracle, second, count, nodes, lens, perm)
    ctx.close()


def test_build_waits_for_writes_of_its_outputs(oracle):
    """Leaves of several objects: the caller clears the rows past the tree, and
    the next build uses the same rows before it compacts."""
    n = 3000
    boxes = _boxes(n, 3)
    buf = torch.from_numpy(boxes).cuda()
    nodes, lens, perm = _outputs(n)
    ctx = _lib.Context(0)
    kw = dict(min_leaf_objects=2, max_leaf_objects=4)
    torch.cuda.synchronize()
    count, _, _ = build_device(ctx, BvhSettings(), nodes, perm, aabbs=buf, out_lens=lens, **kw)
    assert count < lens.shape[0]
    for _ in range(2):
        torch.cuda._sleep(BUSY)
        nodes.zero_()
        lens.zero_()
        count, _, _ = build_device(ctx, BvhSettings(), nodes, perm, aabbs=buf, out_lens=lens, **kw)
        nodes[count * 8:].zero_()
        lens[count:].zero_()
    torch.cuda.synchronize()
    _check(oracle, boxes, count, nodes, lens, perm, min_leaf=2, max_leaf=4)
    ctx.close()


def test_instance_boxes_and_batch_wait(oracle):
    """A frame on a new context: mesh boxes still being written, then the
    instances' world boxes, then the TLAS over them as a batch, with its graph."""
    n, m = 600, 5
    ids, xf = synth.scene_instances(4, m, n)
    bounds = [np.sort(np.random.default_rng(k).normal(size=(m, 2, 3)).astype(np.float32), axis=1).reshape(m, 6)
              for k in range(4)]
    d = [torch.from_numpy(b).cuda() for b in bounds]
    mesh_boxes = torch.from_numpy(_boxes(m, 9)).cuda()
    d_ids, d_xf = torch.from_numpy(ids.view(np.int32)).cuda(), torch.from_numpy(xf).cuda()
    world = torch.zeros((n, 6), device="cuda")
    nodes, lens, perm = _outputs(n)
    ctx = _lib.Context(0)
    ctx.set_graph_capture(True)
    torch.cuda.synchronize()
    replays = []
    for k in range(4):
        torch.cuda._sleep(BUSY)
        mesh_boxes.copy_(d[k])
        instance_aabbs_device(ctx, mesh_boxes, d_ids, d_xf, world)
        offs, _, st = build_batch_device(ctx, BvhSettings(), [{"aabbs": world}], nodes, perm, out_lens=lens)
        replays.append(st["graph_replay"])
        torch.cuda.synchronize()
        want, bad = oracle.instance_aabbs(bounds[k], ids, xf)
        assert bad == 0
        assert np.array_equal(world.cpu().numpy().view(np.uint32), want.view(np.uint32))
        _check(oracle, want, offs[-1], nodes, lens, perm)
    assert replays[0] == 0 and 1 in replays  # graphs are captured under the default stream too
    ctx.close()


def test_proposer_weights_wait():
    """Weights still being written when they are handed over: the trees are
    those of the weights written."""
    v, t = synth.noisy_icosphere(5)
    n = t.shape[0]
    dv, dt = torch.from_numpy(v).cuda(), torch.from_numpy(t.view(np.int32)).cuda()
    good = torch.from_numpy(learned.load_weights().view(np.int16)).cuda()
    w = torch.zeros_like(good)
    trees = []
    for late in (False, True):
        ctx = _lib.Context(0)
        w.zero_()
        torch.cuda.synchronize()
        if late:
            torch.cuda._sleep(BUSY)
        w.copy_(good)
        if not late:
            torch.cuda.synchronize()
        ctx.set_split_proposer(w, True)
        nodes, lens, perm = _outputs(n)
        torch.cuda.synchronize()
        _, _, st = build_device(ctx, BvhSettings(), nodes, perm, vertices=dv, triangles=dt, out_lens=lens)
        trees.append((st["learned_splits"], nodes.cpu().numpy(), perm.cpu().numpy()))
        ctx.close()
    assert trees[0][0] == trees[1][0] > 0
    assert np.array_equal(trees[0][1], trees[1][1]) and np.array_equal(trees[0][2], trees[1][2])
