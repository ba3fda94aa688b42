"""A captured batch and the context's scratch: a larger build on the same
context moves the scratch, so the graph captured before must not be replayed."""
import numpy as np
import pytest

from marigold_b200 import BvhSettings, _lib, build_batch_device, synth
from marigold_b200.bvh import build_device

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _mesh(n, seed):
    v, t = synth.random_triangles(n, seed=seed)
    return torch.from_numpy(v).cuda(), torch.from_numpy(t.view(np.int32)).cuda()


def _outputs(n, meshes=1):
    slots = 2 * n - meshes
    return (torch.zeros(slots * 8, dtype=torch.int32, device="cuda"),
            torch.zeros(slots, dtype=torch.int32, device="cuda"),
            torch.zeros(n, dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("queue", [False, True])
@pytest.mark.parametrize("larger", ["single", "batch"])
def test_graph_goes_with_the_scratch_it_was_captured_on(queue, larger):
    sizes = [20, 700, 3000]
    descs = [{"vertices": v, "triangles": t} for v, t in (_mesh(n, 30 + n) for n in sizes)]
    total = sum(sizes)
    out = _outputs(total, len(sizes))
    ctx = _lib.Context(0)
    ctx.set_graph_capture(True)
    ctx.set_batch_mode(queue)

    def batch():
        for o in out:
            o.zero_()
        offs, _, st = build_batch_device(ctx, BvhSettings(), descs, out[0], out[2], out_lens=out[1])
        return st["graph_replay"], [offs] + [o.cpu().numpy() for o in out]

    first, want = batch()
    again, got = batch()
    assert (first, again) == (0, 1)
    v, t = _mesh(60000, 5)
    big = _outputs(60000)
    if larger == "single":
        build_device(ctx, BvhSettings(), big[0], big[2], vertices=v, triangles=t, out_lens=big[1])
    else:
        ctx.set_batch_mode(False)
        build_batch_device(ctx, BvhSettings(), [{"vertices": v, "triangles": t}], big[0], big[2], out_lens=big[1])
        ctx.set_batch_mode(queue)
    replays = []
    for _ in range(3):
        replay, got = batch()
        replays.append(replay)
        assert got[0] == want[0]
        for a, b in zip(got[1:], want[1:]):
            assert np.array_equal(a, b)
    assert replays == [0, 1, 1]
    ctx.close()
