"""Boxes whose surface areas overflow, and nodes of no area: costs that are
infinite over infinite or zero over zero. The reference's NaN comes before every
other cost; each kernel must take the same split as the oracle."""
import numpy as np
import pytest

from marigold_b200 import BvhSettings, _lib, build_batch_device
from tests.gpuhelp import gpu_build
from tests.treecheck import compare_exact

pytestmark = pytest.mark.gpu

PROFILES = [{}, {"bins": 16, "adaptive_max_n": 0}, {"adaptive_steps": 16}]
SIZES = [5, 30, 200, 1500, 5000]  # one threshold per object, a warp, a CTA, level passes


def _boxes(n, kind):
    rng = np.random.default_rng(n)
    lo = rng.uniform(-1, 1, (n, 3))
    b = np.concatenate([lo, lo + rng.uniform(0, 0.05, (n, 3))], 1)
    if kind == "points":
        b[:, 3:] = b[:, :3]
    elif kind == "some points":
        b[::2, 3:] = b[::2, :3]
    else:
        b *= kind
    return b.astype(np.float32) + np.float32(0.0)


def _check(got, want):
    assert got["status"] == want["status"], got["error"]
    msg = compare_exact(got["nodes"], got["lens"], got["perm"], want["nodes"], want["lens"], want["perm"])
    assert msg is None, msg


@pytest.mark.parametrize("kw", PROFILES)
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("scale", [1e19, 2e19, 1e20, 1e37])
def test_areas_that_overflow(oracle, gpu_ctx, n, scale, kw):
    boxes = _boxes(n, scale)
    for leaf in ({}, {"max_leaf": 4}):
        _check(gpu_build(gpu_ctx, aabbs=boxes, profiling=False, **kw, **leaf), oracle.build(aabbs=boxes, **kw, **leaf))


@pytest.mark.parametrize("kw", PROFILES)
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["points", "some points"])
def test_a_root_of_no_area(oracle, gpu_ctx, n, kind, kw):
    boxes = _boxes(n, kind)
    for bounds in ([0.0] * 6, [1.0] * 3 + [-1.0] * 3):
        _check(gpu_build(gpu_ctx, aabbs=boxes, root_bounds=bounds, profiling=False, **kw),
               oracle.build(aabbs=boxes, root_bounds=bounds, **kw))


@pytest.mark.parametrize("kw", PROFILES)
@pytest.mark.parametrize("n", SIZES)
def test_extents_that_overflow(oracle, gpu_ctx, n, kw):
    """Flat boxes that span more than the largest float: areas are zero times
    infinite, under a root area that is an ordinary number or none of it."""
    rng = np.random.default_rng(n)
    lo = rng.uniform(-3.3e38, 3.3e38, (n, 3))
    boxes = np.concatenate([lo, np.minimum(lo + rng.uniform(0, 1e37, (n, 3)), 3.3e38)], 1)
    boxes[:, [1, 4]] = 0
    boxes = boxes.astype(np.float32) + np.float32(0.0)
    for bounds in (None, [0.0] * 3 + [1.0] * 3, [0.0] * 6):
        _check(gpu_build(gpu_ctx, aabbs=boxes, root_bounds=bounds, profiling=False, **kw),
               oracle.build(aabbs=boxes, root_bounds=bounds, **kw))


@pytest.mark.parametrize("queue", [False, True])
def test_areas_that_overflow_in_a_batch(oracle, queue):
    import torch
    lists = [_boxes(n, 2e19) for n in SIZES]
    total = sum(SIZES)
    slots = 2 * total - len(SIZES)
    nodes = torch.zeros(slots * 8, dtype=torch.int32, device="cuda")
    lens = torch.zeros(slots, dtype=torch.int32, device="cuda")
    perm = torch.zeros(total, dtype=torch.int32, device="cuda")
    ctx = _lib.Context(0)
    ctx.set_batch_mode(queue)
    descs = [{"aabbs": torch.from_numpy(b).cuda()} for b in lists]
    offs, rc, _ = build_batch_device(ctx, BvhSettings(), descs, nodes, perm, out_lens=lens)
    torch.cuda.synchronize()
    assert rc >= 0
    nodes, lens, perm = (x.cpu().numpy().view(np.uint32) for x in (nodes, lens, perm))
    first = 0
    for m, b in enumerate(lists):
        want = oracle.build(aabbs=b)
        msg = compare_exact(nodes.reshape(-1, 8)[offs[m]:offs[m + 1]], lens[offs[m]:offs[m + 1]],
                            perm[first:first + b.shape[0]], want["nodes"], want["lens"], want["perm"])
        assert msg is None, f"{b.shape[0]} boxes: {msg}"
        first += b.shape[0]
    ctx.close()
