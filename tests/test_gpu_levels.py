"""Level passes against the oracle, bit for bit, where tiles and bins meet
(needs a B200): nodes around the tile sizes, runs of neighbours in object
order (lanes that share bins), flat and coincident axes, medians and leaves
among the nodes of one pass, and batched meshes of uneven size."""
import numpy as np
import pytest
import torch

from marigold_b200 import BvhSettings, build_batch_device, synth
from tests.gpuhelp import gpu_build
from tests.treecheck import compare_exact

pytestmark = pytest.mark.gpu


def same(oracle, ctx, **kw):
    o = oracle.build(**kw)
    g = gpu_build(ctx, **kw)
    assert g["status"] == o["status"], (g["status"], g["error"], o["status"])
    if o["status"] >= 0:
        msg = compare_exact(g["nodes"], g["lens"], g["perm"], o["nodes"], o["lens"], o["perm"])
        assert msg is None, msg


def boxes(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "runs":  # a curve in order: neighbours share bins on every axis
        x = np.arange(n) / n
        lo = np.stack([x, np.sin(7 * x), x * x], 1)
    elif kind == "grid":  # rows in order, flat in y
        w = int(np.ceil(np.sqrt(n)))
        i = np.arange(n)
        lo = np.stack([i // w, np.zeros(n), i % w], 1) / w
    elif kind == "half":  # runs, then random objects
        x = np.arange(n) / n
        lo = np.where((np.arange(n) < n // 2)[:, None], np.stack([x, x, 1 - x], 1), rng.random((n, 3)))
    else:
        lo = rng.random((n, 3))
    ext = rng.random((n, 3)) * 0.01
    if kind == "grid":
        ext[:, 1] = 0.0
    return np.concatenate([lo, lo + ext], 1).astype(np.float32) + np.float32(0.0)


@pytest.mark.parametrize("kind", ["random", "runs", "grid", "half"])
def test_tile_edges(oracle, gpu_ctx, kind):
    for n in (1025, 1535, 1536, 1537, 2560, 2561, 5119, 5121, 20480, 65537):
        same(oracle, gpu_ctx, aabbs=boxes(kind, n, n))


@pytest.mark.parametrize("kw", [dict(bins=16), dict(bins=2), dict(max_depth=3), dict(min_leaf=700, max_leaf=3000),
                                dict(min_leaf=1, max_leaf=40000)])
@pytest.mark.parametrize("kind", ["random", "half"])
def test_profiles_and_leaves(oracle, gpu_ctx, kind, kw):
    same(oracle, gpu_ctx, aabbs=boxes(kind, 30011, 5), **kw)


def test_medians_beside_splits(oracle, gpu_ctx):
    b = boxes("random", 12000, 9)
    b[3000:9000] = np.float32([0.25, 0.5, 0.75, 0.5, 0.625, 0.875])
    same(oracle, gpu_ctx, aabbs=b)


@pytest.mark.parametrize("n", [586752, 600000, 1200000, 1600000])
def test_tile_sizes_of_large_builds(oracle, gpu_ctx, n):
    v, t = synth.random_triangles(n, 3)
    same(oracle, gpu_ctx, vertices=v, triangles=t)


def test_batch_of_uneven_meshes(oracle, gpu_ctx):
    sizes = [1, 40, 5000, 700, 1025, 33, 2561, 100000, 2]
    sets = [boxes(("random", "runs", "grid", "half")[i % 4], n, i) for i, n in enumerate(sizes)]
    total = sum(sizes)
    slots = sum(2 * n - 1 for n in sizes)
    nodes = torch.zeros(slots * 8, dtype=torch.int32, device="cuda")
    lens = torch.zeros(slots, dtype=torch.int32, device="cuda")
    perm = torch.zeros(total, dtype=torch.int32, device="cuda")
    dev = [{"aabbs": torch.from_numpy(b).cuda()} for b in sets]
    torch.cuda.synchronize()
    offs, rc, _ = build_batch_device(gpu_ctx, BvhSettings(), dev, nodes, perm, out_lens=lens)
    assert rc == 0
    nh = nodes.cpu().numpy().view(np.uint32).reshape(-1, 8)
    lh, ph = lens.cpu().numpy().view(np.uint32), perm.cpu().numpy().view(np.uint32)
    first = 0
    for i, b in enumerate(sets):
        o = oracle.build(aabbs=b)
        msg = compare_exact(nh[offs[i]:offs[i + 1]], lh[offs[i]:offs[i + 1]], ph[first:first + sizes[i]],
                            o["nodes"], o["lens"], o["perm"])
        assert msg is None, (i, msg)
        first += sizes[i]
