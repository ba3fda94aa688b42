"""Subtree CTAs against the oracle, bit for bit, at the sizes where their parts
meet (needs a B200): nodes split by one warp and by groups of 2 to 16 warps,
centroids on bin boundaries, medians inside a group, and the object counts
around which the CTA's warp count changes."""
import numpy as np
import pytest

from marigold_b200 import synth
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
    if kind == "boundaries":  # centroids at whole 1/32 and 1/16 steps of the root's extent
        c = rng.integers(0, 33, size=(n, 3)) / 32.0
        c[:2] = [[0, 0, 0], [1, 1, 1]]
        h = rng.integers(0, 4, size=(n, 3)) / 64.0
        return np.concatenate([c - h, c + h], axis=1).astype(np.float32) + np.float32(0.0)
    if kind == "near_boundaries":  # one rounding to either side of them
        c = (rng.integers(1, 32, size=(n, 3)) / 32.0).astype(np.float32)
        c = np.nextafter(c, np.where(rng.random((n, 3)) < 0.5, np.float32(0), np.float32(2)), dtype=np.float32)
        c[:2] = [[0, 0, 0], [1, 1, 1]]
        return np.concatenate([c, c], axis=1).astype(np.float32)
    if kind == "coincident":  # medians down to the leaves
        h = rng.integers(1, 64, size=(n, 3)) / 64.0
        return np.concatenate([-h, h], axis=1).astype(np.float32)
    if kind == "chain":  # unbalanced: clusters at geometric distances
        x = 2.0 ** -rng.integers(0, 24, size=(n, 1))
        lo = x * (1.0 + 0.01 * rng.random((n, 3)))
        return np.concatenate([lo, lo * (1.0 + 0.001 * rng.random((n, 3)))], axis=1).astype(np.float32)
    scale = {"random": 1.0, "far": 1.0, "tiny": 2.0 ** -100}[kind]
    lo = (rng.uniform(-1.0, 1.0, size=(n, 3)) + (1000.0 if kind == "far" else 0.0)) * scale
    return np.concatenate([lo, lo + 0.05 * scale * rng.random((n, 3))], axis=1).astype(np.float32) + np.float32(0.0)


@pytest.mark.parametrize("kind", ["random", "far", "tiny", "boundaries", "near_boundaries", "coincident", "chain"])
@pytest.mark.parametrize("kw", [dict(), dict(bins=16, adaptive_max_n=0), dict(bins=31, min_leaf=2, max_leaf=4),
                                dict(max_depth=5)])
def test_subtree_cta(oracle, gpu_ctx, kind, kw):
    for n in (33, 34, 64, 65, 127, 255, 500, 512, 513, 1000, 1023, 1024):
        same(oracle, gpu_ctx, aabbs=boxes(kind, n, 3 * n), **kw)


@pytest.mark.parametrize("kind", ["random", "boundaries", "chain"])
def test_level_passes_and_subtree_ctas(oracle, gpu_ctx, kind):
    for n in (1025, 5000, 30001):
        same(oracle, gpu_ctx, aabbs=boxes(kind, n, n))


@pytest.mark.parametrize("n", [103599, 104400, 150000, 443999, 446000])
def test_object_counts_of_the_warp_count_rule(oracle, gpu_ctx, n):
    v, t = synth.random_triangles(n, 11)
    same(oracle, gpu_ctx, vertices=v, triangles=t)
