"""Subtrees of <= 32 objects against the oracle, bit for bit, at the sizes,
profiles and values where the warp builder's sorted orders and masks can go
wrong (needs a B200): every root size, equal coordinates and centroids, areas
outside the range of the reciprocal form of the cost's division."""
import numpy as np
import pytest

from tests.gpuhelp import gpu_build
from tests.treecheck import compare_exact

pytestmark = pytest.mark.gpu

PROFILES = [dict(), dict(bins=16, adaptive_max_n=0), dict(bins=32, adaptive_steps=16), dict(adaptive_steps=1),
            dict(adaptive_steps=32), dict(bins=3, adaptive_max_n=12, adaptive_steps=5), dict(adaptive_max_n=5)]
LEAVES = [(1, 1), (1, 4), (2, 4), (3, 3)]


def boxes(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "lattice":  # equal coordinates and centroids on every axis
        lo = rng.integers(0, 3, size=(n, 3))
        return np.concatenate([lo, lo + rng.integers(0, 2, size=(n, 3))], axis=1).astype(np.float32)
    if kind == "pairs":  # each box twice: forced medians at the pairs
        lo = rng.uniform(-1.0, 1.0, size=((n + 1) // 2, 3))
        b = np.concatenate([lo, lo + rng.uniform(0.0, 0.2, size=lo.shape)], axis=1)
        return np.repeat(b, 2, axis=0)[rng.permutation(2 * len(b))[:n]].astype(np.float32)
    lo = rng.uniform(-1.0, 1.0, size=(n, 3))
    scale = {"random": 1.0, "tiny": 2.0 ** -31, "denormal_areas": 2.0 ** -66, "huge": 2.0 ** 31}[kind]
    b = np.concatenate([lo, lo + rng.exponential(0.1, size=(n, 3))], axis=1) * scale
    return b.astype(np.float32) + np.float32(0.0)


def same(oracle, ctx, **kw):
    o = oracle.build(**kw)
    g = gpu_build(ctx, **kw)
    assert g["status"] == o["status"], (g["status"], g["error"], o["status"])
    if o["status"] >= 0:
        msg = compare_exact(g["nodes"], g["lens"], g["perm"], o["nodes"], o["lens"], o["perm"])
        assert msg is None, msg


@pytest.mark.parametrize("kind", ["random", "lattice", "pairs", "tiny", "denormal_areas", "huge"])
@pytest.mark.parametrize("profile", range(len(PROFILES)))
def test_subtree_sizes(oracle, gpu_ctx, kind, profile):
    for n in (2, 3, 4, 7, 8, 9, 15, 16, 17, 24, 31, 32):
        for mn, mx in LEAVES:
            same(oracle, gpu_ctx, aabbs=boxes(kind, n, 100 * n + profile), min_leaf=mn, max_leaf=mx,
                 **PROFILES[profile])


@pytest.mark.parametrize("kind", ["random", "lattice", "pairs", "tiny"])
@pytest.mark.parametrize("profile", [0, 1, 2, 5])
def test_many_subtrees(oracle, gpu_ctx, kind, profile):
    same(oracle, gpu_ctx, aabbs=boxes(kind, 3000, 7 + profile), **PROFILES[profile])
    same(oracle, gpu_ctx, aabbs=boxes(kind, 2999, 8 + profile), min_leaf=2, max_leaf=4, max_depth=13,
         **PROFILES[profile])
