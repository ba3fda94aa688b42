"""The training step's register tiles against the float64 reference: batches
around a CTA's 32 samples, weights that allow 16-byte loads and weights that
do not.

Bound: a gradient is a sum of products whose FP32 factors carry at most about
200 roundings (three forward sums of up to 64 terms), relative to the largest
gradient: 200 * 2^-24 = 1.2e-5, rounded up to the 2e-5 of the whole step's test.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from marigold_b200 import _lib, learned

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("B", [1, 31, 32, 33, 4097])
def test_train_step_edges(B, shift):
    from oracle import mlp_ref
    L = _lib.load()
    bits = learned.to_bf16_bits(learned.init_params(21))
    rng = np.random.default_rng(B)
    x = rng.normal(scale=0.6, size=(B, 24)).astype(np.float32)
    label = rng.integers(0, 48, B).astype(np.uint32)
    label[::5] = 0xFFFFFFFF
    label[-1] = 47
    gain = (rng.random(B) < 0.5).astype(np.float32)
    w = torch.zeros(learned.NPARAM + 1, dtype=torch.int16, device="cuda")[shift:shift + learned.NPARAM]
    w.copy_(torch.from_numpy(bits.view(np.int16)))
    dx, dl, dg = (torch.from_numpy(a).cuda() for a in (x, label.view(np.int32), gain))
    grad = torch.zeros(learned.NPARAM, device="cuda")
    loss = torch.zeros(2, device="cuda")
    out = torch.empty(B, 49, device="cuda")
    torch.cuda.synchronize()
    assert L.mgbvh_mlp_train_step_dev(_vp(dx), _vp(dl), _vp(dg), B, _vp(w), _vp(grad), _vp(loss), None) == 0
    assert L.mgbvh_mlp_forward_dev(_vp(dx), B, _vp(w), _vp(out), None) == 0
    torch.cuda.synchronize()
    params = (bits.astype(np.uint32) << 16).view(np.float32)
    ref_loss, ref = mlp_ref.loss_and_grad(params, x, label, gain)
    err = np.abs(grad.cpu().numpy().astype(np.float64) - ref).max()
    assert err <= 2e-5 * np.abs(ref).max(), (err, np.abs(ref).max())
    assert abs(float(loss.double().sum().item()) / B - ref_loss) <= 2e-5 * abs(ref_loss)
    logits, _ = mlp_ref.forward(params, x)
    assert np.abs(out.cpu().numpy() - logits).max() <= 2e-5 * np.abs(logits).max()
