"""The training kernels at the sides where their tiles, bands and pipelines can
go wrong: fewer tiles than pipeline stages, images that end inside a tile,
pitches below and above the 32 positions a staging step covers, several tiles
a CTA.

Two properties that hold exactly but for the order of FP32 sums, so that a
misplaced position, tap, band or tile shows at full size:

* every sample of a batch is its own computation (the forward pass of an image
  does not see the others), so under the mean-squared error the gradient of a
  batch of 4 is the mean of the four samples' gradients: the loss gradient
  scales by an exact power of two, and BF16 rounding commutes with it;
* an image mirrored in both axes, through weights mirrored in both axes, is the
  same network: its gradient is the mirrored gradient, up to BF16 rounding of
  sums added in another order.

Tolerances: the first differs by the order of up to 4 * 258^2 FP32 additions
in tiles of 128, ~sqrt(3e5) * 6e-8 = 3e-5 relative at worst: 1e-4. The second
also flips the BF16 rounding (2^-8) of some activations, whose effect on a
layer's gradient is below 2^-8 itself: 1e-2, where a misplaced tap or band
gives errors of order one.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu

CHANNELS = [(2, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 1)]
SIDES = [8, 10, 30, 32, 62, 64, 126, 130, 258]


def setup(side: int):
    from darcy_cpp_gb300 import learn

    a = np.stack([two_phase(side, seed=s) for s in range(4)])
    rng = np.random.default_rng(side)
    u = 1e-2 * (1.0 + 0.1 * rng.standard_normal(a.shape))
    net = learn.WarmStartNet(side, seed=4)
    net.set_loss("mse")
    net.set_scaling([float(np.log(a).mean()), float(np.log(a).std()) or 1.0, 1e-2, 1.0])
    w = net.params() + 0.05 * rng.standard_normal(net.num_params).astype(np.float32)
    net.set_params(w)
    return net, a, u, w


def layers(flat: np.ndarray):
    at = 0
    for ci, co in CHANNELS:
        n = 9 * ci * co
        yield flat[at:at + n].reshape(co, 3, 3, ci), flat[at + n:at + n + co]
        at += n + co


def close(x: np.ndarray, y: np.ndarray, rel: float) -> bool:
    return float(np.linalg.norm(x - y)) <= rel * float(np.linalg.norm(y))


@pytest.mark.parametrize("side", SIDES)
def test_batch_gradient_is_the_mean_of_its_samples(side) -> None:
    net, a, u, _ = setup(side)
    whole, loss = net.gradients(a, u)
    again, _ = net.gradients(a, u)
    assert np.array_equal(whole, again)
    one = [net.gradients(a[q:q + 1], u[q:q + 1]) for q in range(4)]
    mean = np.mean([g.astype(np.float64) for g, _ in one], axis=0)
    assert abs(loss - np.mean([v for _, v in one])) <= 1e-4 * abs(loss)
    for (wg, bg), (wm, bm) in zip(layers(whole), layers(mean)):
        assert close(wg, wm, 1e-4) and close(bg, bm, 1e-4)


@pytest.mark.parametrize("side", SIDES)
def test_mirrored_problem_has_the_mirrored_gradient(side) -> None:
    net, a, u, w = setup(side)
    g, loss = net.gradients(a, u)
    mirrored = np.concatenate([np.concatenate([k[:, ::-1, ::-1].ravel(), b]) for k, b in layers(w)])
    net.set_params(mirrored)
    gm, loss_m = net.gradients(a[:, ::-1, ::-1], u[:, ::-1, ::-1])
    assert abs(loss - loss_m) <= 1e-2 * abs(loss)
    for (k, b), (km, bm) in zip(layers(g), layers(gm)):
        assert close(km[:, ::-1, ::-1], k, 1e-2) and close(bm, b, 1e-2)
