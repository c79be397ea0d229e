"""The finishing kernels (background blend, SSAA mean, clip; one launch for
all cameras) against the tensor operations they stand for, forward and
backward: odd planes (no 16-byte words), one pixel, more cameras than a
launch holds, a camera without a gradient, NaN and infinities."""

from __future__ import annotations

import pytest
import torch

from meshtryoshka_gb300 import triangle_rasterization as tr

pytestmark = pytest.mark.gpu

BACKGROUND = (0.25, 0.5, 0.875)


def _raw(shapes, ssaa, device, seed=0):
    rng = torch.Generator(device).manual_seed(seed)
    n = sum(4 * h * w * ssaa * ssaa for h, w in shapes)
    return torch.rand(n, generator=rng, device=device) * 1.6 - 0.3  # on both sides of the clip


def _operations(raw, background, shapes, ssaa, clip=True):
    images, start = [], 0
    for h, w in shapes:
        n = 4 * h * w * ssaa * ssaa
        r = raw[start:start + n].view(4, h, ssaa, w, ssaa)
        image = (r[:3] + r[3:] * background[:, None, None, None, None]).mean((2, 4))
        images.append(image.clip(0, 1) if clip else image)
        start += n
    return images


@pytest.mark.parametrize("ssaa", [1, 2, 3])
@pytest.mark.parametrize("shapes", [[(1, 1)], [(4, 6), (5, 7), (33, 1)], [(20, 24)] * 3, [(3, 5)] * 66,
                                    [(70, 61), (1, 1), (64, 64), (129, 100), (16, 128)]],
                         ids=["one", "uneven", "alike", "two-launches", "several-blocks"])
def test_matches_tensor_operations(cuda_device, shapes, ssaa):
    background = torch.tensor(BACKGROUND, device=cuda_device)
    raw = _raw(shapes, ssaa, cuda_device).requires_grad_(True)
    want = _operations(raw, background, shapes, ssaa)
    got = tr.FinishImages.apply(raw, background, tuple(shapes), ssaa, False)
    weights = [torch.randn(x.shape, device=cuda_device) for x in want]
    # A mean within rounding of a clip edge may fall on its other side: no
    # gradient is asked of those values.
    unclipped = _operations(raw, background, shapes, ssaa, clip=False)
    weights = [x * ((u.abs() > 1e-5) & ((u - 1.0).abs() > 1e-5)) for x, u in zip(weights, unclipped)]
    if len(shapes) > 1:
        weights[1] = None  # a camera that the loss does not read
    pairs = lambda images: [(i, x) for i, x in zip(images, weights) if x is not None]  # noqa: E731
    (want_grad,) = torch.autograd.grad(sum((i * x).sum() for i, x in pairs(want)), raw)
    (got_grad,) = torch.autograd.grad(sum((i * x).sum() for i, x in pairs(got)), raw)
    # Values below 2; sums of ssaa^2 of them in some order, one rounding each.
    atol = 0.0 if ssaa == 1 else 2.0 * ssaa * ssaa * 2.0**-24
    for g, w in zip(got, want):
        torch.testing.assert_close(g, w, rtol=0, atol=atol)
    # T's gradient sums three products of gradients (|g| < 6) with the background.
    torch.testing.assert_close(got_grad, want_grad, rtol=0, atol=18.0 * 2.0**-24)


def test_stacked_images_and_unaligned_gradients(cuda_device):
    shapes = ((8, 12),) * 2
    background = torch.tensor(BACKGROUND, device=cuda_device)
    raw = _raw(shapes, 1, cuda_device).view(2, 4, 8, 12).requires_grad_(True)
    got = tr.FinishImages.apply(raw, background, shapes, 1, True)
    torch.testing.assert_close(got, torch.stack(_operations(raw.view(-1), background, shapes, 1)), rtol=0, atol=0)
    grad = torch.randn(got.numel() + 1, device=cuda_device)[1:].view(got.shape)  # 4 bytes past a 16-byte boundary
    (a,) = torch.autograd.grad(got, raw, grad, retain_graph=True)
    (b,) = torch.autograd.grad(got, raw, grad.clone())
    torch.testing.assert_close(a, b, rtol=0, atol=0)


@pytest.mark.parametrize("shape", [(2, 2), (1, 3)])
def test_nan_and_infinities(cuda_device, shape):
    background = torch.tensor(BACKGROUND, device=cuda_device)
    h, w = shape
    raw = torch.tensor([float("nan"), float("inf"), -float("inf"), 0.5], device=cuda_device)[:h * w]
    raw = torch.cat((raw, raw.flip(0), torch.full_like(raw, 0.25), torch.ones_like(raw))).requires_grad_(True)
    (want,) = _operations(raw, background, [shape], 1)
    (got,) = tr.FinishImages.apply(raw, background, (shape,), 1, False)
    torch.testing.assert_close(got, want, rtol=0, atol=0, equal_nan=True)
    (a,) = torch.autograd.grad(want.sum(), raw)
    (b,) = torch.autograd.grad(got.sum(), raw)
    torch.testing.assert_close(b, a, rtol=0, atol=0, equal_nan=True)


def test_other_backgrounds_take_tensor_operations(cuda_device):
    raw = torch.rand(1, 4, 4, 4, device=cuda_device)
    plain = torch.tensor(BACKGROUND, device=cuda_device)
    assert tr._finishable(raw, plain)
    assert not tr._finishable(raw, plain.double())
    assert not tr._finishable(raw, plain[:1])
    assert not tr._finishable(raw, plain.cpu())
    assert not tr._finishable(raw, plain.clone().requires_grad_(True))
    with torch.no_grad():
        assert tr._finishable(raw, plain.clone().requires_grad_(True))
    with torch.autograd.forward_ad.dual_level():
        assert not tr._finishable(raw, torch.autograd.forward_ad.make_dual(plain, torch.ones_like(plain)))


@pytest.mark.parametrize("ssaa", [1, 2])
@pytest.mark.parametrize("shape", [(0, 24), (16, 0), (0, 0)])
def test_images_without_pixels(cuda_device, shape, ssaa):
    """Empty images and zero gradients, from cameras of one size and of several."""
    d = cuda_device
    vertices = torch.tensor([[-1.0, -1, 0], [1, -1, 0], [0, 1, 0]], device=d)
    faces = torch.tensor([[0, 1, 2]], dtype=torch.int32, device=d)
    extrinsics = torch.eye(4, device=d).repeat(2, 1, 1)
    extrinsics[:, 2, 3] = 3.0
    intrinsics = torch.tensor([[10.0, 0, 5], [0, 10, 5], [0, 0, 1]], device=d).repeat(2, 1, 1)
    sdf = torch.zeros(3, device=d, requires_grad=True)
    sh = torch.ones(1, 3, 3, device=d, requires_grad=True)
    args = (vertices, faces, torch.tensor([1], dtype=torch.int32, device=d), sdf, sh, 0, 40.0,
            torch.tensor(BACKGROUND, device=d))
    image = tr.render_fused(extrinsics, intrinsics, shape, *args, ssaa=ssaa)
    assert image.shape == (2, 3, *shape)
    grads = torch.autograd.grad(image.sum(), (sdf, sh))
    assert [g.shape for g in grads] == [(3,), (1, 3, 3)] and not any(g.any() for g in grads)
    if ssaa == 1:
        images = tr.render_cameras(extrinsics, intrinsics, [shape, (0, 7)], *args)
        assert [x.shape for x in images] == [(3, *shape), (3, 0, 7)]
        grads = torch.autograd.grad(sum(x.sum() for x in images), (sdf, sh))
        assert not any(g.any() for g in grads)
        images = tr.render_cameras(extrinsics, intrinsics, [shape, (9, 7)], *args)
        assert [x.shape for x in images] == [(3, *shape), (3, 9, 7)]
