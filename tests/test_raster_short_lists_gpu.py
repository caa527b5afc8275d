"""Raster forward around the list length (twelve records on average) at which tile 16 changes kernel: a count from the
host takes the pair kernel below it, a count that only the device knows always the group kernel.

Both evaluate the same expressions and add a pixel's samples in list order: images, variances and loss adjoints agree bit
for bit. The losses are sums of the same terms in fp64 in two orders, rounded to fp32 once: one unit in the last place."""

import pytest
import torch

from r2splat_b200 import _fused, scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta,variance", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("n,below", [(1, True), (40, True), ("edge", True), ("edge", False), (4000, False)])
def test_forms_agree(device, n, below, beta, variance):
    c, h, w = 3, 75, 101
    lists = c * 5 * 7
    most = 3000 if n == "edge" else n

    def scene(count):
        prims = scenes.random_primitives(most, 8, 0.03, 0.5, beta_range=(0.5, 4.0) if beta else None,
                                         uncertainty_max=0.1 if variance else None)
        return [None if t is None else t[:count].contiguous().to(device) for t in prims]

    viewmats, Ks = (t.to(device) for t in scenes.orbit_cameras(c, 3.0, 120.0, w, h))

    def forward(count):
        means, quats, scales, dens, b, q = scene(count)
        scales[::7, 0] *= 80.0  # unbounded conics: the strict walk
        _, state = _fused.raster_forward(means, quats, scales, dens, viewmats, Ks, w, h, b, q, 1e-8, 3.0)
        return state, q

    if n == "edge":  # the first count past the line, or the last before it
        lo, hi = 1, most
        while lo < hi:
            mid = (lo + hi) // 2
            lo, hi = (lo, mid) if forward(mid)[0].n_isects >= 12 * lists else (mid + 1, hi)
        n = lo - 1 if below else lo
    state, q = forward(n)
    assert (state.n_isects < 12 * lists) == below
    gen = torch.Generator(device=device).manual_seed(1)
    target = torch.rand((c, h, w), device=device, generator=gen)
    n_used = torch.tensor([state.n_isects], dtype=torch.int64, device=device)

    def render(count, on_device):
        image, v = torch.full_like(target, -5.0), torch.full_like(target, -5.0)
        var = torch.full_like(target, -5.0) if variance else None
        loss, value = target.new_empty(()), target.new_empty(())
        ws = _fused._ws(int(_backend.library().r2s_raster_image_loss_workspace(c, 7, 5)), device)
        _backend.call("r2s_raster_render_image_loss", 0, _ptr(state.records), _ptr(q), int(beta), _ptr(state.offsets),
                      _ptr(state.flatten_ids), count, _ptr(n_used) if on_device else None, c, n, w, h, 16, 7, 5, 0,
                      _ptr(target), 0, 1.0, _ptr(image), _ptr(var), _ptr(v), _ptr(loss), _ptr(value), _ptr(ws),
                      ws.numel(), _fused._stream(device))
        return [t for t in (image, v, var) if t is not None], loss

    host, host_loss = render(state.n_isects, False)
    for count in (0, state.n_isects + 50, 1 << 30):  # unknown, a capacity, a capacity far off
        other, other_loss = render(count, True)
        for a, b in zip(host, other):
            assert torch.equal(a, b)
        assert abs(float(host_loss) - float(other_loss)) <= 1.2e-7 * abs(float(host_loss))
