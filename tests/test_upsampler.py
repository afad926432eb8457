"""Learned flow upsampler (vsc_upsampler_*): the tensor-core inference (FP16
weights and activations, FP32 accumulation) against a float64 numpy
restatement of the net that rounds the same operands to FP16, and against
the same net in FP32 (the error FP16 costs); the bilinear fallback; training
that overfits a small batch; the stabilizer's fast mode with the net
attached, whose two flows (one batched launch) equal single-image calls."""
from __future__ import annotations

import numpy as np
import pytest

RNG = np.random.Generator(np.random.PCG64(31))
LAYERS = [(3, 32), (32, 32), (32, 32), (32, 2)]


def test_param_count(vsc):
    n = sum(co * 9 * ci + co for ci, co in LAYERS)
    assert vsc.Upsampler.param_count() == n == 19970


def _np_forward(params, inp, half_acts=False):
    """The net in float64: 3x3 zero-padded convolutions, ReLU between; with
    half_acts the input and every inner activation are rounded to FP16 (the
    tensor-core path's operands)."""
    rnd = (lambda a: a.astype(np.float16).astype(np.float64)) if half_acts else (lambda a: a)  # noqa: E731
    x = rnd(inp.astype(np.float64))
    off = 0
    for li, (ci, co) in enumerate(LAYERS):
        w = params[off:off + co * 9 * ci].reshape(co, 3, 3, ci).astype(np.float64)
        off += co * 9 * ci
        b = params[off:off + co].astype(np.float64)
        off += co
        h, wd = x.shape[:2]
        xp = np.pad(x, ((1, 1), (1, 1), (0, 0)))
        y = np.tile(b, (h, wd, 1))
        for ky in range(3):
            for kx in range(3):
                y += xp[ky:ky + h, kx:kx + wd] @ w[:, ky, kx, :].T
        x = rnd(np.maximum(y, 0)) if li < 3 else y
    return x


def _base(coarse, w, h):
    """Bilinear upsampling (kernel_bilinear's sampling) with vectors scaled."""
    ch, cw = coarse.shape[:2]
    out = np.empty((h, w, 2))
    for y in range(h):
        for x in range(w):
            xx, yy = np.float32(x * cw / w), np.float32(y * ch / h)
            ix, iy = min(int(np.floor(xx)), cw - 1), min(int(np.floor(yy)), ch - 1)
            fx, fy = xx - ix, yy - iy
            ix1, iy1 = min(ix + 1, cw - 1), min(iy + 1, ch - 1)
            v = (coarse[iy, ix, :2] * (1 - fx) * (1 - fy) + coarse[iy, ix1, :2] * fx * (1 - fy)
                 + coarse[iy1, ix, :2] * (1 - fx) * fy + coarse[iy1, ix1, :2] * fx * fy)
            out[y, x] = v * np.array([w / cw, h / ch])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(24, 36), (45, 261)])
def test_inference_matches_numpy_and_fallback(vsc, cuda, h, w):
    """(45, 261): three 128-pixel segments, the last one partial, and a
    partial band of rows."""
    import torch

    coarse = RNG.normal(0, 1.5, (h // 2, w // 2, 3)).astype(np.float32)
    frame = RNG.random((h, w, 3)).astype(np.float32)
    params = (RNG.normal(0, 0.08, vsc.Upsampler.param_count())).astype(np.float32)
    up = vsc.Upsampler(params)
    dc, df = torch.from_numpy(coarse).to(cuda), torch.from_numpy(frame).to(cuda)
    inp = vsc.Upsampler.prepare(dc, df).cpu().numpy()
    base = _base(coarse, w, h)
    assert np.allclose(inp[..., :2], base, atol=1e-5)
    lum = frame @ np.array([0.299, 0.587, 0.114])
    assert np.allclose(inp[..., 2], lum, atol=1e-6)
    p16 = params.astype(np.float16).astype(np.float32)  # inference weights are FP16
    for i, (ci, co) in enumerate(LAYERS):  # biases stay FP32
        start = sum(c * 9 * a + c for a, c in LAYERS[:i]) + co * 9 * ci
        p16[start:start + co] = params[start:start + co]
    r = _np_forward(p16, inp, half_acts=True)
    up.set_max_residual(1e9)
    got = up.apply(dc, df).cpu().numpy()
    # same FP16 operands, FP32 vs float64 accumulation (an activation's FP16
    # rounding may flip one unit where the two sums straddle a rounding point)
    assert np.allclose(got[..., :2], inp[..., :2] + r, atol=1e-3 * (1 + np.abs(r).max()))
    assert np.all(got[..., 2] == 0)
    # the cost of FP16 activations against the net in FP32 (FP16 weights in both)
    r32 = _np_forward(p16, inp)
    assert np.abs(got[..., :2] - (inp[..., :2] + r32)).max() <= 2e-2 * (1 + np.abs(r32).max())
    up.set_max_residual(0.0)  # every residual is refused: the bilinear base
    got0 = up.apply(dc, df).cpu().numpy()
    keep = np.max(np.abs(r), -1) > 1e-3
    assert np.array_equal(got0[..., :2][keep], inp[..., :2][keep])
    up.close()


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1, 1), (7, 125), (8, 126), (9, 127), (17, 128), (24, 253), (330, 1000)])
def test_inference_at_segment_and_group_edges(vsc, cuda, h, w):
    """Segments of 126 output columns and groups of 8 output rows: one short,
    exact and one over, and an image of more than two groups a block.  Same FP16
    operands as the restatement, FP32 vs float64 sums: the bound of the test
    above."""
    import torch

    coarse = torch.from_numpy(RNG.normal(0, 1.5, ((h + 1) // 2, (w + 1) // 2, 3)).astype(np.float32)).to(cuda)
    frame = torch.from_numpy(RNG.random((h, w, 3)).astype(np.float32)).to(cuda)
    params = RNG.normal(0, 0.08, vsc.Upsampler.param_count()).astype(np.float32)
    params = params.astype(np.float16).astype(np.float32)
    up = vsc.Upsampler(params)
    up.set_max_residual(1e9)
    inp = vsc.Upsampler.prepare(coarse, frame).cpu().numpy()
    r = _np_forward(params, inp, half_acts=True)
    got = up.apply(coarse, frame).cpu().numpy()
    assert np.allclose(got[..., :2], inp[..., :2] + r, atol=1e-3 * (1 + np.abs(r).max()))
    assert np.all(got[..., 2] == 0)
    up.close()


@pytest.mark.gpu
def test_training_overfits_a_batch(vsc, cuda):
    import torch

    n, h, w = 4, 32, 32
    inp = torch.from_numpy(RNG.normal(0, 1, (n, h, w, 3)).astype(np.float32)).to(cuda)
    # target: the base shifted by a smooth function of the luma channel
    tgt = (inp[..., :2] + 0.3 * torch.tanh(inp[..., 2:3])).contiguous()
    up = vsc.Upsampler()
    first = up.train_step(inp, tgt, 3e-3)
    for _ in range(400):
        last = up.train_step(inp, tgt, 3e-3)
    assert last < 0.5 * first, (first, last)
    p = up.params()
    assert np.all(np.isfinite(p))
    up.close()


@pytest.mark.gpu
def test_stabilizer_with_learned_upsampler(vsc, cuda):
    """FLOWDOWNSCALE=2 with the net attached: runs, differs from the bilinear
    fast mode, and with every residual refused uses the scaled bilinear base."""
    from vsc_gb300 import synth

    w, h = 128, 96
    s = synth.SyntheticStream(w, h, seed=71)
    frames = [s.frame(i) for i in range(5)]
    a = vsc.Stabilizer(w, h, flow_downscale=2)
    b = vsc.Stabilizer(w, h, flow_downscale=2)
    up = vsc.Upsampler(RNG.normal(0, 0.05, vsc.Upsampler.param_count()).astype(np.float32))
    up.set_max_residual(1e9)
    b.set_upsampler(up)
    for st in (a, b):
        for i in range(3):
            st.load_frame(*frames[i])
        st.step()
    fa, fb = a.buffer(1).cpu().numpy(), b.buffer(1).cpu().numpy()
    assert not np.allclose(fa, fb)
    # both flows come from one batched launch; each equals the single-image call
    # on the same coarse flow and frame (flow(I1 -> I2) with I1, flow(I2 -> I1) with I2)
    import torch

    from vsc_gb300.train_upsampler import nearest

    f1, f2 = (vsc.char_to_float_image(torch.from_numpy(frames[i][0]).to(cuda)) for i in (1, 2))
    ab, ba = vsc.flow_estimate(nearest(f1, w // 2, h // 2), nearest(f2, w // 2, h // 2))
    assert np.allclose(up.apply(ab, f1).cpu().numpy(), fb, atol=1e-5)
    assert np.allclose(up.apply(ba, f2).cpu().numpy(), b.buffer(2).cpu().numpy(), atol=1e-5)
    with pytest.raises(vsc.VscError, match="ESTATE"):
        vsc.Stabilizer(w, h).set_upsampler(up)
    a.close()
    b.close()
    up.close()


def _reference_steps(params, batches, lr):
    """Adam steps of the L1 loss in float64 (torch autograd on the CPU): parameters after each."""
    import torch

    p = torch.from_numpy(params.astype(np.float64)).requires_grad_()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    out = []
    for k, (inp, tgt) in enumerate(batches, 1):
        x = torch.from_numpy(inp.astype(np.float64)).permute(0, 3, 1, 2)
        at = 0
        for li, (ci, co) in enumerate(LAYERS):
            w = p[at:at + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
            at += co * 9 * ci
            x = torch.nn.functional.conv2d(x, w, p[at:at + co], padding=1)
            at += co
            x = x.relu() if li < 3 else x
        d = torch.from_numpy(inp[..., :2].astype(np.float64)) + x.permute(0, 2, 3, 1) - torch.from_numpy(tgt)
        loss = d.abs().sum() / (d.numel() // 2)
        (g,) = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= lr * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
        out.append((float(loss.detach()), p.detach().numpy().copy()))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (1, 2, 31), (2, 9, 33), (3, 7, 50), (1, 33, 64), (5, 8, 32)])
def test_training_steps_match_float64(vsc, cuda, n, h, w):
    """Two steps on different batches (the first Adam step alone shows only the
    gradients' signs) at the edges of the 32 x 8 and 32 x 2 pixel tiles.  The
    FP32 gradients' rounding (about 1e-5 of a layer's gradient scale) moves an
    update by lr * 1e-5 * scale / |g|: 1e-4 lr in the median, and more than
    1e-2 lr only where |g| is below a thousandth of its layer's scale."""
    import torch

    rng = np.random.Generator(np.random.PCG64(100 * n + 10 * h + w))
    lr = 1e-4
    params = rng.normal(0, 0.1, vsc.Upsampler.param_count()).astype(np.float32)
    batches = [(rng.normal(0, 1, (n, h, w, 3)).astype(np.float32), rng.normal(0, 1, (n, h, w, 2)).astype(np.float32))
               for _ in range(2)]
    up = vsc.Upsampler(params)
    for (inp, tgt), (loss, ref) in zip(batches, _reference_steps(params, batches, lr)):
        got = up.train_step(torch.from_numpy(inp).to(cuda), torch.from_numpy(tgt).to(cuda), lr)
        assert abs(got - loss) <= 1e-5 * loss
        # less the parameters' own rounding (|p| < 1: half a unit is 6e-8 at most)
        err = np.maximum(np.abs(up.params() - ref) - 6e-8, 0) / lr
        assert np.median(err) <= 1e-4 and np.quantile(err, 0.99) <= 1e-2 and err.max() <= 2.5, (err.max(), h, w)
    up.close()


@pytest.mark.gpu
def test_training_ignores_values_where_the_gradient_is_zero(vsc, cuda):
    """An infinite input inside a region without a loss gradient (its targets
    are NaN: neither sign) adds nothing to the weight gradients: the step is
    the one with a finite value in its place."""
    import torch

    h, w = 40, 48
    inp = RNG.normal(0, 1, (1, h, w, 3)).astype(np.float32)
    tgt = RNG.normal(0, 1, (1, h, w, 2)).astype(np.float32)
    tgt[0, 10:31, 10:31] = np.nan  # further than the net's four pixels around (20, 20)
    got = []
    for value in (0.5, np.inf):
        inp[0, 20, 20, 0] = value
        up = vsc.Upsampler("default")
        up.train_step(torch.from_numpy(inp).to(cuda), torch.from_numpy(tgt).to(cuda), 1e-3)
        got.append(up.params())
        up.close()
    assert np.all(np.isfinite(got[1]))
    assert np.quantile(np.abs(got[0] - got[1]), 0.99) <= 1e-5  # the sums' order varies


def _taps_outside(h, w):
    """Mask over the parameters: weights of taps that lie outside an h x w image at every pixel."""
    out = []
    for ci, co in LAYERS:
        m = np.zeros((co, 3, 3, ci), bool)
        if h == 1:
            m[:, [0, 2]] = True
        if w == 1:
            m[:, :, [0, 2]] = True
        out += [m.reshape(-1), np.zeros(co, bool)]
    return np.concatenate(out)


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1, 40), (40, 1), (1, 1), (1, 7)])
def test_training_leaves_taps_outside_the_image_out(vsc, cuda, h, w):
    """A tap outside the image adds nothing whatever its weight: in images of one
    row (or column) the taps above and below (beside) are never inside, so weights
    there that are not finite change nothing.  Bounds as in the test above."""
    import torch

    rng = np.random.Generator(np.random.PCG64(h + 100 * w))
    lr = 1e-4
    outside = _taps_outside(h, w)
    params = rng.normal(0, 0.1, vsc.Upsampler.param_count()).astype(np.float32)
    params[outside] = 0.0
    bad = params.copy()
    bad[outside] = np.resize(np.float32([np.nan, np.inf, -np.inf]), outside.sum())
    batches = [(rng.normal(0, 1, (2, h, w, 3)).astype(np.float32), rng.normal(0, 1, (2, h, w, 2)).astype(np.float32))
               for _ in range(2)]
    up = vsc.Upsampler(bad)
    for (inp, tgt), (loss, ref) in zip(batches, _reference_steps(params, batches, lr)):
        got = up.train_step(torch.from_numpy(inp).to(cuda), torch.from_numpy(tgt).to(cuda), lr)
        assert abs(got - loss) <= 1e-5 * loss
        p = up.params()
        assert np.array_equal(p[outside], bad[outside], equal_nan=True)
        err = np.maximum(np.abs(p - ref)[~outside] - 6e-8, 0) / lr
        assert np.median(err) <= 1e-4 and np.quantile(err, 0.99) <= 1e-2 and err.max() <= 2.5, err.max()
    up.close()


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1, 8), (1, 70), (70, 1)])
def test_weight_gradients_leave_taps_outside_the_image_out(vsc, cuda, h, w):
    """The same for the weight gradients where dz is not finite (an overflow on
    the way back: 3e38 * 1e9): the first layer's taps outside the image keep a
    gradient of zero, those inside get one that is not finite."""
    import torch

    params = np.zeros(vsc.Upsampler.param_count(), np.float32)
    at = 0
    for (ci, co), value in zip(LAYERS, (1e-30, 3e38, 1e10, 1.0)):
        params[at + 4 * ci] = value  # output 0, centre tap, channel 0
        at += co * 9 * ci + co
    inp = np.zeros((1, h, w, 3), np.float32)
    inp[..., 0] = 1.0
    up = vsc.Upsampler(params)
    up.train_step(torch.from_numpy(inp).to(cuda), torch.zeros((1, h, w, 2), device=cuda), 1e-3)
    got = up.params()[:27].reshape(3, 3, 3)  # output 0: [ky][kx][channel]
    outside = _taps_outside(h, w)[:27].reshape(3, 3, 3)
    assert np.array_equal(got[outside], params[:27].reshape(3, 3, 3)[outside])
    assert not np.isfinite(got[~outside]).any()
    up.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,h,w", [(1, 32, 64), (32, 64, 64), (1, 1024, 2048)])
def test_weight_gradient_sums_against_float64(vsc, cuda, n, h, w):
    """The gradients' sums over the pixels, read from one Adam step of a learning
    rate so large that the update is all that is left of a parameter, and with
    gradients (1e-10) far below Adam's epsilon, where it is nearly linear in
    them.  Weights of few bits and a target far below give every pixel the same
    dz, exactly, so only the inputs' products and their sums round.  A sum of m equal terms
    in a row is off by about sqrt(m) / 3 units (2^-24) in the root mean square: 32
    copies in four chains 0.9, 19 or fewer blocks a copy 1.5 and 2,048 pixels a
    thread 15, averaged over 32 copies and 608 blocks to 0.3 and 0.6, reading
    the update about 1; all blocks on one sum would be 8.  The largest batch has more
    than 32 tiles a block."""
    import torch

    rng = np.random.Generator(np.random.PCG64(n + h))
    params, at, spans = np.zeros(vsc.Upsampler.param_count(), np.float32), 0, []
    for li, (ci, co) in enumerate(LAYERS):
        k = co * 9 * ci
        params[at:at + k] = rng.integers(1, 4, k) * 2.0 ** (-38 if li == 3 else -8)
        spans.append((at, k, ci, co))
        at += k + co
    x = rng.random((n, h, w, 3), dtype=np.float32)
    inp = torch.from_numpy(x).to(cuda)
    lr = 1e6
    up = vsc.Upsampler(params)
    up.train_step(inp, torch.full((n, h, w, 2), -10.0, device=cuda), lr)
    moved = (params.astype(np.float64) - up.params()) / lr  # g / (|g| + 1e-8)
    up.close()
    moved[spans[3][0]:] = 0  # (the last layer's gradients are far above the epsilon)
    grad = moved * 1e-8 / (1 - np.abs(moved))

    acts = [inp.double().permute(0, 3, 1, 2)]
    wts = []
    for a, k, ci, co in spans:
        wts.append(torch.from_numpy(params[a:a + k].astype(np.float64)).to(cuda).reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
                   .contiguous())
        if len(wts) < 4:
            acts.append(torch.nn.functional.conv2d(acts[-1], wts[-1], padding=1))
    dz = torch.full((n, 2, h, w), 1.0 / (n * h * w), dtype=torch.float64, device=cuda)
    for li in (2, 1, 0):
        dz = torch.nn.functional.conv_transpose2d(dz, wts[li + 1], padding=1)
        a, k, ci, co = spans[li]
        # correlate x with dz, a tap at a time
        xp = torch.nn.functional.pad(acts[li], (1, 1, 1, 1))
        ref = torch.stack([torch.stack([torch.einsum("nohw,nchw->oc", dz, xp[:, :, ky:ky + h, kx:kx + w])
                                        for kx in range(3)], 1) for ky in range(3)], 1).reshape(-1).cpu().numpy()
        db = dz.sum((0, 2, 3)).cpu().numpy()
        for got, want in ((grad[a:a + k], ref), (grad[a + k:a + k + co], db)):
            rms = np.sqrt(np.mean((got / want - 1) ** 2)) * 2 ** 24
            assert rms <= 4.0, (li, got.size, rms)


@pytest.mark.gpu
def test_training_loss_sum_is_exact(vsc, cuda):
    """512 blocks' equal sums: with parameters of zero and a distance c of 22 bits every
    block's sum is exact in FP32 and so is the loss, 2 c, whatever the order of the
    blocks; added up in FP32 they are 43 units of 2^-24 off."""
    import torch

    c = 1 + 838861 * 2.0**-21
    up = vsc.Upsampler(np.zeros(vsc.Upsampler.param_count(), np.float32))
    inp = torch.zeros((32, 64, 64, 3), device=cuda)
    assert up.train_step(inp, torch.full((32, 64, 64, 2), c, device=cuda), 1e-3) == 2 * c
    up.close()


@pytest.mark.gpu
def test_creation_allocates_nothing_for_training(vsc, cuda):
    """An upsampler that only infers holds its parameters, their moments and the packed
    weights, less than half a MiB; the gradient's copies (2.5 MiB) come with the first
    training step."""
    import torch

    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ups = [vsc.Upsampler() for _ in range(64)]
    held = free - torch.cuda.mem_get_info()[0]
    for up in ups:
        up.close()
    assert held <= 64 * 2**19
