"""The training step's reductions, copies and alignment at ragged sizes. Gradients:
the bar of test_gpu_mlp.py (1e-2 relative per tensor against the oracle, which
rounds to BF16 at the same places). Alignment: the sums are taken in double, so
the rotation, rounded to f32, agrees with numpy's to 1e-5."""
import numpy as np
import pytest

import mlp_oracle as M

pytestmark = pytest.mark.gpu


# rows around the reductions' 64-row stages and 8-row groups, outputs around their 8
@pytest.mark.parametrize("n", [1, 7, 63, 64, 65, 129, 4999])
@pytest.mark.parametrize("i,h,o", [(16, 8, 1), (24, 136, 8), (72, 264, 9), (128, 512, 16)])
def test_gradients_at_ragged_sizes(ctx, i, h, o, n):
    net = ctx.mlp(i, h, o, seed=2)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, i)).astype(np.float32) / np.sqrt(i)
    t = rng.standard_normal((n, o)).astype(np.float32)
    loss, grad = net.gradients(x, t)
    want_loss, want = M.loss_and_gradients(M.unpack(net.get_params(), i, h, o), x, t)
    assert loss == pytest.approx(want_loss, rel=1e-3)
    got = net.unpack(grad)
    for name, w in want.items():
        rel = np.linalg.norm(got[name] - w) / max(np.linalg.norm(w), 1e-30)
        assert rel <= 1e-2, (name, rel)


@pytest.mark.parametrize("d", [1, 3, 8, 16])
def test_fit_on_uneven_instances(ctx, d):
    """Instances of uneven size, one smaller than a batch: finite, and the same bits
    twice; points off a 16-byte boundary are refused."""
    torch = pytest.importorskip("torch")
    import evoc_gb300 as E
    i, h, ns = 40, 24, [3000, 50, 1025]
    g = torch.Generator(device="cuda").manual_seed(d)
    pts = [(torch.randn(n, i, generator=g, device="cuda") / i ** 0.5).to(torch.bfloat16)
           for n in ns]
    lay = [torch.randn(n, d, generator=g, device="cuda") for n in ns]
    p = E.MlpTrainParams(steps=9, batch=256, align_every=4, align_rows=1000, seed=3)
    torch.cuda.synchronize()

    def fit(ptrs):
        net = ctx.mlp(i, h, d, seed=1)
        hist = net.fit_device(ptrs, [t.data_ptr() for t in lay], ns, p)
        return hist, net.get_params()

    ptrs = [x.data_ptr() for x in pts]
    (h0, p0), (h1, p1) = fit(ptrs), fit(ptrs)
    assert np.isfinite(h0).all()
    assert np.array_equal(h0.view(np.uint32), h1.view(np.uint32))
    assert np.array_equal(p0.view(np.uint32), p1.view(np.uint32))
    with pytest.raises(E.EvocError):
        fit([ptrs[0] + 4] + ptrs[1:])


def test_first_loss_is_against_the_aligned_layout(ctx):
    """A step's loss equals the mean square of prediction minus the layout as numpy
    aligns it (one instance, all of its rows sampled by draws of the batch)."""
    torch = pytest.importorskip("torch")
    import evoc_gb300 as E
    i, h, d, n = 32, 64, 8, 400
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.standard_normal((n, i)).astype(np.float32) / 6).cuda().to(torch.bfloat16)
    net = ctx.mlp(i, h, d, seed=5)
    y = net.predict(x.float().cpu().numpy())
    q, _ = np.linalg.qr(rng.standard_normal((d, d)))
    lay = ((y - y.mean(0)) @ q.T + 3.0).astype(np.float32)  # a rotated, shifted prediction
    t = torch.from_numpy(lay).cuda()
    torch.cuda.synchronize()
    p = E.MlpTrainParams(steps=1, batch=4096, align_rows=1 << 16, lr=0.0, lr_end=0.0)
    hist = net.fit_device([x.data_ptr()], [t.data_ptr()], [n], p)
    # alignment undoes the rotation, up to the sample's own (drawn with replacement) means and
    # f32: what is left of the layout's variance is below 1e-9 of it
    assert hist[0] <= 1e-9 * float(lay.var())
