"""GPU checks of the conflict predictor's hand-written kernels against the float64 oracle
(oracle/mlp_oracle.py): forward probabilities, the gradient of the mean binary cross-entropy,
the Adam update, and that training learns a separable labelling.

Tolerances (fp32 accumulation of bf16 weights against float64 on the same bf16 weights):
probabilities 2e-5 absolute for 0/1 features (2e-4 for dense features, where a layer-1
activation may round to the neighbouring bf16 value); gradients 1e-4 relative to the
gradient's max-norm, per entry."""
import numpy as np
import pytest

import csmv_gb300 as cg
import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _dev(torch, a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.cuda()


def _features(rng, n, dense=False):
    if dense:  # arbitrary bf16 values exercise the datapath beyond 0/1 indicators
        x = mo.bf16_round(rng.normal(0, 1, (n, mo.IN)).astype(np.float32))
    else:
        x = (rng.random((n, mo.IN)) < 0.25).astype(np.float32)
    return x, mo.bf16_bits(x).view(np.int16)


@pytest.mark.parametrize("n,dense", [(1, False), (63, True), (1000, False), (70000, True)])
def test_forward_and_gradient_match_oracle(n, dense):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    x, xb = _features(rng, n, dense)
    y = (rng.random(n) < 0.4).astype(np.float32)
    with cg.Mlp(seed=7) as m:
        params = m.params()
        params[mo.OFF_B1:mo.OFF_W2] = rng.normal(0, 0.1, mo.HID)  # nonzero biases too
        params[mo.OFF_B3] = 0.3
        m.set_params(params)
        dx, dy = _dev(torch, xb), _dev(torch, y)
        dp = torch.zeros(n, dtype=torch.float32, device="cuda")
        m.forward(n, dx.data_ptr(), dp.data_ptr())
        p_gpu = dp.cpu().numpy()
        loss = m.grad(n, dx.data_ptr(), dy.data_ptr())
        g_gpu = m.grads().astype(np.float64)
    p_ref, _ = mo.forward(params, x)
    # binary features (the scheduler's) give exactly representable layer-1 sums; with dense
    # inputs an fp32 sum can land on the other side of a bf16 rounding boundary than the float64
    # one, moving one activation by one bf16 step (2^-8 relative) and p by up to ~1e-4
    np.testing.assert_allclose(p_gpu, p_ref, rtol=0, atol=2e-4 if dense else 2e-5)
    if dense:
        assert np.mean(np.abs(p_gpu - p_ref) > 2e-5) < 1e-3
    loss_ref, g_ref = mo.loss_and_grads(params, x, y)
    assert abs(loss - loss_ref) < 1e-4 * max(1.0, abs(loss_ref))
    scale = np.abs(g_ref).max()
    np.testing.assert_allclose(g_gpu, g_ref, rtol=0, atol=1e-4 * scale)


def test_adam_step_matches_oracle():
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    x, xb = _features(rng, 512)
    y = (rng.random(512) < 0.5).astype(np.float32)
    with cg.Mlp(seed=9) as m:
        p0 = m.params().astype(np.float64)
        dx, dy = _dev(torch, xb), _dev(torch, y)
        mm = np.zeros_like(p0)
        vv = np.zeros_like(p0)
        for step in (1, 2):
            m.grad(512, dx.data_ptr(), dy.data_ptr())
            g = m.grads().astype(np.float64)
            m.adam_step(1e-3)
            p0, mm, vv = mo.adam(p0, g, mm, vv, step, 1e-3)
            np.testing.assert_allclose(m.params(), p0, rtol=0, atol=1e-6)
            assert not m.grads().any()  # the step clears the accumulator


def test_training_learns_a_separable_labelling():
    """y = x[3] or (x[10] and x[40]): a few hundred Adam steps drive the loss down and the
    predictions to > 97 % accuracy on fresh samples."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)

    def batch(n):
        x, xb = _features(rng, n)
        y = ((x[:, 3] > 0) | ((x[:, 10] > 0) & (x[:, 40] > 0))).astype(np.float32)
        return x, xb, y

    with cg.Mlp(seed=1) as m:
        first = None
        for it in range(300):
            _, xb, y = batch(4096)
            dx, dy = _dev(torch, xb), _dev(torch, y)
            loss = m.grad(4096, dx.data_ptr(), dy.data_ptr())
            first = loss if first is None else first
            m.adam_step(3e-3)
        _, xb, y = batch(20000)
        dx = _dev(torch, xb)
        dp = torch.zeros(20000, dtype=torch.float32, device="cuda")
        m.forward(20000, dx.data_ptr(), dp.data_ptr())
        acc = float(((dp.cpu().numpy() > 0.5) == (y > 0.5)).mean())
    assert loss < 0.25 * first and acc > 0.97, (first, loss, acc)


@pytest.mark.parametrize("n", [31, 127, 128, 129, 152 * 128, 152 * 128 + 1, 2 * 152 * 128 + 77,
                               5 * 152 * 128 + 130])
def test_forward_at_tile_and_grid_edges(n):
    """Inference over partial and whole tiles of 128, one to several tiles a group of the grid's
    CTAs, with biases that do not fit one bf16: probabilities match the float64 oracle, and
    nothing beyond n is written. With such biases a layer-1 sum can round to the neighbouring
    bf16 value, as for dense features above: 2e-4 absolute, 2e-5 for all but 1e-3 of the samples."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    x, xb = _features(rng, n)
    with cg.Mlp(seed=11) as m:
        params = m.params()
        params[mo.OFF_B1:mo.OFF_W2] = rng.normal(0, 0.4, mo.HID)
        params[mo.OFF_B2:mo.OFF_W3] = rng.normal(0, 0.4, mo.HID)
        params[mo.OFF_B3] = -0.2
        m.set_params(params)
        dx, dp = _dev(torch, xb), torch.full((n + 256,), 7.0, device="cuda")
        m.forward(n, dx.data_ptr(), dp.data_ptr())
        p = dp.cpu().numpy()
    off = np.abs(p[:n] - mo.forward(params, x)[0])
    assert off.max() <= 2e-4 and np.mean(off > 2e-5) < 1e-3
    assert (p[n:] == 7.0).all()


def test_forward_after_training_uses_the_new_weights():
    """The inference operands follow Adam's updates of weights and biases."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(2)
    x, xb = _features(rng, 700)
    y = (x[:, 5] > 0).astype(np.float32)
    with cg.Mlp(seed=3) as m:
        dx, dy = _dev(torch, xb), _dev(torch, y)
        dp = torch.zeros(700, device="cuda")
        for _ in range(5):
            m.grad(700, dx.data_ptr(), dy.data_ptr())
            m.adam_step(1e-2)
        m.forward(700, dx.data_ptr(), dp.data_ptr())
        np.testing.assert_allclose(dp.cpu().numpy(), mo.forward(m.params(), x)[0], rtol=0, atol=2e-5)


@pytest.mark.parametrize("n,offset", [(15, 0), (64, 1), (65, 3), (152 * 64, 0), (152 * 64 + 1, 8),
                                      (3 * 152 * 64 + 113, 5)])
def test_gradient_at_tile_and_grid_edges(n, offset):
    """The gradient over partial and whole tiles of 64, one to several tiles a CTA, with the
    features at any element of an allocation (offset elements of 2 bytes): the bounds above, and
    the second call adds to the first one's."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    x, xb = _features(rng, n)
    y = (rng.random(n) < 0.4).astype(np.float32)
    with cg.Mlp(seed=13) as m:
        params = m.params()
        whole = torch.full((offset + n * mo.IN,), 0x7FC0, dtype=torch.int16, device="cuda")
        whole[offset:] = _dev(torch, xb).flatten()
        dy = _dev(torch, y)
        losses = [m.grad(n, whole.data_ptr() + 2 * offset, dy.data_ptr()) for _ in range(2)]
        g = m.grads().astype(np.float64) / 2
    loss_ref, g_ref = mo.loss_and_grads(params, x, y)
    assert max(abs(l - loss_ref) for l in losses) < 1e-4 * max(1.0, abs(loss_ref))
    np.testing.assert_allclose(g, g_ref, rtol=0, atol=1e-4 * np.abs(g_ref).max())


@pytest.mark.parametrize("offset", [1, 4, 7, 8, 15])
def test_forward_refuses_features_off_a_16_byte_boundary(offset):
    """Inference copies its features in 16-byte pieces: a pointer between two of them is refused on
    the host (the gradient takes it), one on a boundary inside an allocation is not."""
    torch = pytest.importorskip("torch")
    n = 130
    x, xb = _features(np.random.default_rng(offset), n)
    with cg.Mlp(seed=5) as m:
        whole = torch.zeros(offset + n * mo.IN, dtype=torch.int16, device="cuda")
        whole[offset:] = _dev(torch, xb).flatten()
        dp = torch.full((n,), 7.0, device="cuda")
        if offset % 8:
            with pytest.raises(cg.CsmvError) as e:
                m.forward(n, whole.data_ptr() + 2 * offset, dp.data_ptr())
            assert e.value.status == 1 and (dp == 7.0).all()
        else:
            m.forward(n, whole.data_ptr() + 2 * offset, dp.data_ptr())
            np.testing.assert_allclose(dp.cpu().numpy(), mo.forward(m.params(), x)[0], rtol=0, atol=2e-5)
