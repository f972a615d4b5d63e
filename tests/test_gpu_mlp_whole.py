"""The whole-network kernels (sbx_mlp_predict, sbx_mlp_train) against the GEMM path, which the
oracle checks (tests/test_gpu_surrogate.py): ragged point counts around the 128-row tiles, one
and several networks, narrow and wide layers, batches of part of a tile to two tiles. Both
paths do the same operations on every element, so predictions agree to FP64 rounding of the
statistics. Training may differ by a BF16 rounding where two FP32 values straddle one: one
such flip among a layer's 256 inputs moves a sum by 2^-8 / 256 of itself, 1.5e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _ensemble(dims, nz, batch, seed=3):
    from softbox_b200.surrogate import MLPEnsemble
    ens = MLPEnsemble(n_nets=nz, dims=dims, batch=batch, seed=seed)
    rng = np.random.default_rng(seed)
    for b in ens.b:
        b.copy_(torch.from_numpy(0.1 * rng.standard_normal(tuple(b.shape)).astype(np.float32)))
    ens.b[-1][:, dims[-1]:] = 0
    x = rng.uniform(size=(2048, dims[0]))
    y = rng.normal(size=(2048, dims[-1]))
    ens.set_normalisation(x, y)
    return ens, x, y


@pytest.mark.parametrize("dims,nz,P", [((6, 256, 256, 256, 256, 3), 5, 1000), ((6, 256, 256, 256, 256, 3), 1, 1),
                                       ((6, 32, 3), 2, 127), ((16, 256, 64, 16), 3, 129), ((1, 96, 1), 1, 128)])
def test_predict_equals_the_gemm_path(dims, nz, P, monkeypatch):
    ens, x, _ = _ensemble(dims, nz, 256)
    whole = ens.predict(x[:P])
    assert ens.err.item() == 0
    monkeypatch.setattr(type(ens), "_net", lambda self, train: None)
    ref = ens.predict(x[:P])
    for a, b, name in zip(whole, ref, ("mean", "std", "y")):
        assert a.shape == b.shape and a.dtype == b.dtype
        assert np.allclose(a, b, rtol=1e-12, atol=1e-12), name


@pytest.mark.parametrize("dims,nz,B", [((6, 256, 256, 256, 256, 3), 5, 256), ((6, 64, 32, 3), 2, 16),
                                       ((16, 96, 16), 1, 144), ((3, 32, 256, 1), 3, 128)])
def test_train_equals_the_separate_kernels(dims, nz, B, monkeypatch):
    steps = 3
    a, x, y = _ensemble(dims, nz, B)
    b, _, _ = _ensemble(dims, nz, B)
    n = steps * B
    ha = a.fit(x[:n], y[:n], epochs=1, seed=5)
    monkeypatch.setattr(type(b), "_net", lambda self, train: None)
    hb = b.fit(x[:n], y[:n], epochs=1, seed=5)
    torch.cuda.synchronize()
    assert a.err.item() == 0 and a.step_no == b.step_no == steps
    assert abs(ha[0] - hb[0]) <= 1e-5 * abs(hb[0])
    for l in range(a.L):
        for k in ("W", "b", "mW", "mb", "vW", "vb", "dW", "db"):
            p, q = getattr(a, k)[l].double(), getattr(b, k)[l].double()
            assert (p - q).norm() <= 2e-5 * q.norm(), f"{k}[{l}]"
        assert torch.equal(a.Wb[l].view(torch.bfloat16), a.W[l].to(torch.bfloat16))
        assert torch.equal(a.WbT[l], a.Wb[l].transpose(1, 2))
        assert a.W[l][:, dims[l + 1]:].abs().sum().item() == 0        # the padding stays zero
    assert a.W[0][:, :, dims[0]:].abs().sum().item() == 0


def test_one_step_on_given_batches_equals_fit():
    a, x, y = _ensemble((6, 64, 64, 3), 2, 64)
    b, _, _ = _ensemble((6, 64, 64, 3), 2, 64)
    t = lambda v, m, s: torch.tensor((v - m) / s, dtype=torch.float32, device="cuda")  # noqa: E731
    X, Y = t(x[:64], a.x_mean, a.x_std), t(y[:64], a.y_mean, a.y_std)
    a.train_step(X.expand(2, 64, 6).contiguous(), Y.expand(2, 64, 3).contiguous())
    idx = torch.arange(64, device="cuda").repeat(2, 1)
    b._train_whole(b._net(True), X, Y, idx, 1)
    torch.cuda.synchronize()
    for l in range(a.L):
        assert torch.equal(a.W[l], b.W[l]) and torch.equal(a.b[l], b.b[l])


@pytest.mark.parametrize("dims,nz,whole", [((6, 32, 3), 64, True), ((6, 32, 3), 148, True), ((6, 32, 3), 300, False),
                                           ((6, 256, 256, 3), 64, True), ((6, 256, 256, 3), 148, False)])
def test_many_networks_train(dims, nz, whole, monkeypatch):
    # past the resident blocks, or with too much work for a network's one block, the separate kernels
    a, x, y = _ensemble(dims, nz, 16)
    b, _, _ = _ensemble(dims, nz, 16)
    assert (a._trains_whole() is not None) == whole
    ha = a.fit(x[:32], y[:32], epochs=1, seed=5)
    monkeypatch.setattr(type(b), "_net", lambda self, train: None)
    hb = b.fit(x[:32], y[:32], epochs=1, seed=5)
    assert abs(ha[0] - hb[0]) <= 1e-5 * abs(hb[0])
    for l in range(a.L):
        p, q = a.W[l].double(), b.W[l].double()
        assert (p - q).norm() <= 2e-5 * q.norm(), l


@pytest.mark.parametrize("whole", [True, False])
def test_a_failed_wait_is_raised_once(whole, monkeypatch):
    # a kernel's error word (set from the host here) ends the call that finds it with an error,
    # and neither stops that call's kernels nor the next call
    from softbox_b200.runtime import SbxError
    a, x, y = _ensemble((6, 64, 64, 3), 2, 64)
    b, _, _ = _ensemble((6, 64, 64, 3), 2, 64)
    if not whole:
        monkeypatch.setattr(type(a), "_net", lambda self, train: None)
    a.err.fill_(1)
    with pytest.raises(SbxError, match="wait ran out"):
        a.fit(x[:1024], y[:1024], epochs=1, seed=5)
    b.fit(x[:1024], y[:1024], epochs=1, seed=5)
    ha, hb = (e.fit(x[:1024], y[:1024], epochs=2, seed=6) for e in (a, b))
    assert np.allclose(ha, hb, rtol=1e-5)               # (the loss is summed in no order)
    for l in range(a.L):
        assert torch.equal(a.W[l], b.W[l]) and torch.equal(a.b[l], b.b[l])
    a.err.fill_(1)
    with pytest.raises(SbxError, match="wait ran out"):
        a.predict(x[:300])
    for p, q in zip(a.predict(x[:300]), b.predict(x[:300])):
        assert np.array_equal(p, q)


@pytest.mark.parametrize("name", ["W", "mW", "vW", "dW", "WbT", "A", "AT", "G", "GT", "Z", "X0T", "bar", "Wb"])
def test_unaligned_training_arrays_are_refused(name):
    from softbox_b200 import abi_types as T
    a, x, y = _ensemble((6, 32, 32, 3), 2, 16)
    net, s = a._net(True), T.MlpTrainState()
    for l in range(a.L):
        for k in ("W", "mW", "vW", "mb", "vb", "dW", "db", "WbT", "A", "AT", "G", "GT", "Z"):
            getattr(s, k)[l] = getattr(a, k)[l].data_ptr()
    s.X0T, s.loss, s.bar, s.err = (v.data_ptr() for v in (a.X0T, a.loss, a.bar, a.err))
    if name in ("X0T", "bar"):
        setattr(s, name, getattr(s, name) + 4)
    else:
        at = net.Wb if name == "Wb" else getattr(s, name)
        at[1] += 4
    X, Y = (torch.zeros(64, n, device="cuda") for n in (6, 3))
    st = a._ctx().raw("sbx_mlp_train", net, s, 16, X, Y, None, 0, 1, 1, 1e-3, 0.9, 0.999, 1e-8)
    assert st == -1                                    # SBX_EINVAL, before anything is launched


def test_large_predictions_are_arrays_of_their_own():
    # a mean that is kept does not keep every network's outputs
    a, x, _ = _ensemble((6, 32, 16), 3, 16)
    mean, std, y = a.predict(x)
    assert mean.shape == std.shape == (2048, 16) and y.shape == (3, 2048, 16)
    for v in (mean, std, y):
        assert v.flags.owndata and v.flags.writeable and v.base is None
