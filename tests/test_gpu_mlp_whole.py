"""The whole-network prediction kernel (sbx_mlp_predict) against the GEMM path, which the
oracle checks (tests/test_gpu_surrogate.py): ragged point counts around the 128-row tiles, one
and several networks, narrow and wide layers. Both paths do the same operations on every
element, so predictions agree to FP64 rounding of the statistics."""
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
