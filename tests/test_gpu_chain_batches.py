"""Batches of chains at the edges of the noise, E-step and pooling launches (more chains than CTAs,
chain counts that are no multiple of four, images): chain c is the single-chain run with chain index
c, and the pooled moments are the chains' combined."""
import numpy as np
import pytest

from test_gpu_parity import make_case, new_reg

pytestmark = pytest.mark.gpu


def image_reg(core, shape):
    from binder_b200 import phantoms
    from binder_b200.utils import initialize_fourier_domain_smoothing as ifs
    p = phantoms.make_pair(shape, 3, bins=6, rms=1.0, spacing=4.0)
    g = np.ascontiguousarray(phantoms.identity_positions(shape).astype(np.float32))
    reg = core.Registration(g, 1, g, g, *shape, 1, *shape, 1, 3, float(np.count_nonzero(p.u)))
    D = ifs(shape, True, 2, 2).astype(np.float32)
    reg.setNonLinearTransformation(1e-2, 1e-2, 1e-2, 1, 1, 1, 1, 1, 1, D)
    reg.setMILikelihood(2.0, np.full((6, 6), 1 / 6, np.float32), 6, 6, 1, p.v, p.u)
    return reg


@pytest.mark.parametrize("shape,chains", [((9, 7, 20), 1), ((9, 7, 20), 5), ((5, 4, 6), 67),
                                          ((40, 41, 42), 3), ((20, 19), 6)])
def test_chains(core, monkeypatch, shape, chains):
    # one chain of a small image would take the fused FP32 M-step, a batch the tensor-core passes
    monkeypatch.setenv("BINDER_B200_FUSED2D", "0")

    def make():
        if len(shape) == 2:
            return image_reg(core, shape)
        c = make_case(shape=shape, seed=8)
        return new_reg(core, c)

    Nb, Ns = 1, 4
    means, covs, pm, pc = make().sampler_chains(77, chains, Nb, Ns, 0, 1, 1, 1, 1)
    for ch in {0, chains // 2, chains - 1}:
        one = make()
        one.set_chain(ch)
        m, v = one.sampler(77, Nb, Ns, 0, 1, 1, 1, 1)
        # the same draws and the same arithmetic (gamma is not sampled, so no cost sum feeds back)
        np.testing.assert_allclose(means[ch], m, rtol=0, atol=1e-5)
        np.testing.assert_allclose(covs[ch], v, rtol=0, atol=1e-4)
    np.testing.assert_allclose(pm, means.mean(0), rtol=0, atol=1e-9)
    dev = means - means.mean(0)
    m2 = (covs * (Ns - 1)).sum(0) + Ns * np.einsum("c...i,c...j->...ij", dev, dev)
    np.testing.assert_allclose(pc, m2 / (chains * Ns - 1), rtol=1e-9, atol=1e-12)
