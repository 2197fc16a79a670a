"""GPU kernels at the edges of their tiles, against numpy in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


# one pair, tiles of 2 x 2 with an odd last band, one and several tiles per
# thread, several groups; spheres of one and of many splits.  FP32: sums of at
# most 2,048 products, each rounding 6e-8 of a running sum, give 3e-6 of
# |a||b| when they add like a random walk
@pytest.mark.parametrize("precision,tol", [(0, 1e-13), (1, 1e-5)])
@pytest.mark.parametrize("nb,buf,L", [(1, 0, 6.0), (5, 0, 6.0), (12, 4, 6.0), (23, 4, 9.0), (33, 0, 9.0), (64, 4, 12.0),
                                      (128, 0, 12.0)])
def test_overlap_pairs(nb, buf, L, precision, tol):
    import derek_gb300 as dg
    rng = np.random.default_rng(nb)
    spec = dg.SystemSpec(np.eye(3) * L, 6.0, [[0, 0, 0], [0.2, 0.1, -0.3]], nb, 1.0)
    with dg.Handle(spec, precision=precision, buffer_bands=buf, use_tensor_cores=0) as h:
        for k in range(2):
            n = h.npw(0, k)
            psi = rng.standard_normal((nb, n)) + 1j * rng.standard_normal((nb, n))
            h.set_wfn(psi, 0, k)
            got = h.wave_dot(0, k)
            if precision:
                psi = psi.astype(np.complex64).astype(np.complex128)
            ref = psi.conj() @ psi.T
            assert rel_err(got, ref) < tol
            assert np.array_equal(got, got.conj().T)
