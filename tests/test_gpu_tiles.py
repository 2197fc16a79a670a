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


# every radix 2..16 of the shared-memory lines, coprime splits (26 = 13 x 2,
# 77 = 11 x 7) and Cooley-Tukey ones (25, 32, 49), a prime length, a length
# below a warp, unequal axes
LINES = [(13, 26, 25), (32, 49, 30), (77, 12, 14), (33, 70, 39), (16, 11, 128), (52, 64, 45), (20, 60, 27)]


@pytest.mark.parametrize("precision,tol", [(0, 1e-11), (1, 2e-5)])
@pytest.mark.parametrize("n", LINES)
def test_shared_memory_lines(oracle, n, precision, tol):
    """H.psi and the density on grids that only the shared-memory lines serve."""
    import derek_gb300 as dg
    from test_gpu_primitives import make_pair
    s, spec = make_pair(oracle, L=6.0, ecut=2.9, nb=3, n_fine=n, seed=n[0])
    kb = oracle.KBasis(s, 0)
    rng = np.random.default_rng(n[1])
    psi = rng.standard_normal((s.nbands, kb.npw)) + 1j * rng.standard_normal((s.nbands, kb.npw))
    v = s.vext + 0.3 * rng.standard_normal(s.nr)
    occ = np.array([[2.0, 0.0, 0.7]])
    with dg.Handle(spec, precision=precision) as h:
        h.set_vloc(v)
        h.set_wfn(psi)
        got, rho = h.pot_apply_wfn(), h.density_calculate(occ)
    assert rel_err(got, oracle.apply_h(s, kb, v, psi)) < tol
    assert rel_err(rho, oracle.band_density(s, kb, psi, occ[0])) < tol


@pytest.mark.parametrize("rows", ["tight", "compact", "all"])
@pytest.mark.parametrize("n", [24, 27, 32, 36, 48, 54, 64, 72])
def test_spinor_register_planes(oracle, n, rows):
    """FP32 spinor H.psi at every length with register lines."""
    import derek_gb300 as dg
    from test_gpu_primitives import reg_plane_pair
    s, spec = reg_plane_pair(oracle, n, rows, ((0.1, 0.2, -0.3),), 3, seed=n)
    spec.nspinor = 2
    spec.nelec = 2.0
    kb = oracle.KBasis(s, 0)
    rng = np.random.default_rng(n + 1)
    psi = rng.standard_normal((2, s.nbands, kb.npw)) + 1j * rng.standard_normal((2, s.nbands, kb.npw))
    nc = rng.standard_normal((s.nr, 2, 2)) + 1j * rng.standard_normal((s.nr, 2, 2))
    with dg.Handle(spec, precision=1) as h:
        h.set_nc_pot(nc)
        h.set_wfn(psi)
        got = h.pot_apply_wfn()
    assert rel_err(got, oracle.apply_h_spinor(s, kb, nc, psi)) < 2e-5


# the largest planes that two blocks of an SM hold (192 threads) and the next
# smooth length (512 threads)
@pytest.mark.parametrize("n,precision,tol", [(56, 0, 1e-11), (60, 0, 1e-11), (84, 1, 2e-5), (88, 1, 2e-5)])
def test_spinor_block_sizes(oracle, n, precision, tol):
    import derek_gb300 as dg
    from test_gpu_primitives import make_pair
    s, spec = make_pair(oracle, L=6.0, ecut=2.9, nb=3, n_fine=(8, n, n), seed=n)
    spec.nspinor = 2
    spec.nelec = 2.0
    kb = oracle.KBasis(s, 0)
    rng = np.random.default_rng(n + 1)
    psi = rng.standard_normal((2, s.nbands, kb.npw)) + 1j * rng.standard_normal((2, s.nbands, kb.npw))
    nc = rng.standard_normal((s.nr, 2, 2)) + 1j * rng.standard_normal((s.nr, 2, 2))
    occ = np.array([[1.0, 0.0, 0.7]])
    with dg.Handle(spec, precision=precision) as h:
        h.set_nc_pot(nc)
        h.set_wfn(psi)
        got = h.pot_apply_wfn()
        rho, mag = h.density_spinor(occ)
    n_ref, m_ref = oracle.spinor_density(s, kb, psi, occ[0])
    assert rel_err(got, oracle.apply_h_spinor(s, kb, nc, psi)) < tol
    assert rel_err(rho, n_ref) < tol and rel_err(mag, m_ref) < tol


# every count of bands per thread of the rotations, odd ones among them, and a
# last G tile that is partly filled: band energies (the lower half, well inside
# the subspace) against the dense Hamiltonian, bounds as tests/test_gpu_nscf.py
@pytest.mark.parametrize("precision,eig_tol,tol", [(0, 1e-10, 1e-8), (1, 5e-6, 2e-5)])
@pytest.mark.parametrize("nb", [1, 7, 8, 9, 17, 25, 33, 49, 64, 65, 97, 124])
def test_rotations_at_every_band_count(oracle, nb, precision, eig_tol, tol):
    import derek_gb300 as dg
    from test_gpu_nscf import dense_eigenvalues
    from test_gpu_primitives import make_pair
    s, spec = make_pair(oracle, L=9.0, ecut=5.0, nb=nb, nelec=1.0, seed=nb)
    nconv = (nb + 1) // 2
    with dg.Handle(spec, precision=precision, buffer_bands=4, use_tensor_cores=0, init_vectors=1) as h:
        h.set_vloc(s.vext)
        (eig,), _ = h.nscf(max_iter=300, eig_tol=eig_tol, nconv=nconv)
    ref = dense_eigenvalues(oracle, s, 0, s.vext, nconv)
    assert np.max(np.abs(eig[0, :nconv] - ref)) < tol


# Jacobi solves on one CTA and on clusters of 2, 4 and 8, one element per lane and
# one block per thread, odd counts, subspaces in shared memory and in global
# scratch: the Ritz vectors diagonalise the projected Hamiltonian
@pytest.mark.parametrize("nb,nk", [(2, 1), (5, 3), (16, 1), (23, 2), (23, 40), (44, 1), (44, 70), (84, 1), (85, 20),
                                   (115, 2), (128, 1)])
def test_jacobi_solves(oracle, nb, nk):
    import derek_gb300 as dg
    from test_gpu_primitives import make_pair
    kpts = [(0.1 + 0.005 * i, 0.2, -0.3 + 0.004 * i) for i in range(nk)]
    s, spec = make_pair(oracle, L=8.0, ecut=4.0, nb=nb, nelec=1.0, kpts=kpts, seed=nb)
    with dg.Handle(spec, precision=0, buffer_bands=0, init_vectors=1, use_tensor_cores=0) as h:
        h.set_vloc(s.vext)
        try:
            h.nscf(max_iter=2, eig_tol=1e-12)
        except dg.DerekError:
            pass   # two iterations do not converge; the Ritz pairs are exact in their subspace
        eig = h.eigenvalues()
        for k in sorted({0, nk - 1}):
            psi = h.get_wfn(0, k)
            hpsi = h.pot_apply_wfn(0, k)
            hs = psi.conj() @ hpsi.T
            # Ritz vectors diagonalise H: rounding times ||H|| ~ 20 Ha
            assert np.max(np.abs(hs - np.diag(eig[k]))) < 1e-10
            assert np.all(np.diff(eig[k]) >= 0)


# half spectra of real grids: odd and even axes (an odd count of rows leaves
# one row without a partner), Nyquist planes of a sheared cell, several tiles.
# The Hartree potential and E_H of a density against full complex transforms
@pytest.mark.parametrize("n", [(11, 13, 9), (16, 12, 20), (27, 32, 25), (36, 33, 40)])
@pytest.mark.parametrize("kerker", [0.0, 0.8])
def test_hartree_half_spectra(oracle, n, kerker):
    import derek_gb300 as dg
    cell = np.array([[6.0, 0.9, 0.3], [0.0, 6.5, -0.8], [0.2, 0.0, 5.5]])
    wells = np.array([[0.3, 0.4, 0.5, 1.5, 1.2]])
    spec = dg.SystemSpec(cell, 1.1, [[0, 0, 0]], 4, 2.0, kT=0.05, wells=wells, n_fine=n)
    nr = int(np.prod(n))
    with dg.Handle(spec, kerker_q0=kerker, mix_alpha=0.5, first_passes=1) as h:
        rng = np.random.default_rng(nr)
        rho0 = np.abs(1.0 + 0.5 * rng.standard_normal(nr)) * 2.0 / abs(np.linalg.det(cell))
        h.set_start_density(rho0)
        rep = h.scf_iterate()[0]
        rho1, v1, vext = h.density(), h.get_vloc(), h.get_vext()
    inv = 2 * np.pi * np.linalg.inv(cell).T
    ax = [np.where(np.arange(k) < k - k // 2, np.arange(k), np.arange(k) - k) for k in n]
    g2 = ((np.stack(np.meshgrid(*ax, indexing="ij"), -1) @ inv.T) ** 2).sum(-1)
    ig2 = np.divide(1.0, g2, out=np.zeros_like(g2), where=g2 > 0)

    def conv(f, kernel):
        return np.fft.ifftn(np.fft.fftn(f.reshape(n)) * kernel).real.ravel()

    vol = abs(np.linalg.det(cell))
    eh = 2 * np.pi * vol * np.sum(np.abs(np.fft.fftn(rho1.reshape(n)) / nr) ** 2 * ig2)
    assert abs(rep["e_hartree"] - eh) < 1e-11 * abs(eh)
    # the next input density (linear mixing, one stored pair) and its potential
    res = rho1 - rho0
    rho_in = rho0 + (conv(res, 0.5 * g2 / (g2 + kerker ** 2)) if kerker > 0 else 0.5 * res)
    vh = conv(rho_in, 4 * np.pi * ig2)
    vxc = oracle.lda_exc_vxc(rho_in)[1]
    assert rel_err(v1, vext + vh + vxc) < 1e-11
