"""Sigma_c between states at the state counts where the 8-state tiles of its Gram kernel begin and end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 7, 8, 9, 16, 17, 24, 33, 41, 50, 57, 64])
def test_matrix_against_numpy(ns):
    from minigw_b200 import B200Backend, generate_transformed_legendre_grid
    from test_panel import _system

    nmo = 67
    sl = _system(nmo - 1, 40, ns, 500 + ns)
    om, w = generate_transformed_legendre_grid(6)
    with B200Backend(0) as be:
        be.load_slices(sl)
        got, _ = be.sigma_c_matrix(om, w, sl.states)
    delta = sl.mo_energy[1:] - sl.mo_energy[0]
    ref = np.zeros((ns, ns, 6), dtype=complex)
    for f, wf in enumerate(om):
        d = np.sqrt(4.0 * delta / (wf * wf + delta * delta))
        low = np.linalg.cholesky(np.eye(len(d)) + d[:, None] * sl.vph * d[None, :])
        y = np.linalg.solve(low, (sl.panel * d).T).reshape(len(d), ns, nmo)
        q = -np.einsum("isk,itk->stk", y, y)
        a = 1j * om[:, None] + sl.fermi_energy - sl.mo_energy[None, :]
        ref -= np.einsum("nk,stk->stn", w[f] * a / (a * a + wf * wf), q) / np.pi
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()  # FP64 sums, condition <= ~1e3
    np.testing.assert_array_equal(got, got.transpose(1, 0, 2))
