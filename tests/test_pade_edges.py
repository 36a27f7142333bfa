"""The Pade continuation where its shortened division chain hands over to the general one: zeros,
constant and purely imaginary rows, values near the ends of the exponent range, NaN, few and many
parameters.  Against the oracle (the reference's arithmetic), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(om, nfreq, seed):
    rng = np.random.default_rng(seed)
    smooth = sum(a / (1j * om - e) for a, e in zip(rng.uniform(0.01, 0.1, 40), rng.uniform(-2.0, 2.0, 40)))
    rows = {"smooth": smooth, "zero": np.zeros(nfreq, complex), "constant": np.full(nfreq, 0.3 - 0.1j),
            "imaginary": 1j * smooth.imag, "real": smooth.real + 0j, "tiny": smooth * 1e-30, "huge": smooth * 1e30,
            "equal parts": smooth.real * (1 + 1j), "some zeros": np.where(np.arange(nfreq) % 5 == 0, 0, smooth),
            "noise": rng.standard_normal(nfreq) + 1j * rng.standard_normal(nfreq)}
    nan = smooth.copy()
    nan[nfreq // 2] = np.nan
    rows["nan"] = nan
    return rows


@pytest.mark.parametrize("nfreq,npade", [(1, 1), (2, 2), (3, 16), (40, 2), (40, 3), (64, 33), (200, 128)])
def test_sweep_and_qp_bit_exact(oracle_lib, cfg1_input, nfreq, npade):
    from minigw_b200 import B200Backend

    om, _ = oracle_lib.grid(nfreq)
    rows = _rows(om, nfreq, 10 * nfreq + npade)
    nmo = cfg1_input.mo_energy.shape[0]
    sigma = np.zeros((nmo, nfreq), dtype=np.complex128)
    for i, r in enumerate(rows.values()):
        sigma[i] = r
    states = list(range(len(rows)))
    with B200Backend(0) as be:
        be.load_system(cfg1_input)
        with np.errstate(all="ignore"):
            for r in rows.values():
                dev = be.pade_sweep(om, r, npade, npts=700, fermi=0.1, x_start=-3.0, interval=0.01)
                np.testing.assert_array_equal(dev, oracle_lib.ec_sweep(om, r, npade, 700, 0.1, -3.0, 0.01))
            sx = be.sigma_x_diag()
            qp = be.qp(om, sigma, npade, states)
            np.testing.assert_array_equal(qp[states], oracle_lib.qp(cfg1_input, sx, om, sigma, states, npade)[states])


def test_sweep_refuses_too_many_parameters_before_any_device_work():
    """A sweep of more points than any device holds and more parameters than the kernels take is refused for the
    parameters: nothing was allocated, and no copy of the caller's arrays begun, when the call returns."""
    from minigw_b200 import B200Backend
    from minigw_b200._lib import STATUS, dptr, lib

    om, row, out = np.linspace(0.1, 1.0, 200), np.zeros(200, complex), np.zeros(3)
    with B200Backend(0) as be:
        rc = lib.gwb200_pade_sweep(be._h, dptr(om), 200, dptr(row), 129, 10**12, 0.0, -6.5, 0.1, dptr(out))
    assert STATUS[rc] == "GWB200_BAD_SHAPE" and b"Pade limit" in lib.gwb200_last_error()


def test_sweep_of_a_capped_handle_keeps_no_memory():
    import torch

    from minigw_b200 import B200Backend

    om = np.linspace(0.1, 1.0, 40)
    row = 0.1 / (1j * om + 0.5)
    npts = 4_000_000  # 96 MB of points
    torch.cuda.mem_get_info(0)
    with B200Backend(0) as be:
        be.set_memory_limit(1 << 27)
        be.pade_sweep(om, row, 8, npts=1000)
        before = torch.cuda.mem_get_info(0)[0]
        be.pade_sweep(om, row, 8, npts=npts)
        assert before - torch.cuda.mem_get_info(0)[0] < 16 << 20


def test_a_failed_allocation_does_not_fail_the_next_call():
    from minigw_b200 import B200Backend
    from minigw_b200._lib import STATUS, dptr, lib

    om, out = np.linspace(0.1, 1.0, 40), np.zeros(3)
    row = 0.1 / (1j * om + 0.5)
    with B200Backend(0) as be:
        rc = lib.gwb200_pade_sweep(be._h, dptr(om), 40, dptr(row), 8, 10**12, 0.0, -6.5, 0.1, dptr(out))
        assert STATUS[rc] == "GWB200_OOM"
        assert np.isfinite(be.pade_sweep(om, row, 8, npts=100)).all()
