"""The panel step of the plain form (diagonal block with its inverse, rows below) at the sizes where
its tiles begin and end: 64- and 128-wide blocks, 16-wide panels, 32-row tiles, and the pivot it reports."""
import numpy as np
import pytest

from minigw_b200.gw_input import GwSlices

pytestmark = pytest.mark.gpu


def _system(n, rank, nstates, seed):
    """nocc = 1, so n = nmo - 1: V_ph = F F^T of the given rank, random right-hand sides."""
    rng = np.random.default_rng(seed)
    nmo = n + 1
    mo = np.concatenate([[-0.6], np.sort(rng.uniform(0.05, 3.0, n))])
    f = rng.standard_normal((n, rank)) * 0.4
    panel = rng.standard_normal((nstates * nmo, n)) * 0.2
    return GwSlices(mo_energy=mo, nocc=1, fermi_energy=-0.2, states=np.arange(nstates), vph=f @ f.T, panel=panel,
                    xdiag=np.zeros((nmo, 1)), vxc_diag=np.zeros(nmo))


def _forms(sl, omegas):
    """x^T W_c x = -||L^{-1} D^{1/2} x||^2 with numpy in FP64."""
    delta = sl.mo_energy[1:] - sl.mo_energy[0]
    out = []
    for w in omegas:
        d = np.sqrt(4.0 * delta / (w * w + delta * delta))
        low = np.linalg.cholesky(np.eye(len(d)) + d[:, None] * sl.vph * d[None, :])
        out.append(-(np.linalg.solve(low, (sl.panel * d).T) ** 2).sum(axis=0))
    return np.array(out).reshape(len(omegas), len(sl.states), -1)


@pytest.mark.parametrize("n,nstates", [(1, 1), (15, 1), (16, 2), (17, 1), (63, 1), (64, 1), (65, 1), (127, 1), (128, 1),
                                       (129, 1), (191, 1), (192, 1), (193, 2), (257, 1), (320, 3)])
def test_forms_at_block_edges(n, nstates):
    from minigw_b200 import B200Backend

    sl = _system(n, max(1, n // 2), nstates, 100 + n)
    omegas = np.array([1e-3, 0.4, 7.0])
    with B200Backend(0) as be:
        be.load_slices(sl)
        q, _ = be.screened_forms(omegas, sl.states)
    ref = _forms(sl, omegas)
    # the bound of the other form tests: condition <= ~1e3 here, FP64 sums of length n
    assert np.abs(q - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("update", ["dmma", "ozaki"])
@pytest.mark.parametrize("n", [129, 193, 256, 257, 321, 385])
def test_next_block_beside_the_update(n, update, monkeypatch):
    """The next diagonal block, 64 or 128 wide, left out of the trailing update and factored beside it (few
    frequencies) or before it (more than there are SMs): the same forms bit for bit."""
    from minigw_b200 import B200Backend

    monkeypatch.setenv("GWB200_FP64_UPDATE", update)
    sl = _system(n, n // 2, 1, 900 + n)
    few = np.array([1e-3, 0.4, 7.0])
    with B200Backend(0) as be:
        be.load_slices(sl)
        q, _ = be.screened_forms(few, sl.states)
        many, _ = be.screened_forms(np.tile(few, 67), sl.states)
    ref = _forms(sl, few)
    assert np.abs(q - ref).max() <= 1e-11 * np.abs(ref).max()  # as above
    np.testing.assert_array_equal(many.reshape(67, 3, -1), np.broadcast_to(q.reshape(3, -1), (67, 3, q[0].size)))


@pytest.mark.parametrize("n", [257, 449, 512, 513, 577, 641])
def test_int8_update_in_pairs_of_blocks(n, monkeypatch):
    """One, two and three pairs of 128-column blocks with 64 or 128 columns or another block behind them: the
    forms of numpy, and scaled exactly with right-hand sides that are scaled by a power of two."""
    from minigw_b200 import B200Backend

    monkeypatch.setenv("GWB200_FP64_UPDATE", "ozaki")
    sl = _system(n, n // 2, 1, 1300 + n)
    omegas = np.array([1e-2, 0.9])
    with B200Backend(0) as be:
        be.load_slices(sl)
        q, _ = be.screened_forms(omegas, sl.states)
        sl.panel = sl.panel * 2.0**-300
        be.load_slices(sl)
        small, _ = be.screened_forms(omegas, sl.states)
        sl.panel = sl.panel * 2.0**300
    ref = _forms(sl, omegas)
    assert np.abs(q - ref).max() <= 1e-11 * np.abs(ref).max()  # as above
    np.testing.assert_array_equal(small * 2.0**600, q)


@pytest.mark.parametrize("n,pivot", [(40, 0), (40, 15), (40, 16), (100, 63), (100, 64), (200, 127), (200, 128), (200, 199)])
def test_reported_pivot(n, pivot):
    from minigw_b200 import B200Backend
    from minigw_b200._lib import GwB200Error

    sl = _system(n, 3, 1, 7)
    sl.vph = np.zeros((n, n))
    sl.vph[pivot, pivot] = -1e6  # eps is diagonal, negative at this one row
    with B200Backend(0) as be:
        be.load_slices(sl)
        with pytest.raises(GwB200Error) as e:
            be.screened_forms(np.array([0.3, 1.0]), sl.states)
        assert e.value.status == "GWB200_NOT_SPD" and f"pivot {pivot + 1} " in str(e.value)
        sl.vph[pivot, pivot] = 0.0
        be.load_slices(sl)  # the handle is usable afterwards
        q, _ = be.screened_forms(np.array([0.3]), sl.states)
    assert np.abs(q - _forms(sl, [0.3])).max() <= 1e-11 * np.abs(q).max()


def _forms_complex(sl, omegas, eta):
    """x^T W_c x with W_c = (I - diag(Pi0) V)^{-1} diag(Pi0), numpy in complex FP64."""
    delta = sl.mo_energy[1:] - sl.mo_energy[0]
    out = []
    for w in omegas:
        p = 2.0 * (1.0 / (1j * w - delta + 1j * eta) - 1.0 / (1j * w + delta - 1j * eta))
        y = np.linalg.solve(np.eye(len(p)) - p[:, None] * sl.vph, p[:, None] * sl.panel.T)
        out.append((sl.panel.T * y).sum(axis=0))
    return np.array(out).reshape(len(omegas), len(sl.states), -1)


@pytest.mark.parametrize("n,nstates", [(1, 1), (15, 1), (16, 1), (17, 2), (63, 1), (64, 1), (65, 1), (128, 1), (129, 1),
                                       (193, 1), (257, 2)])
def test_complex_forms_at_block_edges(n, nstates):
    from minigw_b200 import B200Backend

    sl = _system(n, max(1, n // 2), nstates, 300 + n)
    omegas = np.array([1e-3, 0.4, 7.0])
    with B200Backend(0) as be:
        be.load_slices(sl)
        q, _ = be.screened_forms_complex(omegas, sl.states, eta=0.02)
    ref = _forms_complex(sl, omegas, 0.02)
    assert np.abs(q - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("pivot", [0, 15, 16, 63, 64, 99])
def test_complex_reported_pivot(pivot):
    from minigw_b200 import B200Backend
    from minigw_b200._lib import GwB200Error

    sl = _system(100, 3, 1, 7)
    sl.vph = np.zeros((100, 100))
    sl.vph[pivot, pivot] = np.nan
    with B200Backend(0) as be:
        be.load_slices(sl)
        with pytest.raises(GwB200Error) as e:
            be.screened_forms_complex(np.array([0.3]), sl.states, eta=0.02)
        assert e.value.status == "GWB200_NOT_SPD" and f"pivot {pivot + 1} " in str(e.value)


@pytest.mark.parametrize("n,nstates", [(35, 8), (64, 5), (65, 5), (96, 6), (97, 6), (128, 4)])
def test_small_system_with_many_rows(n, nstates):
    """Systems of one kernel (n <= 128) whose row tiles are dealt out over the idle SMs: one frequency, a
    few, and more than there are SMs, the same forms bit for bit."""
    from minigw_b200 import B200Backend

    sl = _system(n, n // 2, nstates, 1500 + n)
    omegas = np.array([1e-3, 0.4, 7.0])
    with B200Backend(0) as be:
        be.load_slices(sl)
        q, _ = be.screened_forms(omegas, sl.states)
        one, _ = be.screened_forms(omegas[1:2], sl.states)
        many, _ = be.screened_forms(np.tile(omegas, 100), sl.states)
    ref = _forms(sl, omegas)
    assert np.abs(q - ref).max() <= 1e-11 * np.abs(ref).max()  # as above
    np.testing.assert_array_equal(one[0], q[1])
    np.testing.assert_array_equal(many.reshape(100, 3, -1), np.broadcast_to(q.reshape(3, -1), (100, 3, q[0].size)))


def test_few_frequencies_of_many_rows_use_the_idle_sms():
    """Two frequencies leave 146 SMs idle: 3510 rows (110 row tiles) may not take three times as long as 117
    rows (4 tiles).  Walked by one CTA per frequency they take ten times as long."""
    from minigw_b200 import B200Backend

    def best(nstates):
        sl = _system(116, 50, nstates, 1700)
        with B200Backend(0) as be:
            be.load_slices(sl)
            return min(be.screened_forms(np.array([0.1, 1.0]), sl.states)[1]["device_ms_screening"] for _ in range(10))

    assert best(30) < 3 * best(1)


def test_int8_update_with_rows_near_the_end_of_the_exponent_range(monkeypatch):
    """Rows that couple to the columns before them by 1e-295 .. 1e-323 alone, subnormal ones among them: nothing
    of theirs reaches the forms, and their scales may not either."""
    from minigw_b200 import B200Backend

    monkeypatch.setenv("GWB200_FP64_UPDATE", "ozaki")
    n, first = 449, 390
    sl = _system(n, n // 2, 1, 2100)
    weak = 10.0 ** -np.linspace(295.0, 323.0, n - first)
    sl.vph[first:, :] = weak[:, None]
    sl.vph[:, first:] = weak[None, :]
    sl.vph[np.arange(first, n), np.arange(first, n)] = 0.5
    omegas = np.array([1e-2, 0.9])
    with B200Backend(0) as be:
        be.load_slices(sl)
        q, _ = be.screened_forms(omegas, sl.states)
    ref = _forms(sl, omegas)
    assert np.abs(q - ref).max() <= 1e-11 * np.abs(ref).max()  # as above


@pytest.mark.parametrize("n", [65, 129, 193, 257])
def test_complex_next_block_beside_the_update(n):
    """eta != 0: the next diagonal block factored beside the trailing update (few frequencies) or before it (more
    than there are SMs), the same forms bit for bit."""
    from minigw_b200 import B200Backend

    sl = _system(n, n // 2, 1, 2300 + n)
    few = np.array([1e-3, 0.4, 7.0])
    with B200Backend(0) as be:
        be.load_slices(sl)
        q, _ = be.screened_forms_complex(few, sl.states, eta=0.02)
        many, _ = be.screened_forms_complex(np.tile(few, 67), sl.states, eta=0.02)
    ref = _forms_complex(sl, few, 0.02)
    assert np.abs(q - ref).max() <= 1e-11 * np.abs(ref).max()
    np.testing.assert_array_equal(many.reshape(67, 3, -1), np.broadcast_to(q.reshape(3, -1), (67, 3, q[0].size)))
