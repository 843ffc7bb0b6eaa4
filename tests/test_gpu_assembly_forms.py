"""Black-oil assembly at the cells and connections that leave the assembly's short form -- no-oil cells and
potential differences of exactly zero -- beside the ones that take it (both states,
below the connate saturation, an empty kro denominator), over the orders of the unknowns and equations, with capillary
pressure and with and without gravity: the oracle's J and R bit for bit (the oracle restates the reference's operations
one by one, so no tolerance applies)."""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,eq", [((1, 2), (0, 1, 2)), ((2, 1), (2, 0, 1))])
@pytest.mark.parametrize("gravity", [0.0, 1.0 / 144.0])
@pytest.mark.parametrize("no_oil", [False, True])
def test_short_and_full_forms_match_oracle(slots, eq, gravity, no_oil):
    pytest.importorskip("torch")
    from oracle import Oracle
    from ressim_gb300.assembly import BlackOilAssembler
    z = dict(np.load(os.path.join(GOLDEN, "waterflood_asm.npz"), allow_pickle=False))
    z["vars"] = np.array([*slots, *eq], dtype=z["vars"].dtype)
    z["gravity"] = np.array([gravity])
    z["pcow_y"] = np.linspace(9.0, 0.0, z["pcow_x"].size) ** 2
    z["pcog_y"] = np.linspace(0.0, 4.0, z["pcog_x"].size)
    na = int(z["na"][0])
    rng = np.random.default_rng(7)
    p = rng.uniform(500.0, 6000.0, na)
    sw = rng.uniform(0.0, 0.9, na)
    state = rng.integers(0, 2, na).astype(np.uint8)
    x = np.where(state == 1, rng.uniform(0.0, 0.5, na), rng.uniform(0.0, 1.2, na))
    acc = rng.standard_normal(3 * na)
    sw[:40:2] = float(z["krw_x"][0])                 # connate water
    x[:40:4] = 0.0                                   # ... and no gas: nothing to weigh kro with
    p[100:140], sw[100:140], x[100:140], state[100:140] = 3000.0, 0.4, 0.3, 1     # equal potentials along a row
    if no_oil:
        state[200:260:3] = 2
    args = (p, sw, x, state, acc, 3.0)
    Jo, Ro = Oracle().bo_assemble(z, *args)
    with BlackOilAssembler(z) as asm:
        J, R = asm.assemble(*args)
    assert np.array_equal(J, Jo), np.flatnonzero(J != Jo)[:10]
    assert np.array_equal(R, Ro), np.flatnonzero(R != Ro)[:10]


@pytest.mark.parametrize("slots,eq", [((1, 2), (0, 1, 2)), ((2, 1), (2, 0, 1))])
@pytest.mark.parametrize("gravity", [0.0, 1.0 / 144.0])
@pytest.mark.parametrize("general", ["sw", "x", "both", "tables"])
def test_general_cells_among_plain_ones_match_oracle(slots, eq, gravity, general):
    """Cells that take the full form although everything stays finite: saturations just above 2^256 (single cells among plain
    ones, neighbours of each other and of no-oil cells), and a model whose tables hold a value that is not finite and that no
    cell reaches, which makes every cell general."""
    pytest.importorskip("torch")
    from oracle import Oracle
    from ressim_gb300.assembly import BlackOilAssembler
    z = dict(np.load(os.path.join(GOLDEN, "waterflood_asm.npz"), allow_pickle=False))
    z["vars"] = np.array([*slots, *eq], dtype=z["vars"].dtype)
    z["gravity"] = np.array([gravity])
    na = int(z["na"][0])
    rng = np.random.default_rng(11)
    p = rng.uniform(500.0, 6000.0, na)
    sw = rng.uniform(0.2, 0.8, na)
    state = rng.integers(0, 2, na).astype(np.uint8)
    x = np.where(state == 1, rng.uniform(0.0, 0.2, na), rng.uniform(0.0, 1.2, na))
    acc = rng.standard_normal(3 * na)
    wide = np.array([7, 8, 60, 61, 200, na - 1])
    if general in ("sw", "both"):
        sw[wide[::2]] = 2.0 ** 256 * np.array([1.0, -1.5, 1.25])
    if general in ("x", "both"):
        state[wide[1::2]] = 1
        x[wide[1::2]] = 2.0 ** 256 * np.array([1.0, -1.25, 1.5])
        state[wide[1] + 1] = 2
    if general == "tables":
        z["deadB_x"], z["deadB_y"] = np.array([0.0, 1.0]), np.array([np.inf, 1.0])   # (live oil does not read the dead-oil tables)
    args = (p, sw, x, state, acc, 3.0)
    Jo, Ro = Oracle().bo_assemble(z, *args)
    assert np.isfinite(Jo).all() and np.isfinite(Ro).all()
    with BlackOilAssembler(z) as asm:
        J, R = asm.assemble(*args)
    assert np.array_equal(J, Jo), np.flatnonzero(J != Jo)[:10]
    assert np.array_equal(R, Ro), np.flatnonzero(R != Ro)[:10]
