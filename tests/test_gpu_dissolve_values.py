"""The dissolution update's arithmetic over the whole range of acid values, bit for bit against
the oracle's sequential sweep: quotients by one flux sum formed from its reciprocal (normal
range), divisions outside it (subnormal, tiny and huge acid), zeros, negative acid (a solve's
undershoot), faces on the domain boundary, both label widths, more slices than one pass of the
schedule table."""
import numpy as np
import pytest

from helpers import params
from leachingsim_gb300.runtime import Context

pytestmark = pytest.mark.gpu

PORE, ROCK, SULPHIDE, PRECIPITATE = 2, 3, 4, 5


@pytest.mark.parametrize("label_bytes", [1, 2])
@pytest.mark.parametrize("kind", ["unit", "wide", "tiny", "mixed"])
def test_update_matches_oracle_bit_for_bit(oracle_mod, label_bytes, kind):
    shape = (13, 9, 22)
    rng = np.random.default_rng(len(kind) * 10 + label_bytes)
    lab = rng.choice([1, PORE, ROCK, SULPHIDE, PRECIPITATE], size=shape, p=[0.05, 0.35, 0.25, 0.3, 0.05])
    acid = {"unit": rng.random(shape), "wide": 10.0 ** rng.uniform(-250, 1, shape),
            "tiny": 10.0 ** rng.uniform(-323, -290, shape),
            "mixed": np.where(rng.random(shape) < 0.5, rng.random(shape), 10.0 ** rng.uniform(-320, -200, shape))}[kind]
    acid = np.where(rng.random(shape) < 0.2, 0.0, acid)
    if kind != "tiny":
        acid = np.where(rng.random(shape) < 0.1, -1e-3 * acid, acid)
    frac = np.where(lab >= SULPHIDE, rng.uniform(0.05, 1.0, shape), 0.0).astype(np.float32)
    p = params(kreac=0.7, D=1.3, dx=0.9, time_scalar=3.0)
    o = oracle_mod.Oracle(shape, label_bytes=label_bytes, params=p, mode=oracle_mod.SOLVE_TIGHT)
    o.load_labels(lab.astype(np.uint8 if label_bytes == 1 else np.uint16))
    o.init_all()
    g = Context(shape, label_bytes=label_bytes, params=p)
    g.upload("label", lab.astype(np.uint8 if label_bytes == 1 else np.uint16))
    g.init_all()
    o.set("frac", frac)
    g.upload("frac", frac)
    o.set("acid", acid)
    g.upload("acid", acid)
    for _ in range(2):
        n_o, io = o.dissolve(1.0)
        n_g, ig = g.dissolve(1.0)
        assert n_o == n_g and io["num_steps"] == ig["num_steps"]
        np.testing.assert_array_equal(g.download("label"), o.get("label").astype(g.download("label").dtype))
        for f in ("frac", "acid", "conc", "precipitate"):
            np.testing.assert_array_equal(g.download(f), o.get(f), err_msg=f)
    g.close()


def test_many_substeps(oracle_mod):
    """600 sub-steps: a level holds more slices than one pass of the schedule (512)."""
    shape = (80, 60, 1200 // 10)
    rng = np.random.default_rng(3)
    lab = np.full(shape, ROCK, np.uint8)
    sel = rng.random(shape) < 0.002
    lab[sel] = SULPHIDE
    acid = np.full(shape, 1.0)
    frac = np.where(sel, 1.0, 0.0).astype(np.float32)
    p = params(kreac=1e9, D=20.0, time_scalar=0.5)  # rate 6 * 20 * 0.5 = 60 per unit time: 600 sub-steps
    o = oracle_mod.Oracle(shape, params=p, mode=oracle_mod.SOLVE_TIGHT)
    o.load_labels(lab)
    o.init_all()
    g = Context(shape, params=p)
    g.upload("label", lab)
    g.init_all()
    for a, up in ((o, o.set), (g, g.upload)):
        up("frac", frac)
        up("acid", acid)
    n_o, io = o.dissolve(1.0)
    n_g, ig = g.dissolve(1.0)
    assert io["num_steps"] == ig["num_steps"] > 512 and n_o == n_g
    np.testing.assert_array_equal(g.download("frac"), o.get("frac"))
    np.testing.assert_array_equal(g.download("acid"), o.get("acid"))
    g.close()
