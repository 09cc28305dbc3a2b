"""The four-lane cell loop against the lane-per-cell loop and the oracle, bit for bit.

Sizes around a warp's 8 cells, a block's 32 and the resident groups; rulesets
with every conflict of transporters and effectors, cofactors equal to the
substrate or the product, zero rates; values that send a cell to its serial
form (NaN, infinities, -0, negative, above c_max, huge rates).
"""
import numpy as np
import pytest

from helpers import clustered_positions, random_cells, random_field

pytestmark = pytest.mark.gpu

DIMS = (40, 32, 24)


def phase(marl, dims, p, field, light, cells, lanes, reps=2):
    ctx = marl.Context(dims, p, cell_capacity=max(len(cells), 1))
    assert marl.load().marl_ctx_set_cell_lanes(ctx.h, lanes) == 0
    ctx.upload_field(field)
    ctx.upload_light(light)
    ctx.upload_cells(cells)
    ev = [ctx.cell_phase() for _ in range(reps)]
    out = ctx.download_field(), ctx.download_cells(), np.concatenate(ev)
    ctx.close()
    return out


def same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8))


def check(marl, oracle_mod, dims, field, light, cells, p=None, against_oracle=True):
    p = p or marl.default_params()
    quad = phase(marl, dims, p, field, light, cells, 32)
    same(quad, phase(marl, dims, p, field, light, cells, 31))  # 31 cells a warp: the lane-per-cell loop
    if not against_oracle:
        return
    w = oracle_mod.World(dims, p, seed=0, seed_count=None)
    w.set_field(field)
    w.set_cells(cells)
    w.set_light(light)
    for _ in range(2):
        ev = w.cell_phase()
    # As numbers: the CPU's NaN has other bits than the GPU's.
    np.testing.assert_array_equal(quad[0], w.field())
    np.testing.assert_array_equal(quad[1]["internal"], w.cells()["internal"])
    np.testing.assert_array_equal(quad[2][len(cells):].astype(np.int32), np.asarray(ev).astype(np.int32))


def case(seed, n=None, frac=0.2, dims=DIMS):
    rng = np.random.default_rng(seed)
    pos = clustered_positions(dims, frac, rng)
    cells = random_cells(dims, len(pos), rng, positions=pos)
    cells = cells if n is None else cells[:n]
    light = rng.random(dims[::-1], dtype=np.float32)
    return rng, random_field(dims, rng, 2.0), light, cells


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 32, 33, 257, None])
def test_sizes(marl, oracle_mod, n):
    _, field, light, cells = case(3, n)
    check(marl, oracle_mod, DIMS, field, light, cells)


def test_more_cells_than_groups(marl, oracle_mod):
    dims = (96, 96, 48)
    _, field, light, cells = case(5, frac=0.12, dims=dims)
    assert len(cells) > 32 * 6 * 148
    check(marl, oracle_mod, dims, field, light, cells)


@pytest.mark.parametrize("kind", ["one_pair", "two_pairs", "cofactors", "zero_rates", "idle", "invalid_slots", "boxed_in"])
def test_rulesets(marl, oracle_mod, kind):
    rng, field, light, cells = case(11, 900, frac=0.5 if kind == "boxed_in" else 0.2)
    rs, n = cells["ruleset"], len(cells)
    if kind in ("one_pair", "two_pairs"):  # every slot conflicts with the one before, or the one before that
        k = np.arange(8) % (1 if kind == "one_pair" else 2)
        for part in ("transport", "effectors"):
            rs[part]["int_species"], rs[part]["ext_species"] = k, k + 3
        rs["effectors"]["threshold"] *= np.float32(0.05)
    elif kind == "cofactors":  # cofactor = substrate, product, catalyst or another
        rx = rs["reactions"]
        pick = rng.integers(0, 4, (n, 16))
        other = rng.integers(0, 16, (n, 16))
        rx["cofactor"] = np.choose(pick, [rx["substrate"], rx["product"], rx["catalyst"], other])
    elif kind == "zero_rates":
        for part, names in (("transport", ("uptake_rate", "secrete_rate")), ("effectors", ("rate",))):
            for name in names:
                rs[part][name] *= rng.random((n, 8)) < 0.4
        rs["reactions"]["v_max"] *= rng.random((n, 16)) < 0.3
        cells["internal"] *= rng.random((n, 16)) < 0.3
        field *= rng.random(field.shape) < 0.5
    elif kind == "idle":
        rs["transport"]["uptake_rate"] = rs["transport"]["secrete_rate"] = rs["effectors"]["rate"] = 0
        rs["reactions"]["v_max"] = 0
    elif kind == "invalid_slots":  # species that do not exist: such slots do nothing
        for part in ("transport", "effectors"):
            for name in ("int_species", "ext_species"):
                bad = rng.random((n, 8)) < 0.2
                rs[part][name][bad] = 200
        for name in ("substrate", "product", "catalyst", "cofactor"):
            bad = rng.random((n, 16)) < 0.1
            rs["reactions"][name][bad] = 77
    check(marl, oracle_mod, DIMS, field, light, cells, against_oracle=kind != "invalid_slots")


@pytest.mark.parametrize("kind", ["negative_rates", "huge_rates", "denormal", "over_c_max", "nan", "inf", "minus_zero",
                                  "negative_field", "light", "c_max_inf"])
def test_values_out_of_the_ordinary(marl, oracle_mod, kind):
    rng, field, light, cells = case(17, 700)
    rs, n = cells["ruleset"], len(cells)
    p = marl.default_params()
    some = rng.random(n) < 0.3  # the others share warps with them
    if kind == "negative_rates":
        rs["reactions"]["v_max"][some] *= rng.choice([-1.0, 1.0], (some.sum(), 16)).astype(np.float32)
        rs["transport"]["uptake_rate"][some] *= np.float32(-1)
        rs["effectors"]["rate"][some] *= np.float32(-1)
    elif kind == "huge_rates":
        rs["transport"]["secrete_rate"][some] *= np.float32(3e38)
        rs["reactions"]["v_max"][some] *= np.float32(1e37)
    elif kind == "denormal":
        field *= np.float32(1e-39)
        cells["internal"][some] *= np.float32(1e-38)
    elif kind == "over_c_max":
        cells["internal"][some] += np.float32(20)
    elif kind in ("nan", "inf"):
        cells["internal"][some, 3] = np.float32(kind)
        field[rng.random(field.shape) < 0.01] = np.float32(kind)
    elif kind == "minus_zero":
        cells["internal"][some] = np.float32(-0.0)
        field[rng.random(field.shape) < 0.3] = np.float32(-0.0)
    elif kind == "negative_field":
        field -= np.float32(0.5)
    elif kind == "light":
        light[rng.random(light.shape) < 0.3] = np.float32(50)
        light[rng.random(light.shape) < 0.1] = np.float32(-1)
    else:
        p.c_max = np.float32("inf")
    check(marl, oracle_mod, DIMS, field, light, cells, p, against_oracle=kind not in ("nan", "inf"))
