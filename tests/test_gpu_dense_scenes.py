"""Scenes that reach every way through the colour pass's lists, the body tiles' chains of
displacement and the record and temperature read-outs, against the oracle bit for bit.

The colour pass lists the cells that a rule may change and treats apart liquids that flow,
liquids in free fall, liquids beside another liquid, cells that emit several particles, and
chunks whose edge or world width rules out its wider accesses: the scenes mix all of
these in worlds at and around those edges. All results are whole numbers or bit
patterns, so every comparison is exact.
"""
import numpy as np
import pytest

from helpers import compare_particles, compare_states, material_types
from oracle.binding import ORDER_PART

pytestmark = pytest.mark.gpu

MATERIALS = ("GENERIC_AIR", "GENERIC_SAND", "DIRT", "GOLD_ORE", "WATER", "LAVA", "GENERIC_LIQUID", "GENERIC_GAS",
             "STEAM", "STONE", "FIRE")


def _scene(fse, w, h, seed, f32, fire=True):
    """Random planes: every material, liquid amounts from nothing to 40 (a cell in free
    fall then becomes ten particles), settled and unsettled, with pending diffs; AIR
    bands of four and more rows for cells to fall into."""
    rng = np.random.default_rng(seed)
    ids = np.array([fse.material_find(n) for n in MATERIALS])
    p = np.array([0.16, 0.16, 0.06, 0.04, 0.2, 0.06, 0.06, 0.08, 0.04, 0.12, 0.02])
    if not fire:
        p[-1] = 0.0
    idp = rng.choice(ids, (h, w), p=p / p.sum()).astype(np.uint16)
    for y in range(9, h, 23):
        idp[y:y + int(rng.integers(4, 8))] = ids[0]
    types = material_types(fse)
    soup = types[idp] == 3
    amount = np.where(rng.random((h, w)) < 0.15, rng.uniform(8.0, 40.0, (h, w)), rng.choice(
        [0.0, 0.0004, 0.0006, 0.004, 0.006, 0.3, 0.5, 1.0, 2.0, 3.7], (h, w)))
    diff = rng.choice([0.0, 0.0, 0.0, 0.2, -0.1, 1.5], (h, w))
    if f32:
        sc, df = amount.astype(np.float32).view(np.int32), diff.astype(np.float32).view(np.int32)
    else:
        sc, df = (amount * 65536).astype(np.int32), (diff * 65536).astype(np.int32)
    temp = rng.integers(-600, 900, (h, w)).astype(np.int32)
    air = types[idp] == 0
    return {"id": idp, "colour": np.where(air, 0, rng.integers(0, 1 << 32, (h, w))).astype(np.uint32),
            "scalar": np.where(soup, sc, np.where(air, 0, temp)).astype(np.int32),
            "flags": np.where(air, 0, rng.choice([0, 3, 9, 0x80, 0x80 | 10], (h, w))).astype(np.uint8),
            "diff": np.where(soup, df, 0).astype(np.int32)}


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("w,h,chunk,fire", [(132, 131, 128, False), (127, 260, 128, True), (256, 128, 128, False),
                                            (70, 66, 64, True), (40, 48, 16, False)])
def test_dense_scene_matches_oracle(fse, oracle_mod, w, h, chunk, fire, f32):
    types = material_types(fse)
    seed = w * 7 + h + chunk
    world = fse.World(w, h, chunk_size=chunk, seed=seed, f32_fluid=f32)
    world.upload(_scene(fse, w, h, seed, f32, fire))
    ow = oracle_mod.OracleWorld(w, h, chunk, 3, seed)
    ow.set_f32(f32)
    ow.set_state(world.state())
    many = 0
    for t in range(4):
        world.step(1)
        ow.step(1, ORDER_PART)
        what = "%dx%d chunk %d f32 %d step %d" % (w, h, chunk, f32, t)
        compare_states(world.state(), ow.state(), types, what)
        compare_particles(world.particles(), ow.particles(), what)
        many += len(world.particles())
    assert many > 0
    np.testing.assert_array_equal(world.ledger(), ow.ledger())
    world.close()


def test_sinking_by_density_matches_oracle(fse, oracle_mod):
    """Sand sinks into AIR and into what is less dense: equal, negative and NaN densities."""
    om = oracle_mod.Oracle()
    extra = [("NAN_SAND", 2, float("nan")), ("NEG_SAND", 2, -3.0), ("SAND_A", 2, 1.5), ("SAND_B", 2, 1.5),
             ("NAN_LIQUID", 3, float("nan")), ("NEG_LIQUID", 3, -4.0)]
    try:
        names = ["GENERIC_AIR", "GENERIC_SAND", "WATER", "STONE"]
        for k, (name, kind, density) in enumerate(extra):
            a = fse.RegisterMaterial(200 + k, name, name, kind, 8, 255, density, 2)
            b = om.register(200 + k, name, name, kind, 8, 255, density, 2)
            assert a == b
            names.append(name)
        fse.PushMaterials()
        types = material_types(fse)
        w, h, seed = 160, 96, 5
        rng = np.random.default_rng(seed)
        ids = rng.choice([fse.material_find(n) for n in names], (h, w)).astype(np.uint16)
        world = fse.World(w, h, seed=seed)
        world.upload({"id": ids, "colour": rng.integers(0, 1 << 32, (h, w)).astype(np.uint32),
                      "scalar": np.where(types[ids] == 3, 65536, 0).astype(np.int32),
                      "flags": rng.choice([0, 0x80], (h, w)).astype(np.uint8), "diff": np.zeros((h, w), np.int32)})
        ow = oracle_mod.OracleWorld(w, h, 128, 3, seed)
        ow.set_state(world.state())
        for t in range(4):
            world.step(1)
            ow.step(1, ORDER_PART)
            compare_states(world.state(), ow.state(), types, "densities step %d" % t)
            compare_particles(world.particles(), ow.particles(), "densities step %d" % t)
        world.close()
    finally:
        fse.InitMaterials()
        fse.PushMaterials()
        om.reset_materials()


@pytest.mark.parametrize("n,side,spread", [(1, 8, 200), (60, 24, 60), (12, 64, 20)])
def test_overlapping_bodies_match_oracle(fse, oracle_mod, n, side, spread):
    """Boxes on top of each other and across the world's edge: long chains of displacement."""
    types = material_types(fse)
    w, h, seed = 260, 200, 40 + n
    world = fse.World(w, h, seed=seed)
    world.generate(fse.GEN_MIX, seed)
    ow = oracle_mod.OracleWorld(w, h, 128, 3, seed)
    ow.set_state(world.state())
    rng = np.random.default_rng(seed)
    b = np.zeros(n, fse.BODY_DTYPE)
    b["w"], b["h"] = rng.integers(1, side + 1, n), rng.integers(1, side + 1, n)
    b["x"] = rng.uniform(-4, spread, n)
    b["y"] = rng.uniform(-4, spread, n)
    a = rng.uniform(0, 2 * np.pi, n)
    b["sin_a"], b["cos_a"] = np.sin(a), np.cos(a)
    b["id"] = fse.material_find("GENERIC_OBJECT")
    b["colour"] = 0xFF808080
    ob = b.copy()
    for t in range(2):
        world.object_stamp(b)
        ow.object_stamp(ob)
        compare_states(world.state(), ow.state(), types, "stamp %d" % t)
        compare_particles(world.particles(), ow.particles(), "stamp %d" % t)
        world.step(1)
        ow.step(1, ORDER_PART)
        assert world.object_readback(b) == ow.object_readback(ob)
        compare_states(world.state(), ow.state(), types, "readback %d" % t)
        np.testing.assert_array_equal(b, ob)
    np.testing.assert_array_equal(world.ledger(), ow.ledger())
    world.trim()
    world.close()


@pytest.mark.parametrize("n", [1, 255, 257, (1 << 18) + 37])
def test_particle_records_come_back(fse, n):
    """Every field of every record, across the blocks and pieces of the read-out."""
    world = fse.World(64, 64, particle_capacity=1 << 19)
    rng = np.random.default_rng(n)
    p = np.zeros(n, fse.PARTICLE_DTYPE)
    for name in p.dtype.names:
        dt = p.dtype[name]
        if name not in ("reserved", "temperature", "id"):
            p[name] = rng.uniform(-9, 9, n) if dt.kind == "f" else rng.integers(0, 120, n)
    p["id"] = fse.material_find("WATER")
    world.addCell(p)
    want = p.copy()
    want["flags"] &= 0xBF  # bit 6 is reserved and cleared as particles are added
    assert world.particles().tobytes() == want.tobytes()
    world.trim()
    assert world.particles().tobytes() == want.tobytes()
    world.close()


@pytest.mark.parametrize("w,h", [(1, 1), (7, 1), (37, 13), (64, 8)])
def test_temperatures_come_back(fse, w, h):
    """Sizes that are no multiple of the cells a thread reads at once."""
    rng = np.random.default_rng(w * h)
    world = fse.World(w, h, temperature=True)
    ids = rng.choice([fse.material_find(n) for n in ("GENERIC_AIR", "WATER", "STONE")], (h, w)).astype(np.uint16)
    world.upload({"id": ids, "colour": np.zeros((h, w), np.uint32), "scalar": np.full((h, w), 70000, np.int32),
                  "flags": np.zeros((h, w), np.uint8), "diff": np.zeros((h, w), np.int32)})
    t = rng.integers(-32768, 32768, (h, w)).astype(np.int16)
    world.set_temperature(t)
    np.testing.assert_array_equal(world.temperature(), t)
    world.close()
