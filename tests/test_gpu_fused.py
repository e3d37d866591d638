"""The fused one- and two-step passes (csrc/yee_fused.cuh) against the
separate H and E kernels: every value comes from the same operations in the
same order, so fields, probe traces and energies are the same bits."""
import numpy as np
import pytest

import openems_b200 as oe
from scenarios import (Scenario, cpml_scenarios, mur_scenarios, odd_scenarios, probe_scenario, reference_scenarios,
                       run_engine, run_oracle)
from test_gpu_parity import assert_parity

pytestmark = pytest.mark.gpu


def random_scenario(seed, dims, layers=None, mur=0, disp=False, steps=37):
    """Boxes, PEC, soft and hard sources (two on one cell), probes on the
    faces and inside; an odd step count in uneven batches, energies that cut
    the spans."""
    rng = np.random.default_rng(seed)
    n = np.array(dims)

    def box():
        a = rng.integers(0, n)
        b = np.minimum(a + rng.integers(1, np.maximum(n // 2, 2)), n)
        return tuple(int(v) for d in range(3) for v in (a[d], b[d]))

    def cell():
        return tuple(int(v) for v in rng.integers(0, n))

    tau = 1.0 / (np.pi * 20e9)
    c0 = cell()
    exc = [oe.Excitation.gaussian_pulse(tau, 0.5 * tau, int(rng.integers(3)), cell()) for _ in range(3)]
    exc += [oe.Excitation.gaussian_pulse(tau, 0.5 * tau, 1, c0).hard_source(),
            oe.Excitation.gaussian_pulse(tau, 0.3 * tau, 1, c0)]
    probes = [(int(rng.integers(6)), cell()) for _ in range(5)]
    probes += [(2, (0, 0, 0)), (4, tuple(int(v) - 1 for v in n)), (1, c0)]
    sc = Scenario(f"random_{seed}", tuple(dims), 1e-3,
                  materials=[(float(rng.uniform(1, 9)), float(rng.uniform(1, 3)), float(rng.uniform(0, 0.2)),
                              float(rng.uniform(0, 50)), box()) for _ in range(4)],
                  pec=[box()], excitations=exc, num_steps=steps, sample_interval=5, probes=probes,
                  batches=(steps - 12, 12))
    if layers is not None:
        sc.cpml = oe.CpmlBoundaries(layers=layers, alpha_max=0.05, kappa_max=2.0)
    if mur:
        sc.mur = oe.MurAbcConfig.all(mur)
    if disp:
        cells = np.unique(np.array([cell() for _ in range(40)], dtype=np.uint64), axis=0)
        sc.dispersive = [(oe.DrudeMaterial(2e11, 1e9, second_order=True), cells), (oe.DebyeMaterial(1e-11, 2.0), cells[:7])]
    return sc


# rows of one chunk, one plane, a chunk count below, at and above a tile;
# more rows than any CTA holds; rows longer than a CTA's threads
SIZES = [(1, 1, 1), (2, 3, 5), (1, 40, 33), (33, 1, 64), (40, 33, 1), (9, 130, 12), (5, 20, 2100), (30, 61, 67),
         (70, 66, 130)]
LAYERS = {(9, 130, 12): (3, 2, 8, 8, 5, 6), (30, 61, 67): (8, 0, 6, 10, 0, 9), (70, 66, 130): (8,) * 6,
          (5, 20, 2100): (0, 2, 5, 5, 7, 8), (1, 40, 33): (0, 0, 8, 8, 8, 8)}


def same(a, b):
    assert a["engine"].launch_info()["staged"] == 5 and b["engine"].launch_info()["staged"] != 5
    assert np.array_equal(a["fields"], b["fields"]), np.abs(a["fields"] - b["fields"]).max()
    assert np.array_equal(a["traces"], b["traces"]) and a["energy"] == b["energy"]


@pytest.mark.parametrize("dims", SIZES)
def test_sizes_against_separate_kernels(dims):
    for layers in (None, LAYERS.get(dims)):
        sc = random_scenario(sum(dims), dims, layers)
        ref = run_engine(sc, kernels="register", autotune=False)
        same(run_engine(sc, autotune=False), ref)
        if layers is not None or dims == (2, 3, 5):
            same(run_engine(sc), ref)
            same(run_engine(sc, compressed=True, graphs=False), ref)


@pytest.mark.parametrize("dims,layers", [((2, 2300, 2310), None), ((8, 2000, 2000), (2, 2, 8, 8, 8, 8))])
def test_wide_planes(dims, layers):
    """More tiles in one (y, z) plane than 16 items an SM."""
    sc = random_scenario(12, dims, layers, steps=17)
    sc.batches = (12, 5)
    same(run_engine(sc, autotune=False), run_engine(sc, kernels="register", autotune=False))


def test_one_grid_with_other_slabs():
    """Engines of one size whose slabs lie on other faces each get boxes of
    their own (plans are kept per grid and slab layout)."""
    for layers in ((8, 0, 0, 0, 0, 0), (0, 8, 0, 0, 0, 0), (0, 0, 8, 0, 0, 0), (0, 0, 0, 8, 0, 0), (0, 0, 0, 0, 8, 0),
                   (0, 0, 0, 0, 0, 8), (4, 4, 0, 0, 0, 0)):
        sc = random_scenario(11, (70, 66, 130), layers)
        same(run_engine(sc), run_engine(sc, kernels="register", autotune=False))


@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_two_byte_storage(storage):
    for layers in (None, (8, 0, 6, 10, 0, 9)):
        sc = random_scenario(5, (30, 61, 67), layers)
        same(run_engine(sc, storage=storage), run_engine(sc, storage=storage, kernels="register", autotune=False))


@pytest.mark.parametrize("mur,disp", [(1, False), (2, False), (0, True), (2, True)])
def test_hooks_run_one_step_a_pass(mur, disp):
    sc = random_scenario(6, (30, 31, 35), (6,) * 6 if disp and not mur else None, mur, disp)
    sc.rlc = [oe.RlcElement.parallel_rlc((15, 15, 15), 2, r=50.0, c=1e-13)] if disp else []
    # (untimed: the tuner may find the separate kernels faster for one-step passes)
    same(run_engine(sc, autotune=False), run_engine(sc, kernels="register", autotune=False))


@pytest.mark.parametrize("compressed", [False, True])
@pytest.mark.parametrize("mur,disp", [(1, False), (0, True)])
def test_timed_route_of_one_step_passes(mur, disp, compressed):
    """Whichever of the two the tuner takes, with what it ran on the way."""
    sc = random_scenario(9, (30, 31, 35), (6,) * 6 if disp else None, mur, disp)
    ref = run_engine(sc, kernels="register", autotune=False)
    for _ in range(2):
        got = run_engine(sc, compressed=compressed)
        assert {r["kind"] for r in got["engine"].tune_report()} > {5}
        assert np.array_equal(got["fields"], ref["fields"]) and np.array_equal(got["traces"], ref["traces"])
        assert got["energy"] == ref["energy"]


def test_many_coefficient_sets():
    """More than 256 sets take 2-byte ids; more than 65,536 keep the full
    arrays (and the separate kernels)."""
    sc = random_scenario(7, (20, 30, 41), (4,) * 6)
    rng = np.random.default_rng(7)
    sc.materials = [(float(rng.uniform(1, 9)), 1.0, 0.0, 0.0, (i, i + 1, j, j + 1, 3, 30))
                    for i in range(20) for j in range(30)]
    same(run_engine(sc), run_engine(sc, kernels="register", autotune=False))
    sc = random_scenario(8, (41, 42, 43))
    sc.materials = [(1.0 + 1e-4 * (i * 1806 + j * 43 + k), 1.0, 0.0, 0.0, (i, i + 1, j, j + 1, k, k + 1))
                    for i in range(41) for j in range(42) for k in range(43)]
    got = run_engine(sc, autotune=False)
    assert got["engine"].launch_info()["staged"] != 5
    assert np.array_equal(got["fields"], run_engine(sc, kernels="register", autotune=False)["fields"])


@pytest.mark.parametrize("sc", reference_scenarios() + odd_scenarios() + cpml_scenarios() + mur_scenarios() +
                         [probe_scenario()], ids=lambda s: s.name)
def test_against_the_oracle(sc):
    got = run_engine(sc)
    assert got["engine"].launch_info()["staged"] == 5
    assert_parity(got, run_oracle(sc))


@pytest.mark.parametrize("layers,mur,disp,storage", [((8, 0, 6, 10, 0, 9), 0, False, "f32"), (None, 0, False, "f16"),
                                                     ((6,) * 6, 0, True, "f32"), (None, 2, False, "f32")])
def test_state_after_an_odd_number_of_passes(layers, mur, disp, storage):
    """The buffers a pass swaps are the current ones for whatever reads or
    writes the state next: energies, checkpoints to and from the separate
    kernels, resets and written fields."""
    sc = random_scenario(13, (30, 31, 35), layers, mur, disp)  # 25 + 12 steps: 19 passes, or 37

    def more(run, n, start):
        eng, dt = run["engine"], run["operator"].timestep()
        eng.run_batch(oe.EngineBatch(num_steps=n, excitations=[
            oe.ScheduledExcitation.from_excitation(x, start, n, dt) for x in sc.excitations]))
        return np.concatenate(eng.read_fields())

    def fresh(**kw):
        return run_engine(sc, storage=storage, autotune=False, **kw)

    def story(run, other):
        eng, out = run["engine"], []
        out += [run["fields"], np.array(eng.energy())]
        blob = eng.save_state()
        out += [more(run, 9, 37), more(run, 3, 46)]  # 5 passes more, then 2
        eng.load_state(blob)
        out += [np.concatenate(eng.read_fields()), np.array(eng.energy()), more(run, 9, 37)]
        other["engine"].load_state(blob)
        out += [more(other, 9, 37)]
        f = np.random.default_rng(1).standard_normal((2, 3, 30, 31, 35)).astype(np.float16).astype(np.float32)
        eng.write_fields(f[0], f[1] / 512)
        out += [np.concatenate(eng.read_fields()), more(run, 5, 46)]
        eng.reset()
        out += [np.concatenate(eng.read_fields()), more(run, 25, 0), np.array(eng.energy())]
        return out

    a, b = fresh(), fresh(kernels="register")
    assert a["engine"].launch_info()["staged"] == 5 and b["engine"].launch_info()["staged"] != 5
    for x, y in zip(story(a, fresh(kernels="register")), story(b, fresh())):
        assert np.array_equal(x, y)
