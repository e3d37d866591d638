"""What the engine library's host code does when a call fails or a limit is
reached: the library's own sources built against fake_cudart.cpp (device
memory on the host, kernels that only leave their names), each test in a
process of its own."""
import os
import subprocess
import sys
import textwrap

import pytest

from openems_b200 import build as engine_build

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(HERE, "_build")
LIB = os.path.join(OUT, "liboems_fake.so")

HEAD = """
import ctypes, sys
import numpy as np
import openems_b200._native as N
N.LIB_PATH = %r
import openems_b200 as oe
L, F = N.lib(), ctypes.CDLL(N.LIB_PATH)
for f in ("fake_launched", "fake_pool_used", "fake_pinned", "fake_pins", "fake_instantiated", "fake_largest_graph"):
    getattr(F, f).restype = ctypes.c_longlong
F.fake_set.argtypes = [ctypes.c_char_p, ctypes.c_longlong]

def knob(key, value):
    F.fake_set(key.encode(), value)

def launched(part, reset=False):
    return F.fake_launched(part.encode(), int(reset))

def engine(dims, layers=None, **kw):
    e = oe.Engine(oe.Operator(oe.Grid.uniform(*dims, 1e-3), oe.BoundaryConditions.all_pec()), **kw)
    if layers:
        e.add_cpml(oe.CpmlBoundaries(layers=layers))
    return e

def batch(n):
    return oe.EngineBatch(num_steps=n)

def fused(e):
    return e.launch_info()["staged"] == 5
"""


@pytest.fixture(scope="module")
def child():
    os.makedirs(OUT, exist_ok=True)
    csrc = os.path.join(engine_build.HERE, "csrc")
    fake = os.path.join(HERE, "fake_cudart.cpp")
    deps = [fake] + [os.path.join(csrc, f) for f in os.listdir(csrc)] + \
           [os.path.join(engine_build.ROOT, "include", f) for f in os.listdir(os.path.join(engine_build.ROOT, "include"))]
    if not os.path.exists(LIB) or max(map(os.path.getmtime, deps)) > os.path.getmtime(LIB):
        flags = ["-gencode", "arch=compute_100a,code=compute_100a", "-O1", "-Xcicc", "-O0", "-std=c++17", "-Xcompiler",
                 "-fPIC", "--expt-relaxed-constexpr", "-I", os.path.join(engine_build.ROOT, "include")]
        jobs, objs = [], []
        for src in [os.path.join(engine_build.HERE, s) for s in engine_build.SOURCES] + [fake]:
            objs.append(os.path.join(OUT, os.path.basename(src) + ".o"))
            jobs.append(subprocess.Popen([engine_build._nvcc(), *flags, "-c", src, "-o", objs[-1]]))
        assert [j.wait() for j in jobs] == [0] * len(jobs)
        subprocess.run(["g++", "-shared", "-Wl,--no-undefined", "-o", LIB + ".tmp", *objs, "-lpthread", "-ldl"], check=True)
        os.replace(LIB + ".tmp", LIB)

    def run(code):
        r = subprocess.run([sys.executable, "-c", HEAD % LIB + textwrap.dedent(code)], cwd=engine_build.ROOT,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-3000:]
    return run


@pytest.mark.parametrize("add", [
    "oe.fdtd.Nf2ffBox(e[1], (4, 4, 4), (15, 15, 15), [1e9])",
    "e[1].add_mur(oe.MurAbcConfig.all(1))",
    "e[1].add_dispersive(oe.DrudeMaterial(2e11, 1e9), np.array([[8, 8, 8]], dtype=np.uint64))",
])
def test_pack_refuses_what_was_added_after_it_was_made(child, add):
    """A recorder's tables are filled for its own engine's batches only: the
    pack's passes would read none, or another batch's."""
    child(f"""
    e = [engine((20, 20, 20)) for _ in range(2)]
    p = oe.Pack(e)
    p.run_batch([batch(4), batch(4)])
    {add}
    launched("", True)
    try:
        p.run_batch([batch(4), batch(4)])
    except oe.ConfigError:
        pass
    else:
        raise AssertionError("accepted")
    assert launched("") == 0
    p.run_batch([batch(4), None])  # the others go on
    assert launched("k_fused") > 0
    """)


# 64 items of 2,048 cells fill four SMs' limit of 16 items each; a whole
# (y, z) plane of these grids takes more
@pytest.mark.parametrize("dims,layers", [((8, 500, 500), None), ((1, 600, 600), None), ((24, 400, 400), (8,) * 6)])
@pytest.mark.parametrize("autotune", [True, False])
def test_wide_planes_have_a_plan(child, dims, layers, autotune):
    child(f"""
    knob("sms", 4)
    e = engine({dims}, {layers}, autotune={autotune})
    e.run_batch(batch(5))
    assert fused(e) and launched("k_fused") > 0
    """)


def test_pack_of_small_shares_has_plans(child):
    """An engine beside much larger ones plans for one SM."""
    child("""
    e = [engine((1, 300, 300)), engine((4, 300, 300), (1, 1, 8, 8, 8, 8)), engine((40, 300, 300))]
    knob("sms", 8)
    oe.Pack(e).run_batch([batch(5)] * 3)
    assert all(map(fused, e)) and launched("k_update") == 0
    """)


def test_profiles_beyond_shared_memory_keep_the_separate_kernels(child):
    """6 x 4 B x 20,000 layers of one profile: no CTA holds them."""
    child("""
    e = [engine((20010, 3, 3), (20000, 0, 0, 0, 0, 0)) for _ in range(2)]
    e[0].run_batch(batch(5))
    assert not fused(e[0]) and launched("k_update_h") > 0 and launched("k_fused") == 0
    oe.Pack(e[1:]).run_batch([batch(5)])
    assert launched("k_update_h_pack") > 0 and launched("k_fused") == 0
    """)


# the sets' hash table is 2 MB; ids 1.1 MB; the second fields 26 MB; psi 5 MB
@pytest.mark.parametrize("refused", [2 << 20, 1 << 20, 20 << 20, 4 << 20])
def test_no_room_for_fused_buffers_keeps_the_separate_kernels(child, refused):
    child(f"""
    e = engine((100, 100, 110), (8,) * 6, autotune=False)
    used = F.fake_pool_used()
    knob("fail_pool_from", {refused})
    e.run_batch(batch(5))
    assert not fused(e) and launched("k_update_h") > 0
    assert F.fake_pool_used() - used < 1 << 20  # nothing of the attempt stays
    """)


def test_no_room_for_taps_shortens_the_spans(child):
    child("""
    e = engine((30, 150, 150))
    e.add_probe(oe.fdtd.current_probe((15, 20, 20), (15, 120, 120), 0))
    e.run_batch(batch(2))
    knob("fail_pool_from", 1 << 20)
    assert e.run_batch(batch(3000)).timesteps_executed == 3000 and fused(e)
    """)


# A span's first run goes without a graph, per parity of the buffers.  The
# second of two captured passes (which swap the buffers) cannot be launched; the
# graph cannot be made; it cannot be launched, when new or when kept.
@pytest.mark.parametrize("steps,runs,knobs", [(3, 1, 'knob("pass_kernel", 1), knob("fail_kernel", 1)'),
                                              (1, 2, 'knob("fail_instantiate", 1)'), (1, 2, 'knob("fail_graph_launch", 1)'),
                                              (1, 4, 'knob("fail_graph_launch", 1)')])
@pytest.mark.parametrize("layers", [None, (4,) * 6])
def test_a_graph_that_fails_leaves_the_fields_current(child, steps, runs, knobs, layers):
    """(Kernels do nothing here: what was written must come back.)"""
    child(f"""
    e = engine((20, 21, 22), {layers}, autotune=False)
    for _ in range({runs}):
        e.run_batch(batch({steps}))
    f = np.random.default_rng(0).standard_normal((2, 3, 20, 21, 22), dtype=np.float32)
    e.write_fields(f[0], f[1])
    {knobs}
    try:
        e.run_batch(batch({steps}))
    except N.CudaError:
        pass
    else:
        raise AssertionError("no error")
    assert fused(e)
    got = e.read_fields()
    assert np.array_equal(got[0], f[0]) and np.array_equal(got[1], f[1])
    """)


def test_graphs_of_both_parities_are_kept(child):
    """Eight span lengths were kept before a span had a graph per parity."""
    child("""
    e = engine((20, 21, 22), autotune=False)
    lengths = (1, 3, 5, 9, 11, 13, 17, 19)
    for _ in range(5):
        for n in lengths:
            e.run_batch(batch(n))
    before = F.fake_instantiated()
    assert before > 0
    for _ in range(3):
        for n in lengths:
            e.run_batch(batch(n))
    assert F.fake_instantiated() == before
    """)


def test_no_workspace_takes_the_forms_without(child):
    """The GEMM's split sums and the column sum's parts are memory that the
    one-part forms do not need."""
    child("""
    def calls():
        a, b, c = (np.zeros(n, np.float32) for n in (128 * 4096, 640 * 4096, 128 * 640))
        N.check(L.oems_tc_gemm_bf16(a.ctypes.data, 4096, b.ctypes.data, 4096, c.ctypes.data, 640, 128, 640, 4096, 0.0, None, None))
        N.check(L.oems_pk_colsum(b.ctypes.data, 20480, 128, c.ctypes.data, None))
        return [launched(k) for k in ("k_gemm_tc", "k_gemm_sum", "k_colsum_part", "k_colsumEPK")]
    assert calls() == [1, 1, 1, 0]
    knob("fail_pool_from", 0)
    launched("", True)
    assert calls() == [1, 0, 0, 1]
    """)


@pytest.mark.parametrize("nz,rows", [(24, False), (31, False), (32, True), (33, False), (38, False), (64, True), (65, False),
                                     (96, True), (106, False), (127, False), (128, True), (129, True), (160, True)])
def test_cylindrical_form(child, nz, rows):
    """The row form leaves lanes idle in short rows that do not fill their
    warps: up to 1.6 times as long as the flat form."""
    child(f"""
    from openems_b200.cylindrical import CylindricalEngine, CylindricalGrid, CylindricalOperator
    g = CylindricalGrid.uniform(0.005, 0.015, 5, 8, 0.0, 0.01, {nz})
    assert g.dimensions()[2] == {nz}
    with CylindricalEngine(CylindricalOperator(g, 1e-13)) as eng:
        eng.step(2)
    assert (launched("k_cyl_rows") > 0) == {rows} and (launched("k_cyl_flat") > 0) != {rows}
    """)


# no pinned memory; some of the lanes; none for the second call's larger pieces
@pytest.mark.parametrize("passed", [0, 1, 3])
@pytest.mark.parametrize("dims", [(60, 61, 62), (100, 120, 127)])  # one lane; several
def test_refused_pinned_memory_does_not_fail_a_read(child, passed, dims):
    child(f"""
    e = engine({dims})
    f = np.random.default_rng(0).standard_normal((2, 3) + {dims}, dtype=np.float32)
    e.write_fields(f[0], f[1])
    knob("pass_host", {passed}), knob("fail_host", -1)
    for _ in range(4):
        got = e.read_fields()
        assert np.array_equal(got[0], f[0]) and np.array_equal(got[1], f[1])
    """)


def test_concurrent_reads_share_the_pinned_buffers(child):
    """Made once, whatever the number of callers, and bounded."""
    child("""
    from concurrent.futures import ThreadPoolExecutor
    es, fs = [], []
    for k in range(6):
        es.append(engine((100, 120, 121 + k)))
        fs.append(np.random.default_rng(k).standard_normal((2, 3, 100, 120, 121 + k), dtype=np.float32))
        es[k].write_fields(fs[k][0], fs[k][1])
    for _ in range(30):  # (the buffers grow with what has been copied)
        es[0].read_fields()
    before = F.fake_pins()
    with ThreadPoolExecutor(6) as pool:
        for _ in range(20):
            for got, f in zip(pool.map(lambda e: e.read_fields(), es), fs):
                assert np.array_equal(got[0], f[0]) and np.array_equal(got[1], f[1])
    assert F.fake_pins() - before <= 16 and F.fake_pinned() <= 65 << 20
    L.oems_release_cached_memory(0)
    assert F.fake_pinned() < 1 << 20
    """)


def test_a_small_first_read_pins_little(child):
    """Pinned memory takes longer to make than a read of a few MB."""
    child("""
    engine((40, 40, 65)).read_fields()
    assert F.fake_pinned() <= 1 << 20
    """)


def test_scenes_of_other_materials_share_their_plans(child):
    """A plan was found by up to 33 timings again whenever the number of
    distinct coefficient sets was another."""
    child("""
    def one(n):
        op = oe.Operator(oe.Grid.uniform(30, 31, 32, 1e-3), oe.BoundaryConditions.all_pec())
        for k in range(n):
            op.set_material(2.0 + k, 1.0, 0.0, 0.0, (k, k + 1, 0, 31, 0, 32))
        e = oe.Engine(op, compressed=True)
        e.add_cpml(oe.CpmlBoundaries(layers=(4,) * 6))
        launched("", True)
        e.run_batch(batch(5))
        return launched("k_fused"), len(e.tune_report())
    first = one(2)
    assert first[0] > 200 and first[1] > 20
    for n in (5, 9, 20):
        again = one(n)
        assert again[0] < 20 and again[1] == first[1]
    """)


def test_plans_of_one_step_engines_are_searched(child):
    """A Mur engine of a grid that a plain engine ran before tunes its
    one-step passes as if it had been the first, and so does an engine that is
    given a recorder later."""
    child("""
    def tried(e):
        e.run_batch(batch(4))
        return sorted(r["extra"] % 10 for r in e.tune_report() if r["kind"] == 5)
    plain = engine((30, 31, 32))
    got = tried(plain)  # (batches of one step are all one-step passes)
    assert got.count(2) > 10 and got.count(1) > 10 and launched("k_fused") > 0
    mur = engine((30, 31, 32))
    mur.add_mur(oe.MurAbcConfig.all(1))
    assert tried(mur).count(1) > 10 and tried(mur).count(2) == 0
    late = engine((30, 31, 33))
    assert tried(late).count(2) > 10
    oe.fdtd.Nf2ffBox(late, (4, 4, 4), (15, 15, 15), [1e9])
    assert tried(late).count(1) > 10 and fused(late) and late.launch_info()["stages"] == 1
    """)


def test_memory_that_is_tight_once_is_not_held_against_an_engine(child):
    """The quarter counts what the pool holds free, and is looked at again."""
    child("""
    mb = 24 * 64 ** 3 / 2.0 ** 20  # fields of an engine; coefficients are twice that
    knob("capacity", int(12 * mb * 2 ** 20))
    big = [engine((64, 64, 64), autotune=False) for _ in range(3)]
    e = big[0]
    e.run_batch(batch(4))
    assert not fused(e)
    big[2].close()  # to the pool, not to the driver
    big[1].close()
    e.run_batch(batch(4))
    assert fused(e)
    """)


def test_a_pack_that_cannot_run_fused_holds_nothing_for_it(child):
    child("""
    knob("capacity", 1 << 30)
    e = [engine((40, 41, 44)), engine((40, 41, 44), kernels="register"), engine((20010, 3, 3), (20000, 0, 0, 0, 0, 0))]
    for other in e[1:]:  # kernels asked for by name; profiles that no CTA holds
        e[0].reset()
        used = F.fake_pool_used()
        p = oe.Pack([e[0], other])
        p.run_batch([batch(4)] * 2)
        assert launched("k_fused") == 0 and launched("k_update_h_pack") > 0
        assert F.fake_pool_used() - used < 1 << 20
    """)


def test_graphs_of_long_spans_are_small(child):
    """An engine's first batch of 400 steps with hooks and a recorder: no graph
    of thousands of launches, and none for what is run once."""
    child("""
    e = engine((30, 31, 32), (4,) * 6, autotune=False)
    e.add_dispersive(oe.DrudeMaterial(2e11, 1e9), np.array([[8, 8, 8]], dtype=np.uint64))
    oe.fdtd.Nf2ffBox(e, (6, 6, 6), (20, 20, 20), [1e9])
    assert e.run_batch(batch(400)).timesteps_executed == 400
    assert 0 < F.fake_largest_graph() <= 256 and F.fake_instantiated() <= 2
    for _ in range(3):
        e.run_batch(batch(400))
    assert F.fake_instantiated() <= 4
    plain, before = engine((30, 31, 32), autotune=False), F.fake_instantiated()
    plain.run_batch(batch(100))
    assert F.fake_instantiated() == before
    plain.run_batch(batch(100)), plain.run_batch(batch(100))
    assert F.fake_instantiated() == before + 1
    """)


def test_pieces_of_a_span_are_all_run(child):
    """Every step of spans around the pieces' lengths, probes included."""
    child("""
    e = engine((20, 21, 22), (4,) * 6, autotune=False, graphs=False)
    e.add_point_probe(0, (3, 3, 3))
    e.run_batch(batch(1))
    for n in (511, 512, 513, 700, 1023, 1025, 3003):  # (one launch a pass: 512 steps a piece)
        launched("", True)
        e.run_batch(batch(n))
        passes, sums = launched("k_fused"), launched("k_probe_sums")
        assert passes == (n + 1) // 2 and sums == launched("k_set_i64") == -(-n // 512), (n, passes, sums)
    """)


# us of a pass' launch and of an update kernel's; the update takes two a step
@pytest.mark.parametrize("what,dims,pass_us,update_us,want", [
    ("mur", (30, 31, 32), 20, 13, True), ("mur", (30, 31, 32), 20, 11, False),
    ("recorder", (30, 31, 32), 20, 10.1, True), ("recorder", (30, 31, 32), 20, 9.9, False),
    ("plain", (30, 31, 32), 80, 10, True), ("plain", (1, 80, 90), 80, 21, True), ("plain", (1, 80, 90), 80, 19, False),
    ("mur", (170, 171, 172), 80, 1, True)])
def test_one_step_passes_are_taken_where_they_are_faster(child, what, dims, pass_us, update_us, want):
    """Timed against the separate kernels, but for a grid past the L2 whose
    bytes alone take those longer (5 M cells: 92 us)."""
    child(f"""
    knob("pass_ns", int({pass_us} * 1000)), knob("update_ns", int({update_us} * 1000))
    def make():
        e = engine({dims})
        if {what!r} == "mur":
            e.add_mur(oe.MurAbcConfig.all(1))
        if {what!r} == "recorder":
            oe.fdtd.Nf2ffBox(e, (4, 4, 4), (15, 15, 15), [1e9])
        return e
    for e in (make(), make()):  # tuned, and from what was tuned
        for _ in range(2):
            e.run_batch(batch(6))
            assert fused(e) == {want}, e.tune_report()
        used = F.fake_pool_used()
    e = engine({dims}, autotune=False)
    e.run_batch(batch(6))
    assert fused(e)
    """)


@pytest.mark.parametrize("rows,w,parts", [(4096, 33, False), (8192, 128, False), (12265, 128, False), (12266, 128, True),
                                          (6132, 256, False), (6133, 256, True), (4095, 640, False), (4096, 640, True),
                                          (2048, 640, False), (16384, 16, False), (24576, 16, True), (65536, 128, True)])
def test_column_sums_in_parts_where_they_pay(child, rows, w, parts):
    """From 4,096 rows on whatever the width, 8,192 x 128 took 10.2 us instead
    of 8.2."""
    child(f"""
    x, y = np.zeros({rows} * {w}, np.float32), np.zeros({w}, np.float32)
    N.check(L.oems_pk_colsum(x.ctypes.data, {rows}, {w}, y.ctypes.data, None))
    assert (launched("k_colsum_part") == 1) == {parts} and (launched("k_colsumEPK") == 1) != {parts}
    """)


@pytest.mark.parametrize("m,n,k,split", [(128, 1024, 2048, True), (128, 1024, 1984, False), (512, 512, 2048, True),
                                         (640, 640, 2048, False), (1000, 512, 4032, False), (640, 640, 4096, True)])
def test_gemm_split_where_it_pays(child, m, n, k, split):
    """1000 x 512 x 2048 took 20.0 us in parts and 16.5 whole."""
    child(f"""
    a, b, c = (np.zeros(q, np.float32) for q in ({m} * {k} // 2 + 8, {n} * {k} // 2 + 8, {m} * {n}))
    at = [q.ctypes.data + -q.ctypes.data % 16 for q in (a, b)]
    N.check(L.oems_tc_gemm_bf16(at[0], {k}, at[1], {k}, c.ctypes.data, {n}, {m}, {n}, {k}, 0.0, None, None))
    assert launched("k_gemm_tc") == 1 and (launched("k_gemm_sum") == 1) == {split}
    """)


@pytest.mark.parametrize("b,t,c,wide", [(8, 64, 128, False), (1, 16, 8, False), (8, 128, 128, True), (4, 8192, 6, False)])
def test_column_gather_form(child, b, t, c, wide):
    """Small launches are shorter with the plain kernel (4.0 us against 4.2)."""
    child(f"""
    x, y = np.zeros({b} * {t} * {c} * 5 + 4, np.float32), np.zeros({b} * {t} * {c} + 4, np.float32)
    at = [q.ctypes.data + -q.ctypes.data % 16 for q in (x, y)]
    N.check(L.oems_pk_col2im_causal(at[0], 5 * {c}, at[1], {b}, {t}, {c}, 5, 2, None))
    assert (launched("k_col2im_causal4") == 1) == {wide} and launched("k_col2im_causal") == 1
    """)


@pytest.mark.parametrize("update_us,fused_wins", [(150, True), (12, False)])
@pytest.mark.parametrize("every", [0, 10])
def test_packs_take_the_faster_route(child, update_us, fused_wins, every):
    """Three engines: 3 x 50 us a pass of two steps, or two shared launches a
    step; run by one, then by the other, on the clock."""
    child(f"""
    knob("pass_ns", 50000), knob("update_ns", {update_us} * 1000)
    def batches(n):
        return [oe.EngineBatch(num_steps=n, energy_monitoring=oe.EnergyMonitorConfig(sample_interval={every}, track_peak=True))] * 3
    def make():
        return [engine((20, 21, 22 + k)) for k in range(3)]
    def route(p, n):  # a length of its own is launched or captured anew
        launched("", True)
        p.run_batch(batches(n))
        f, u = launched("k_fused"), launched("k_update_h_pack")
        assert (f > 0) != (u > 0), (f, u)
        return f > 0
    es = make()
    p = oe.Pack(es)
    knob("real_time", 1)
    for n in (300, 300, 300):
        p.run_batch(batches(n))
    assert launched("k_fused") > 0 and launched("k_update_h_pack") > 0  # both have run
    assert es[2].current_timestep() == 900
    assert route(p, 23) == {fused_wins}
    launched("", True)
    fs = make()
    q = oe.Pack(fs)  # another pack of such grids: no tuning, no clock
    assert route(q, 37) == {fused_wins} and launched("k_update") < 100
    """)


def test_source_tables_are_sent_when_they_change(child):
    child("""
    def run(e, n, cells):
        dt = 1e-12
        x = [oe.Excitation.gaussian_pulse(1e-11, 1e-11, 2, c) for c in cells]
        before = F.fake_copies()
        e.run_batch(oe.EngineBatch(num_steps=n, excitations=[oe.ScheduledExcitation.from_excitation(q, 0, n, dt) for q in x]))
        return F.fake_copies() - before
    F.fake_copies.restype = ctypes.c_longlong
    e = engine((20, 21, 22), autotune=False)
    a, b = [(3, 4, 5), (6, 7, 8)], [(3, 4, 5), (6, 7, 9)]
    run(e, 2, a)
    again = run(e, 2, a)
    assert run(e, 2, a) == again
    assert run(e, 2, b) == again + 2  # two tables
    assert run(e, 2, b) == again
    assert run(e, 3, b) == again + 2  # other sample counts
    assert run(e, 2, a) == again + 2
    """)


def test_no_room_to_time_the_separate_kernels_keeps_the_passes(child):
    """Tuning them saves fields and psi in one block; the passes' own buffers
    are smaller."""
    child("""
    e = engine((60, 61, 64), (8,) * 6)
    e.add_mur(oe.MurAbcConfig.all(1))
    knob("fail_pool_from", 24 * 60 * 61 * 64 + 4096)
    knob("pass_ns", 10 ** 9)
    e.run_batch(batch(4))
    assert fused(e)
    """)
