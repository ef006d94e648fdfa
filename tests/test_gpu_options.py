"""Combinations of options that the other GPU tests do not reach, each against
the oracle, FP64 or the same run without the option."""
import threading

import numpy as np
import pytest

from gpu_helpers import rel_l2
from test_gpu_kernel_edges import CASES, deck, start

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wqlmod():
    import wql
    return wql


@pytest.fixture(scope="module")
def ctx(wqlmod):
    c = wqlmod.Context(0)
    yield c
    c.close()


def fill(sim, dims):
    for b in range(2):
        f = start((dims[3], dims[2], dims[b]), 10 + b)
        for c in range(9):
            sim.set_field(b, c, f[c])


ANELASTIC = "&anelastic_list\n c = 2.0,\n weight_exp = 0.6,\n fref = 1.0 /\n"


# (mesh, operator, (nq1, nq2, nr, ns), npml): row remainders, s slabs that overlap or meet, per-point and TMA gradients
@pytest.mark.parametrize("mesh,op,dims,npml", [
    ("cartesian", "traditional", (27, 22, 29, 18), 10),
    ("curvilinear", "traditional", (33, 25, 20, 22), 12),
    ("cartesian", "upwind 6", (41, 34, 25, 21), 14),
    ("curvilinear", "upwind 6", (30, 31, 24, 28), 17),
    ("cartesian", "upwind 4", (26, 23, 19, 20), 11),
])
def test_attenuation_in_slabs_that_overlap(wqlmod, oracle_lib, ctx, tmp_path, mesh, op, dims, npml):
    """Where the two slabs of an axis overlap, the strain rates lose the + side's fields alone, in
    the kernel that forms the gradient and in the one that is handed it.  FP32C is held to 1e-6 in
    the velocities and in the stresses: ten times what FP32 coefficients and rates alone leave."""
    text = deck(mesh, op, dims, npml, ",\n response = 'anelastic'") + ANELASTIC
    path = tmp_path / "an.in"
    path.write_text(text)
    o = oracle_lib.Oracle(str(path))
    runs = [wqlmod.Scenario(ctx, text=text, precision=p) for p in (wqlmod.FP64, wqlmod.FP32C)]
    for r in [o] + runs:
        fill(r, dims)
        r.step(12)
    for b in range(2):
        ref, d, f = (r.fields(b) for r in [o] + runs)
        assert rel_l2(d, ref) < 1e-11
        assert rel_l2(f[:3], d[:3]) < 1e-6
        assert rel_l2(f[3:], d[3:]) < 1e-6


# odd row lengths in both blocks; the upwind pair; a component of over 64 MiB (two chunks)
@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
@pytest.mark.parametrize("mesh,op,dims,npml", [
    ("curvilinear", "traditional", (33, 27, 21, 23), 6),
    ("cartesian", "upwind 6", (41, 35, 22, 24), 0),
    ("cartesian", "traditional", (355, 13, 170, 180), 0),
])
def test_reads_leave_a_run_as_it_is(wqlmod, ctx, mesh, op, dims, npml, prec):
    """Reads between steps, between stages, and from other threads during steps: the run ends bit for
    bit where it ends without them, and threads reading at once each get their own component."""
    p = wqlmod.FP64 if prec == "fp64" else wqlmod.FP32C
    plain, read = (wqlmod.Scenario(ctx, text=deck(mesh, op, dims, npml), precision=p) for _ in range(2))
    for s in (plain, read):
        fill(s, dims)
    plain.step(9)
    got = read.fields(0)
    f = start((dims[3], dims[2], dims[0]), 10)
    assert np.array_equal(got, f if prec == "fp64" else f.astype(np.float32).astype(float))
    read.step(2)
    read.fields(1)
    for k in range(1, 6):
        read.stage(k)
        read.fields(k % 2)
    done = threading.Event()

    def monitor():
        while not done.is_set():
            read.field(0, 4)
            read.field(1, 1)

    t = [threading.Thread(target=monitor) for _ in range(2)]
    for x in t:
        x.start()
    for _ in range(6):
        read.step(1)
        read.sync()
    done.set()
    for x in t:
        x.join()
    want = [plain.fields(b) for b in range(2)]
    for b in range(2):
        assert np.array_equal(read.fields(b), want[b])
    wrong = []

    def reader(c):
        for _ in range(4):
            if not np.array_equal(read.field(0, c), want[0][c]):
                wrong.append(c)

    t = [threading.Thread(target=reader, args=(c,)) for c in range(9)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not wrong


@pytest.mark.parametrize("op", ["traditional", "upwind 8", "upwind_drp 66"])
def test_curvilinear_rounding(wqlmod, ctx, op):
    """FP32C on a regular grid: written as a curvilinear block, its error against FP64 is that of the
    Cartesian one (the same factors, rounded as often), within a tenth: a product of factors that is
    rounded once for all points shifts every point alike and shows as a quarter or more."""
    dims, err = (61, 54, 47, 51), {}
    for mesh in ("cartesian", "curvilinear"):
        d, f = (wqlmod.Scenario(ctx, text=deck(mesh, op, dims, 0), precision=p) for p in (wqlmod.FP64, wqlmod.FP32C))
        for s in (d, f):
            fill(s, dims)
            s.step(6)
        err[mesh] = [np.hypot(*(rel_l2(f.fields(b)[c], d.fields(b)[c]) for b in range(2)))
                     for c in (slice(0, 3), slice(3, 9))]
    assert all(k < 1.1 * c for k, c in zip(err["curvilinear"], err["cartesian"])), err


def stencil_ms(s, tuning=None, steps=40):
    """Least device time of one step's stencil launches in five runs."""
    if tuning:
        s.set_tuning(*tuning)
    s.step(3)
    best = 1e9
    for _ in range(5):
        s.profile(True)
        s.step(steps)
        best = min(best, s.kernel_times()["stencil"][0] / steps)
    s.profile(False)
    return best


@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
@pytest.mark.parametrize("mesh,dims", [("cartesian", (41, 41, 41, 41)), ("curvilinear", (64, 64, 48, 57))])
def test_autotune_is_no_slower_than_the_default(wqlmod, ctx, mesh, dims, prec):
    """The trial launches what a step launches, so the choice cannot lose to the default by more than
    the noise of launches of some 20 us."""
    s = wqlmod.Scenario(ctx, text=deck(mesh, "traditional", dims, 0), precision=wqlmod.FP64 if prec == "fp64" else wqlmod.FP32C)
    fill(s, dims)
    default = stencil_ms(s)
    choice = s.autotune(20)
    tuned = stencil_ms(s)
    assert tuned < 1.15 * default, (choice, tuned, default)


@pytest.mark.parametrize("variant,launches", [(0, 5), (1, 5), (2, 10), (6, 5)])
def test_profile_counts_launches(wqlmod, ctx, variant, launches):
    """wql_kernel_times counts the stencil's launches: one a stage over both blocks, or one a block."""
    s = wqlmod.Scenario(ctx, text=deck("curvilinear", "traditional", (33, 27, 21, 23), 0), precision=wqlmod.FP32C)
    s.set_tuning(variant, 0)
    s.profile(True)
    s.step(3)
    assert s.kernel_times()["stencil"][1] == 3 * launches


@pytest.mark.parametrize("op,nr", [("traditional", 12), ("traditional", 13), ("upwind 6", 13)])
def test_tile_width_for_short_r_axes(wqlmod, ctx, op, nr):
    """Rows whose closures 40 x 8 tiles would not hold take the 32 x 12 tiles, not the per-point kernel."""
    dims, out = (76, 75, nr, 40), {}
    for v in (0, 6, 1):
        s = wqlmod.Scenario(ctx, text=deck("cartesian", op, dims, 0), precision=wqlmod.FP32C)
        s.set_tuning(v, 0)
        fill(s, dims)
        s.step(4)
        out[v] = np.stack([s.fields(b)[:, 3:-3, 3:-3, 3:70] for b in range(2)])
    assert np.array_equal(out[0], out[6])
    assert not np.array_equal(out[6], out[1])  # the two kernels round differently


@pytest.mark.parametrize("dims", [(280, 280, 41, 41), (120, 120, 100, 100), (76, 75, 150, 150), (120, 160, 14, 60)])
def test_tile_width_by_schedule(wqlmod, ctx, dims):
    """The width that the schedules choose is no slower than 32-wide tiles (but for noise), and faster
    where 40-wide ones save planes."""
    s = wqlmod.Scenario(ctx, text=deck("cartesian", "traditional", dims, 0), precision=wqlmod.FP32C)
    fill(s, dims)
    default, narrow = stencil_ms(s, (0, 0), 20), stencil_ms(s, (6, 0), 20)
    assert default < 1.08 * narrow
    if dims[0] in (76, 120) and dims[2] in (150, 14):
        assert default < 0.97 * narrow


def test_late_request_joins_the_running_one(wqlmod, ctx):
    """A request whose set-up is done 7 ms before another's end joins it: the server does not queue the
    rest of a run ahead of the device.  Four tries, since set-up times vary."""
    import time
    import wql_configs
    medium, steps = wql_configs.config4_medium(48), 160
    reqs = [wql_configs.config4_request(i, n_lo=24, n_hi=44, steps=steps, medium=medium) for i in range(2)]
    srv = wqlmod.Server(ctx, hbm_budget_bytes=64 << 30, round_steps=4)

    def serve(delay):
        ids = [srv.submit(reqs[0][0], steps, media=reqs[0][1])]
        while srv.stats()["active"] < 1 and srv.stats()["completed"] < 1:
            time.sleep(0.0002)
        time.sleep(delay)
        ids.append(srv.submit(reqs[1][0], 8, media=reqs[1][1]))
        for r in ids:
            assert srv.wait(r, 300.0) == 1
        return [srv.result(r, 0)[1] for r in ids]

    t = [serve(0.3)[k] for _ in range(3) for k in range(2)]  # one after the other
    run, setup = min(x[2] - x[1] for x in t[::2]), min(x[1] - x[0] for x in t[1::2])
    tries = [serve(max(0.0, run - setup - 0.007)) for _ in range(4)]
    srv.close()
    assert any(b[1] < a[2] - 0.001 for a, b in tries), (run, setup, tries)


@pytest.mark.parametrize("mesh,op,dims,npml", CASES, ids=[f"{m}-{o}-{d}-{n}".replace(" ", "") for m, o, d, n in CASES])
def test_fp32c_velocities_and_stresses(wqlmod, ctx, mesh, op, dims, npml):
    """The edge sizes with velocities and stresses held apart, so that the larger ones do not hide the
    others, to ten times the 1e-7 that FP32 coefficients leave."""
    d, f = (wqlmod.Scenario(ctx, text=deck(mesh, op, dims, npml), precision=p) for p in (wqlmod.FP64, wqlmod.FP32C))
    for s in (d, f):
        fill(s, dims)
        s.step(3)
    for b in range(2):
        x, y = f.fields(b), d.fields(b)
        assert rel_l2(x[:3], y[:3]) < 1e-6
        assert rel_l2(x[3:], y[3:]) < 1e-6


@pytest.mark.parametrize("mesh,dims,npml", [("cartesian", (41, 34, 25, 21), 7), ("curvilinear", (33, 27, 29, 23), 8)])
def test_return_map_beside_slabs(wqlmod, oracle_lib, ctx, tmp_path, mesh, dims, npml):
    """Viscoplasticity on odd extents, where the box outside the slabs starts and ends in the middle of tiles."""
    text = deck(mesh, "traditional", dims, npml, ",\n response = 'plastic',\n plastic_model = 'scec'")
    text = text.replace("TPV5", "TPV26") + "&plastic_list\n cohesion = 0.5,\n friction = 0.02,\n Tv = 0.03 /\n"
    path = tmp_path / "pl.in"
    path.write_text(text)
    o, d = oracle_lib.Oracle(str(path)), wqlmod.Scenario(ctx, text=text, precision=wqlmod.FP64)
    for r in (o, d):
        fill(r, dims)
        r.step(6)
    for b in range(2):
        assert rel_l2(d.fields(b), o.fields(b)) < 1e-11
