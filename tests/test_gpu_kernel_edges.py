"""The step's kernels at the sizes where they can go wrong -- tile and chunk
remainders, odd row lengths, slabs that meet or overlap, the smallest blocks --
against the oracle (FP64, 1e-11) and FP64 (FP32C, 1e-5), from a seeded field
that fills the blocks so that every slab and face has work in the first stage."""
import numpy as np
import pytest

from gpu_helpers import rel_l2
from inputs import problem

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


def deck(mesh, op, dims, npml, response=""):
    nq1, nq2, nr, ns = dims
    extra = "" if op == "traditional" else f",\n fd_type = '{op.split()[0]}',\n order = {op.split()[1]}"
    extra += response
    s = problem("TPV5", "slip-weakening_friction", mesh, extra=extra, w_fault="F") + "&block_list\n"
    for b, (n, lo, hi) in enumerate(((nq1, -3.0, 0.0), (nq2, 0.0, 3.0))):
        i = b + 1
        s += (f"btp({i})%nqrs = {n}, {nr}, {ns},\nbtp({i})%aqrs = {lo}, 6.0, -1.5,\nbtp({i})%bqrs = {hi}, 9.0, 1.5,\n"
              f"btp({i})%rho_s_p = 2.67, 3.464, 6.0,\nbtp({i})%lqrs = {1 - b}, 2, 1,\nbtp({i})%rqrs = {b}, 1, 1,\n")
        if npml:
            s += (f"btp({i})%pml_lqrs = {'FT'[1 - b]}, F, T,\nbtp({i})%pml_rqrs = {'FT'[b]}, T, T,\n"
                  f"btp({i})%npml = {npml},\n")
    return s + " /\n"


def start(shape, seed):
    """Nine smooth components: sine products of 8 to 20 points' length."""
    rng = np.random.default_rng(seed)
    out = np.zeros((9,) + shape)
    for c in range(9):
        ax = [np.sin(np.arange(n) * 2 * np.pi / rng.uniform(8, 20) + rng.uniform(0, 6)) for n in shape]
        out[c] = (0.02 if c < 3 else 0.3) * ax[0][:, None, None] * ax[1][None, :, None] * ax[2][None, None, :]
    return out


# (mesh, operator, (nq1, nq2, nr, ns), npml)
CASES = [
    ("cartesian", "traditional", (12, 13, 12, 12), 0),       # the smallest blocks of the FP64 kernel
    ("curvilinear", "traditional", (33, 47, 15, 37), 0),     # one column, one row and one plane into a tile
    ("curvilinear", "traditional", (64, 31, 24, 32), 0),     # whole tiles
    ("cartesian", "traditional", (76, 41, 25, 18), 7),       # 40-wide tiles, odd rows
    ("curvilinear", "traditional", (25, 26, 34, 19), 9),     # s slabs that meet but for one plane
    ("cartesian", "traditional", (27, 22, 29, 18), 10),      # s slabs that overlap
    ("curvilinear", "traditional", (41, 34, 27, 30), 26),    # slabs wider than the q tiles of the pre-kernel
    ("cartesian", "upwind 6", (40, 45, 29, 22), 6),
    ("curvilinear", "upwind 6", (33, 30, 22, 26), 5),
    ("curvilinear", "upwind 5", (23, 26, 21, 24), 5),
    ("cartesian", "upwind_drp 6", (31, 34, 27, 25), 7),
    ("curvilinear", "upwind 9", (28, 33, 26, 27), 4),
    ("cartesian", "upwind 2", (22, 35, 24, 23), 0),
]


@pytest.mark.parametrize("mesh,op,dims,npml", CASES, ids=[f"{m}-{o}-{d}-{n}".replace(" ", "") for m, o, d, n in CASES])
def test_kernel_edges(wqlmod, oracle_lib, ctx, tmp_path, mesh, op, dims, npml):
    path = tmp_path / "edges.in"
    path.write_text(deck(mesh, op, dims, npml))
    runs = [oracle_lib.Oracle(str(path))] + [wqlmod.Scenario(ctx, str(path), precision=p)
                                             for p in (wqlmod.FP64, wqlmod.FP32C)]
    for r in runs:
        for b in range(2):
            f = start((dims[3], dims[2], dims[b]), 10 + b)
            for c in range(9):
                r.set_field(b, c, f[c])
        r.step(3)
    for r in runs[1:]:
        r.sync(check_nan=True)
    for b in range(2):
        o, d, f = (r.fields(b) for r in runs)
        assert rel_l2(d, o) < 1e-11
        assert rel_l2(f, d) < 1e-5
